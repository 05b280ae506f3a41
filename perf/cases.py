"""The work that users of this package have it do, as measurable cases.

Three kinds, each through the public entry points:

* ``encode``     inference of the DeBERTa-v3 backbone (``FlashDebertaV2Model``), base and large geometry, bf16: one short
                 query, a padded batch with its mask, a full batch, a packed batch of documents;
* ``attention``  the fused attention alone (``ops.disentangled_attention`` / ``..._fp8``), as a caller with its own model uses
                 it: dense, right-padded and packed layouts, bf16 and e4m3;
* ``train``      forward and backward of the attention, through the module (projections and position tables included) or
                 through the operator, all gradients.

Both position terms (c2p and p2c) over 256 log buckets, head size 64, 12 or 16 heads: what every DeBERTa-v3 checkpoint has.
"""
import math
import random

import torch

BUCKETS, MAX_REL, HEAD_DIM, PAD = 256, 512, 64, 0
#: hidden size, layers, heads, feed-forward size
SIZES = {"base": (768, 12, 12, 3072), "large": (1024, 24, 16, 4096)}
VOCAB = 128100


def listed():
    return [
        # one short query through the backbone: what a search or classification service waits for
        {"name": "encode_query", "kind": "encode", "size": "base", "layout": "full", "batch": 1, "seqlen": 29, "shortest": 29},
        # a tokenizer's batch of paragraphs, right-padded to its longest, with the mask made from the ids
        {"name": "encode_padded", "kind": "encode", "size": "base", "layout": "padded", "batch": 16, "seqlen": 253, "shortest": 61},
        # eight documents of one length: the encoder configuration that the package is tuned on
        {"name": "encode_full", "kind": "encode", "size": "base", "layout": "full", "batch": 8, "seqlen": 2048, "shortest": 2048},
        # indexing: documents of every length back to back, the large model (the benchmark's batch, fewer sequences)
        {"name": "encode_packed_large", "kind": "encode", "size": "large", "layout": "packed", "batch": 56, "seqlen": 6007, "shortest": 64},
        # the attention of two ordinary inputs
        {"name": "attn_small", "kind": "attention", "heads": 12, "dtype": "bf16", "layout": "full", "batch": 2, "seqlen": 512, "shortest": 512},
        # a batch of odd, ragged lengths in padded form
        {"name": "attn_padded", "kind": "attention", "heads": 12, "dtype": "bf16", "layout": "padded", "batch": 24, "seqlen": 779, "shortest": 130},
        # long context with trailing padding
        {"name": "attn_long", "kind": "attention", "heads": 12, "dtype": "bf16", "layout": "padded", "batch": 1, "seqlen": 32768, "shortest": 29491},
        # packed documents, 16 heads
        {"name": "attn_packed", "kind": "attention", "heads": 16, "dtype": "bf16", "layout": "packed", "batch": 48, "seqlen": 4099, "shortest": 64},
        # the e4m3 option at its layer shape
        {"name": "attn_e4m3", "kind": "attention", "heads": 16, "dtype": "e4m3", "layout": "full", "batch": 2, "seqlen": 4096, "shortest": 4096},
        # fine-tuning on padded paragraphs: the attention module with its projections
        {"name": "train_padded", "kind": "train", "heads": 12, "through": "module", "layout": "padded", "batch": 12, "seqlen": 509, "shortest": 120},
        # training on long full sequences
        {"name": "train_full", "kind": "train", "heads": 12, "through": "op", "layout": "full", "batch": 4, "seqlen": 2048, "shortest": 2048},
        # training on packed documents
        {"name": "train_packed", "kind": "train", "heads": 16, "through": "op", "layout": "packed", "batch": 32, "seqlen": 1531, "shortest": 48},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["encode", "attention", "train"])
    layout = rng.choice(["full", "padded", "packed"])
    case = {"kind": kind}
    if kind == "encode":
        case["size"] = rng.choice(["base", "large"])
        longest = _spread(rng, 16, 4096 if layout == "packed" else 2048)
        rows, most = _spread(rng, 16, 40000), 64
    elif kind == "attention":
        case["heads"] = rng.choice([12, 16])
        case["dtype"] = rng.choice(["bf16", "bf16", "bf16", "e4m3"])
        longest = _spread(rng, 64, 32768)
        rows, most = _spread(rng, 512, 65536), 256
    else:
        case["heads"] = rng.choice([12, 16])
        case["through"] = "op" if layout == "packed" else rng.choice(["op", "module"])
        longest = _spread(rng, 32, 4096)
        rows, most = _spread(rng, 512, 16384), 64
    shortest = longest
    mean = longest
    if layout != "full":
        shortest = max(1, int(longest * rng.uniform(0.02 if layout == "packed" else 0.2, 0.9)))
        if layout == "packed" and shortest < longest:
            mean = (longest - shortest) / math.log(longest / shortest)
    case.update(layout=layout, batch=max(1, min(most, int(rows / mean))), seqlen=longest, shortest=shortest)
    return case


def _lengths(case):
    """The sequences' lengths: spread evenly over the logarithm from `shortest` to `seqlen`, in an arbitrary fixed order.  A
    padded batch is as wide as its longest sequence; with one sequence alone the rest of its row is padding."""
    n, lo, hi = case["batch"], case["shortest"], case["seqlen"]
    if case["layout"] == "full":
        return [hi] * n
    if n == 1:
        return [lo if case["layout"] == "padded" else hi]
    lens = [int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]
    random.Random(n * 7919 + hi).shuffle(lens)
    return lens


def _cu_seqlens(lens, dev):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32, device=dev)


def _config(size, **extra):
    from transformers.models.deberta_v2.configuration_deberta_v2 import DebertaV2Config
    hidden, layers, heads, ffn = SIZES[size]
    cfg = DebertaV2Config(
        vocab_size=VOCAB, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=heads, intermediate_size=ffn,
        hidden_act="gelu", max_position_embeddings=512, type_vocab_size=0, layer_norm_eps=1e-7, relative_attention=True,
        max_relative_positions=-1, position_buckets=BUCKETS, norm_rel_ebd="layer_norm", share_att_key=True,
        pos_att_type="c2p|p2c", position_biased_input=False, pad_token_id=PAD, hidden_dropout_prob=0.0,
        attention_probs_dropout_prob=0.0)
    for k, v in extra.items():
        setattr(cfg, k, v)
    return cfg


def _random_parameters(module, gen):
    """Weights N(0, 0.02); norm weights around one and biases around zero, as after training."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() > 1:
                p.normal_(0.0, 0.02, generator=gen)
            else:
                p.normal_(1.0 if "LayerNorm.weight" in name else 0.0, 0.02, generator=gen)


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    lens = _lengths(case)
    batch, width, layout = case["batch"], case["seqlen"], case["layout"]
    state = {"case": case}

    if case["kind"] == "encode":
        from flashdeberta_b200.model import FlashDebertaV2Model
        with torch.device("meta"):
            model = FlashDebertaV2Model(_config(case["size"]))
        model = model.to(torch.bfloat16).to_empty(device=dev).eval()
        model.embeddings.position_ids = torch.arange(512, device=dev).view(1, -1)
        _random_parameters(model, gen)
        state["model"] = model
        if layout == "packed":
            state["ids"] = torch.randint(1, VOCAB, (1, sum(lens)), generator=gen, device=dev)
            state["cu"], state["longest"] = _cu_seqlens(lens, dev), max(lens)
        else:
            ids = torch.randint(1, VOCAB, (batch, width), generator=gen, device=dev)
            valid = torch.arange(width, device=dev)[None, :] < torch.tensor(lens, device=dev)[:, None]
            state["ids"] = torch.where(valid, ids, PAD)
        return state

    heads = case["heads"]
    rows = (sum(lens),) if layout == "packed" else (batch, width)
    draw_normal = lambda *shape: torch.randn(*shape, generator=gen, device=dev, dtype=torch.bfloat16)  # noqa: E731
    if case["kind"] == "train" and case["through"] == "module":
        from flashdeberta_b200.attention import FlashDisentangledSelfAttention
        hidden = heads * HEAD_DIM
        cfg = _config("base", hidden_size=hidden, num_attention_heads=heads, pos_att_type=["c2p", "p2c"], max_relative_positions=MAX_REL)
        module = FlashDisentangledSelfAttention(cfg).to(dev).to(torch.bfloat16).train()
        _random_parameters(module, gen)
        state["module"] = module
        state["x"] = draw_normal(*rows, hidden).requires_grad_(True)
        state["rel"] = draw_normal(2 * BUCKETS, hidden).requires_grad_(True)
        state["dout"] = draw_normal(*rows, hidden)
        state["mask"] = (torch.arange(width, device=dev)[None, :] < torch.tensor(lens, device=dev)[:, None]).long()
        return state

    state["qkv"] = [draw_normal(*rows, heads, HEAD_DIM) for _ in range(3)]
    state["tables"] = [0.5 * draw_normal(heads, 2 * BUCKETS, HEAD_DIM) for _ in range(2)]
    state["layout"] = {"max_seqlen": max(lens) if layout == "packed" else width, "position_buckets": BUCKETS,
                       "max_relative_positions": MAX_REL}
    if layout == "packed":
        state["layout"]["cu_seqlens"] = _cu_seqlens(lens, dev)
    elif layout == "padded":
        state["layout"]["seq_lens"] = torch.tensor(lens, dtype=torch.int32, device=dev)
    if case["kind"] == "train":
        for t in state["qkv"] + state["tables"]:
            t.requires_grad_(True)
        state["dout"] = draw_normal(*rows, heads, HEAD_DIM)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "encode":
        with torch.no_grad():
            if case["layout"] == "packed":
                return state["model"](input_ids=state["ids"], cu_seqlens=state["cu"], max_seqlen=state["longest"]).last_hidden_state
            mask = (state["ids"] != PAD).long()  # every batch comes with its own mask
            return state["model"](input_ids=state["ids"], attention_mask=mask).last_hidden_state
    if case["kind"] == "train" and case["through"] == "module":
        leaves = [state["x"], state["rel"], *state["module"].parameters()]
        out, _ = state["module"](state["x"], state["mask"], rel_embeddings=state["rel"])
        return [out.detach(), *torch.autograd.grad(out, leaves, state["dout"])]
    from flashdeberta_b200 import ops
    if case["kind"] == "train":
        leaves = [*state["qkv"], *state["tables"]]
        out = ops.disentangled_attention(*leaves, **state["layout"])
        return [out.detach(), *torch.autograd.grad(out, leaves, state["dout"])]
    with torch.no_grad():
        if case["dtype"] == "e4m3":
            return ops.disentangled_attention_fp8(*state["qkv"], *state["tables"], **state["layout"])
        return ops.disentangled_attention(*state["qkv"], *state["tables"], **state["layout"])


def _attention_flops(lens, heads):
    """Q.K^T and P.V over the valid tokens, and every token against both position tables once."""
    return sum(heads * (4 * n * n * HEAD_DIM + 2 * 2 * n * 2 * BUCKETS * HEAD_DIM) for n in lens)


def work(case):
    lens = _lengths(case)
    tokens = sum(lens)
    rows = tokens if case["layout"] == "packed" else case["batch"] * case["seqlen"]
    if case["kind"] == "encode":
        hidden, layers, heads, ffn = SIZES[case["size"]]
        weights = layers * (4 * hidden * hidden + 2 * hidden * ffn)
        tables = layers * 2 * 2 * BUCKETS * hidden  # the two projected position tables of every layer
        return {"bytes": 2 * (weights + tables) + 2 * tokens * hidden + 8 * rows + 2 * rows * hidden,
                "flops": 2 * tokens * weights + layers * _attention_flops(lens, heads)}
    heads = case["heads"]
    hidden = heads * HEAD_DIM
    table = 2 * BUCKETS * hidden
    forward = _attention_flops(lens, heads)
    if case["kind"] == "attention":
        return {"bytes": 2 * (3 * tokens * hidden + 2 * table + rows * hidden), "flops": forward}
    # backward: five products of the forward's two (the scores again, dP, dV, dQ, dK), three per position term
    flops = forward + sum(heads * (10 * n * n * HEAD_DIM + 3 * 2 * 2 * n * 2 * BUCKETS * HEAD_DIM) for n in lens)
    if case["through"] == "op":
        return {"bytes": 2 * (4 * tokens * hidden + 4 * rows * hidden + 4 * table), "flops": flops}
    # three projections of the tokens, two of the position embeddings, each once forward and twice backward
    flops += 3 * (3 * 2 * tokens * hidden * hidden + 2 * 2 * table * hidden)
    return {"bytes": 2 * (2 * tokens * hidden + 2 * rows * hidden + 2 * table + 2 * 3 * hidden * hidden), "flops": flops}


def tolerance(case):
    if case["kind"] == "encode":  # bf16 activations through 12 or 24 layers
        return {"rel": 2e-2 if case["size"] == "base" else 3e-2}
    if case["kind"] == "train":   # probabilities, their gradients and the bucket sums are rounded to bf16 on the way
        return {"rel": 1.5e-2}
    return {"rel": 3e-2 if case["dtype"] == "e4m3" else 1e-2}

"""GPU parity tests of the attention backward: the two CUDA stages (csrc/attn_bwd.cu) behind
flashdeberta_b200.backward, the autograd wiring of the custom op, and training steps through the module and the model.

Reference gradients: autograd through the fp32 oracle on the host for the op-level tests (same bf16-grid inputs), the
eager backend of the same model with shared weights for the model-level tests.  The reference holds its own backward to
atol = rtol = 5e-3 in fp16 (tests/backward.py:99-102); here inputs, P and dS are bf16 (8 bits of mantissa), so a gradient
tensor is held to  max|got - want| <= 2e-2 * max|want|  and  mean|got - want| <= 2e-3 * max|want|.
"""
import pytest
import torch

from oracle import disentangled_attention as oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"
REL_MAX, REL_MEAN = 2e-2, 2e-3


def _reference(q, k, v, pk, pq, starts, lens, sm, buckets, max_rel, dout):
    leaves = [t.float().cpu().clone().requires_grad_(True) if t is not None else None for t in (q, k, v, pk, pq)]
    with torch.enable_grad():
        out = oracle.attention_core.__wrapped__(leaves[0], leaves[1], leaves[2], leaves[3], leaves[4], starts, lens, sm,
                                                buckets, max_rel)
        grads = torch.autograd.grad(out, [t for t in leaves if t is not None], dout.float().cpu())
    it = iter(grads)
    return [next(it) if t is not None else None for t in leaves]


def _close(got, want, what, rel_max=REL_MAX, rel_mean=REL_MEAN):
    assert torch.isfinite(got.float()).all(), what
    scale = want.abs().max().item() + 1e-20
    diff = (got.float().cpu().reshape(want.shape) - want).abs()
    assert diff.max().item() <= rel_max * scale, (what, "max", diff.max().item() / scale)
    assert diff.mean().item() <= rel_mean * scale, (what, "mean", diff.mean().item() / scale)


def _run_op(q, k, v, pk, pq, dout, **kw):
    from flashdeberta_b200 import ops
    leaves = [t.clone().requires_grad_(True) if t is not None else None for t in (q, k, v, pk, pq)]
    out = ops.disentangled_attention(*leaves, **kw)
    assert out.requires_grad
    grads = torch.autograd.grad(out, [t for t in leaves if t is not None], dout)
    torch.cuda.synchronize()
    ops.check_status()
    it = iter(grads)
    return [next(it) if t is not None else None for t in leaves]


@pytest.mark.parametrize("buckets,max_rel,c2p,p2c", [(256, 512, True, True), (256, 512, True, False),
                                                     (256, 512, False, True), (-1, -1, False, False),
                                                     (-1, 128, True, True), (32, 64, True, True)])
def test_dense_ragged_gradients_vs_oracle_autograd(buckets, max_rel, c2p, p2c):
    g = torch.Generator().manual_seed(21)
    B, L, H, D = 2, 700, 2, 64
    lens = [700, 333]
    span = (buckets if buckets > 0 else max_rel) if (c2p or p2c) else 0
    q, k, v, dout = (torch.randn(B, L, H, D, generator=g).bfloat16().to(DEV) for _ in range(4))
    pk = torch.randn(H, 2 * span, D, generator=g).bfloat16().to(DEV) if c2p else None
    pq = torch.randn(H, 2 * span, D, generator=g).bfloat16().to(DEV) if p2c else None
    sm = oracle.sm_scale_for(D, c2p, p2c)
    got = _run_op(q, k, v, pk, pq, dout, seq_lens=torch.tensor(lens, dtype=torch.int32, device=DEV), max_seqlen=L,
                  sm_scale=sm, position_buckets=buckets, max_relative_positions=max_rel)
    flat = lambda t: t.reshape(-1, H, D)
    dmask = torch.zeros(B, L, 1, 1, device=DEV)
    for b, n in enumerate(lens):
        dmask[b, :n] = 1
    want = _reference(flat(q), flat(k), flat(v), pk, pq, [0, L], lens, sm, buckets, max_rel, flat(dout * dmask))
    for name, a, b in zip(("dq", "dk", "dv", "dpos_key", "dpos_query"), got, want):
        assert (a is None) == (b is None), name
        if a is not None:
            _close(a, b, name)
    assert got[0][1, 333:].abs().max().item() == 0 and got[2][1, 333:].abs().max().item() == 0


def test_packed_gradients_in_several_blocks_vs_oracle_autograd():
    """Packed sequences (an empty one, one of a single token, one of 1500) with the row blocks forced small, so that the p2c sums are
    accumulated over many blocks and the block edges fall inside the bucketed band."""
    from flashdeberta_b200 import backward, ops
    g = torch.Generator().manual_seed(22)
    H, D = 3, 64
    lens = [1500, 0, 1, 261]  # an empty sequence, a single token, an odd length
    cu = [0, 1500, 1500, 1501, 1762]
    T = cu[-1]
    q, k, v, dout = (torch.randn(T, H, D, generator=g).bfloat16().to(DEV) for _ in range(4))
    pk, pq = (torch.randn(H, 512, D, generator=g).bfloat16().to(DEV) for _ in range(2))
    sm = oracle.sm_scale_for(D, True, True)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=DEV)
    kw = dict(cu_seqlens=cu_t, max_seqlen=1500, sm_scale=sm, position_buckets=256, max_relative_positions=512)
    out, lse = ops.disentangled_attention(q, k, v, pk, pq, return_lse=True, **kw)
    got = backward.attention_backward(dout, q, k, v, pk, pq, out, lse, block_bytes=12 * H * 1500 * 192, **kw)
    whole = backward.attention_backward(dout, q, k, v, pk, pq, out, lse, **kw)
    torch.cuda.synchronize()
    want = _reference(q, k, v, pk, pq, cu[:-1], lens, sm, 256, 512, dout)
    for name, a, w, b in zip(("dq", "dk", "dv", "dpos_key", "dpos_query"), got, whole, want):
        _close(a, b, name)
        _close(w, b, name + " (one block)")


def test_gradients_at_2048_keys_with_far_tiles():
    """One sequence long enough that most keys of a row sit at the saturated ends of the tables (the long runs of the
    c2p sums) and that the forward inside the backward op takes its usual launches."""
    g = torch.Generator().manual_seed(23)
    L, H, D = 2048, 2, 64
    q, k, v, dout = (torch.randn(1, L, H, D, generator=g).bfloat16().to(DEV) for _ in range(4))
    pk, pq = (torch.randn(H, 512, D, generator=g).bfloat16().to(DEV) for _ in range(2))
    sm = oracle.sm_scale_for(D, True, True)
    got = _run_op(q, k, v, pk, pq, dout, max_seqlen=L, sm_scale=sm, position_buckets=256, max_relative_positions=512)
    want = _reference(q[0], k[0], v[0], pk, pq, [0], [L], sm, 256, 512, dout[0])
    for name, a, b in zip(("dq", "dk", "dv", "dpos_key", "dpos_query"), got, want):
        _close(a, b, name)


@pytest.mark.parametrize("buckets,max_rel,c2p,p2c", [(256, 512, True, True), (512, 1024, True, True), (32, 64, True, False),
                                                     (-1, 100, False, True), (-1, -1, False, False)])
@pytest.mark.parametrize("layout", ["packed", "padded"])
def test_fused_gradients_at_tile_edges_match_the_block_form(buckets, max_rel, c2p, p2c, layout):
    """Lengths around the edges of the fused kernels' tiles (128 rows, 64 columns), rows outside every sequence, strided inputs,
    and tables of one, several and more than 512 rows, against the block form of the same gradients."""
    from flashdeberta_b200 import backward, ops
    g = torch.Generator().manual_seed(buckets + max_rel)
    H, D, lens = 2, 64, [1, 63, 64, 65, 0, 127, 128, 129, 191, 600]
    span = (buckets if buckets > 0 else max_rel) if (c2p or p2c) else 0
    if layout == "packed":
        cu = torch.tensor([5 + sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
        rows, kw = (int(cu[-1]) + 37,), dict(cu_seqlens=cu, max_seqlen=max(lens))
        inside = torch.arange(rows[0], device=DEV)
        inside = (inside >= 5) & (inside < int(cu[-1]))
    else:
        rows, n = (len(lens), 601), torch.tensor(lens, dtype=torch.int32, device=DEV)
        kw, inside = dict(seq_lens=n, max_seqlen=601), torch.arange(601, device=DEV)[None, :] < n[:, None]
    q, k, v = torch.randn(*rows, 3, H, D, generator=g).bfloat16().to(DEV).unbind(-3)
    dout = torch.randn(*rows, H, D, generator=g).bfloat16().to(DEV)
    pk = torch.randn(H, 2 * span, D, generator=g).bfloat16().to(DEV) if c2p else None
    pq = torch.randn(H, 2 * span, D, generator=g).bfloat16().to(DEV) if p2c else None
    kw.update(sm_scale=oracle.sm_scale_for(D, c2p, p2c), position_buckets=buckets, max_relative_positions=max_rel)
    with torch.no_grad():
        out, lse = ops.disentangled_attention(q, k, v, pk, pq, return_lse=True, **kw)
    out = torch.where(inside[..., None, None], out, 0)
    lse = torch.where(inside.reshape(-1, 1), lse, 0)
    got = backward.attention_backward(dout, q, k, v, pk, pq, out, lse, **kw)
    want = backward.attention_backward(dout * inside[..., None, None], q, k, v, pk, pq, out, lse, block_bytes=1 << 28, **kw)
    torch.cuda.synchronize()
    ops.check_status()
    for name, a, b in zip(("dq", "dk", "dv", "dpos_key", "dpos_query"), got, want):
        assert (a is None) == (b is None), name
        if a is not None:
            _close(a, b.float().cpu(), name)
    for t in got[:3]:
        assert t[~inside].abs().max().item() == 0


def _small_config(backend, **kw):
    from transformers.models.deberta_v2.configuration_deberta_v2 import DebertaV2Config
    cfg = DebertaV2Config(vocab_size=2000, hidden_size=256, num_hidden_layers=2, num_attention_heads=4,
                          intermediate_size=512, relative_attention=True, position_buckets=256,
                          max_relative_positions=512, pos_att_type="c2p|p2c", share_att_key=True,
                          norm_rel_ebd="layer_norm", position_biased_input=False, type_vocab_size=0,
                          layer_norm_eps=1e-7, hidden_dropout_prob=0.0, attention_probs_dropout_prob=0.0,
                          pooler_dropout=0.0, cls_dropout=0.0, **kw)
    cfg.attn_backend = backend
    return cfg


@pytest.mark.parametrize("mask_type,rel_rows,frozen", [(None, 512, ()), (torch.int64, 512, ("rel",)), (torch.bool, 515, ("x", "key_proj")),
                                                       (torch.bfloat16, 512, ("value_proj", "query_proj", "key_proj"))])
def test_module_as_one_node_matches_the_operators(monkeypatch, mask_type, rel_rows, frozen):
    """Training through the module (projections, tables and attention in one autograd node) against the same module operator by
    operator: output and every gradient, with and without a mask, with inputs and projections that need no gradient."""
    from flashdeberta_b200 import ops, projected
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    torch.manual_seed(5)
    module = FlashDisentangledSelfAttention(_small_config("b200")).to(DEV).bfloat16().train()
    B, L = 3, 321
    x, rel = torch.randn(B, L, 256, device=DEV).bfloat16(), torch.randn(rel_rows, 256, device=DEV).bfloat16()
    dout = torch.randn(B, L, 256, device=DEV).bfloat16()
    mask = None
    if mask_type is not None:
        mask = (torch.arange(L, device=DEV)[None, :] < torch.tensor([321, 128, 1], device=DEV)[:, None]).to(mask_type)
        dout = dout * mask[..., None].to(dout.dtype)
    x.requires_grad_("x" not in frozen)
    rel.requires_grad_("rel" not in frozen)
    for name in frozen:
        if hasattr(module, name):
            getattr(module, name).requires_grad_(False)
    leaves = {n: p for n, p in [("x", x), ("rel", rel), *module.named_parameters()] if p.requires_grad}

    def run():
        out, _ = module(x, mask, rel_embeddings=rel)
        return [out.detach(), *torch.autograd.grad(out, list(leaves.values()), dout)]

    assert projected.covers(module, x, None, mask, rel)
    got = run()
    monkeypatch.setattr(projected, "covers", lambda *a: False)
    want = run()
    ops.check_status()
    for name, a, b in zip(["out", *leaves], got, want):
        assert a.dtype == b.dtype and a.shape == b.shape, name
        _close(a, b.float().cpu(), name)


@pytest.mark.parametrize("pack", [True, False])
def test_training_step_of_the_model_matches_the_eager_backend(pack):
    """loss.backward() through FlashDebertaV2ForSequenceClassification in train mode on a ragged batch: every parameter's
    gradient against the eager backend (fp32, same weights).  Packed and padded paths."""
    from flashdeberta_b200 import FlashDebertaV2ForSequenceClassification
    torch.manual_seed(3)
    ref = FlashDebertaV2ForSequenceClassification(_small_config("eager", num_labels=3)).to(DEV).float().train()
    cfg = _small_config("b200", num_labels=3)
    cfg.pack_sequences = pack
    fused = FlashDebertaV2ForSequenceClassification(cfg).to(DEV)
    fused.load_state_dict(ref.state_dict())
    fused = fused.bfloat16().train()
    g = torch.Generator().manual_seed(4)
    B, L, lens = 3, 400, (400, 222, 64)
    ids = torch.randint(1, 2000, (B, L), generator=g).to(DEV)
    mask = torch.zeros(B, L, device=DEV)
    for b, n in enumerate(lens):
        mask[b, :n] = 1
    labels = torch.tensor([0, 2, 1], device=DEV)
    loss_ref = ref(input_ids=ids, attention_mask=mask, labels=labels).loss
    loss_ref.backward()
    loss = fused(input_ids=ids, attention_mask=mask, labels=labels).loss
    loss.backward()
    torch.cuda.synchronize()
    assert abs(loss.item() - loss_ref.item()) < 5e-2
    checked = 0
    for (name, p_ref), (name2, p) in zip(ref.named_parameters(), fused.named_parameters()):
        assert name == name2
        if p_ref.grad is None:
            assert p.grad is None or p.grad.abs().max().item() == 0, name
            continue
        assert p.grad is not None, name
        scale = p_ref.grad.abs().max().item()
        if scale < 1e-6:
            continue
        diff = (p.grad.float() - p_ref.grad).abs()
        # whole bf16 model against an fp32 one: bf16 weights, activations and GEMMs on top of the attention itself
        assert diff.max().item() <= 0.15 * scale, (name, diff.max().item() / scale)
        assert diff.mean().item() <= 0.02 * scale, (name, diff.mean().item() / scale)
        checked += 1
    assert checked > 20
    attn = fused.deberta.encoder.layer[0].attention.self
    assert attn.query_proj.weight.grad.abs().max().item() > 0 and fused.deberta.encoder.rel_embeddings.weight.grad.abs().max().item() > 0


@pytest.mark.parametrize("varlen", [False, True])
def test_module_gradients_like_the_reference_suite(varlen):
    """The reference's backward test (tests/backward.py:66-200) on this module: 8 heads, 32 buckets / 64 positions, separate
    position projections, fixed-length and right-padded batches; gradients of the input, of the relative embeddings and
    of every parameter against transformers' module in fp32 (the reference compares in fp16 with atol = rtol = 5e-3; the
    bf16 module is held to 3e-2 of each gradient's largest entry)."""
    from transformers.models.deberta_v2.modeling_deberta_v2 import DisentangledSelfAttention
    from flashdeberta_b200 import FlashDisentangledSelfAttention

    class Cfg:
        hidden_size, num_attention_heads = 512, 8
        attention_probs_dropout_prob = hidden_dropout_prob = 0.0
        pos_att_type, relative_attention = ["c2p", "p2c"], True
        position_buckets, max_relative_positions, max_position_embeddings, share_att_key = 32, 64, 512, False

    torch.manual_seed(0)
    eager = DisentangledSelfAttention(Cfg()).to(DEV).eval()
    with torch.no_grad():
        for p in eager.parameters():
            p.copy_(p.bfloat16().float())
    flash = FlashDisentangledSelfAttention(Cfg()).to(DEV).eval()
    flash.load_state_dict(eager.state_dict())
    flash = flash.bfloat16()
    g = torch.Generator().manual_seed(1)
    B, L = 3, 384
    hs = torch.randn(B, L, 512, generator=g).bfloat16().float().to(DEV)
    rel = torch.randn(64, 512, generator=g).bfloat16().float().to(DEV)
    mask = torch.ones(B, L, device=DEV)
    if varlen:
        for b, n in enumerate((384, 201, 17)):
            mask[b, n:] = 0
    ext = mask.unsqueeze(1).unsqueeze(2)
    ext = ext * ext.squeeze(-2).unsqueeze(-1)
    grad_out = torch.randn(B, L, 512, generator=g).to(DEV) * mask.unsqueeze(-1)

    hs_a, rel_a = hs.clone().requires_grad_(True), rel.clone().requires_grad_(True)
    (eager(hs_a, ext, rel_embeddings=rel_a)[0] * grad_out).sum().backward()
    hs_b, rel_b = hs.bfloat16().requires_grad_(True), rel.bfloat16().requires_grad_(True)
    (flash(hs_b, mask, rel_embeddings=rel_b)[0].float() * grad_out).sum().backward()
    torch.cuda.synchronize()

    def check(name, got, want):
        scale = want.abs().max().item()
        diff = (got.float() - want).abs().max().item()
        # the reference's own criterion has the same absolute floor (tests/backward.py:52-54): pos_key_proj.bias shifts
        # every score of a row alike, its true gradient is zero and what is compared there is rounding noise
        assert diff <= 3e-2 * scale or diff <= 5e-3, (name, diff, scale)

    check("hidden_states", hs_b.grad, hs_a.grad)
    check("rel_embeddings", rel_b.grad, rel_a.grad)
    n_checked = 0
    for (name, pa), (_, pb) in zip(eager.named_parameters(), flash.named_parameters()):
        if pa.grad is None:
            continue
        assert pb.grad is not None, name
        check(name, pb.grad, pa.grad)
        n_checked += 1
    assert n_checked >= 8  # q, k, v and the two position projections, weights and biases


def test_backward_through_the_compiled_module():
    """The attention module traced as one graph (forward op and backward op both opaque nodes) gives the eager-mode
    gradients of the same module."""
    from flashdeberta_b200 import FlashDisentangledSelfAttention
    cfg = _small_config("b200")
    torch.manual_seed(5)
    mod = FlashDisentangledSelfAttention(cfg).to(DEV).bfloat16().train()
    g = torch.Generator().manual_seed(6)
    x = torch.randn(2, 256, 256, generator=g).bfloat16().to(DEV)
    rel = torch.randn(512, 256, generator=g).bfloat16().to(DEV)
    mask = torch.ones(2, 256, device=DEV)
    mask[1, 200:] = 0

    def grads(fn):
        xs = x.clone().requires_grad_(True)
        mod.zero_grad()
        out = fn(xs, mask, rel_embeddings=rel)[0]
        out.float().square().sum().backward()
        return xs.grad.clone(), mod.query_proj.weight.grad.clone()

    eager = grads(mod)
    compiled = grads(torch.compile(mod, fullgraph=True, backend="aot_eager"))
    for a, b in zip(eager, compiled):  # same kernels; the p2c sums add in shared memory in no fixed order
        assert (a.float() - b.float()).abs().max().item() <= 1e-2 * b.float().abs().max().item()


def test_fp8_attention_refuses_to_train():
    from flashdeberta_b200 import ops
    q = torch.randn(1, 128, 2, 64, device=DEV).bfloat16().requires_grad_(True)
    with pytest.raises(RuntimeError, match="forward-only"):
        ops.disentangled_attention_fp8(q, q, q, None, None, max_seqlen=128)


@pytest.mark.parametrize("x_width,rel_width,weight", [(320, 256, None), (192, 256, None), (256, 320, None), (256, 128, None),
                                                      (256, 256, (256, 320)), (256, 256, (192, 256)), (256, 256, (320, 256))])
def test_module_in_training_refuses_widths_that_do_not_fit(x_width, rel_width, weight):
    """Sizes that the projections do not have are an error, not a read beyond the weights: the fused node hands on addresses alone."""
    from flashdeberta_b200 import projected
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    module = FlashDisentangledSelfAttention(_small_config("b200")).to(DEV).bfloat16().train()
    if weight is not None:
        module.key_proj.weight = torch.nn.Parameter(torch.randn(*weight, device=DEV).bfloat16())
    x = torch.randn(2, 100, x_width, device=DEV).bfloat16().requires_grad_(True)
    rel = torch.randn(512, rel_width, device=DEV).bfloat16()
    assert not projected.covers(module, x, None, None, rel)
    with pytest.raises((RuntimeError, ValueError)):
        module(x, None, rel_embeddings=rel)


def test_module_in_training_takes_only_masks_that_fit():
    from flashdeberta_b200 import projected
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    module = FlashDisentangledSelfAttention(_small_config("b200")).to(DEV).bfloat16().train()
    x = torch.randn(2, 100, 256, device=DEV).bfloat16().requires_grad_(True)
    rel = torch.randn(512, 256, device=DEV).bfloat16()
    covered = lambda mask: projected.covers(module, x, None, mask, rel)
    assert covered(torch.ones(2, 100, device=DEV)) and covered(torch.full((2,), 100, device=DEV))
    assert not any(covered(m) for m in (torch.ones(2, 100), torch.ones(1, 100, device=DEV), torch.ones(2, 99, device=DEV), torch.ones(1, device=DEV)))


def test_lengths_on_the_host():
    """Lengths, offsets and masks on the host are brought to the device; too few lengths are an error."""
    from flashdeberta_b200 import backward, ops
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    g = torch.Generator().manual_seed(8)
    q, k, v, dout = (torch.randn(2, 200, 2, 64, generator=g).bfloat16().to(DEV) for _ in range(4))
    pk, pq = (torch.randn(2, 64, 64, generator=g).bfloat16().to(DEV) for _ in range(2))
    kw = dict(max_seqlen=200, position_buckets=32, max_relative_positions=64)
    lens, cu = torch.tensor([200, 77], dtype=torch.int32), torch.tensor([0, 200, 377])

    def both(call, t):
        want, got = call(t.to(DEV)), call(t)
        assert all(torch.equal(a, b) for a, b in zip(want, got))

    flat = lambda t: t.reshape(-1, 2, 64)[:377]
    both(lambda n: _run_op(q, k, v, pk, pq, dout, seq_lens=n, **kw), lens)
    both(lambda n: _run_op(flat(q), flat(k), flat(v), pk, pq, flat(dout), cu_seqlens=n, **kw), cu)
    with torch.no_grad():
        both(lambda n: [ops.disentangled_attention_fp8(q, k, v, pk, pq, seq_lens=n, **kw)], lens)
        out, lse = ops.disentangled_attention(q, k, v, pk, pq, seq_lens=lens, return_lse=True, **kw)
        both(lambda n: backward.attention_backward(dout, q, k, v, pk, pq, out, lse, seq_lens=n, sm_scale=0.07, block_bytes=1 << 28, **kw), lens)
        with pytest.raises(ValueError):
            ops.disentangled_attention(q, k, v, pk, pq, seq_lens=lens[:1], **kw)
    module = FlashDisentangledSelfAttention(_small_config("b200")).to(DEV).bfloat16().train()
    x, rel = torch.randn(2, 200, 256, device=DEV).bfloat16().requires_grad_(True), torch.randn(512, 256, device=DEV).bfloat16()
    mask = (torch.arange(200)[None] < lens[:, None]).long()
    got = torch.autograd.grad(module(x, mask, rel_embeddings=rel)[0].sum(), x)[0]
    _close(got, torch.autograd.grad(module(x, mask.to(DEV), rel_embeddings=rel)[0].sum(), x)[0].float().cpu(), "host mask")
    ops.check_status()


@pytest.mark.parametrize("form", ["offset", "transposed", "expanded rows", "expanded"])
def test_gradients_that_start_or_stride_anywhere(form):
    """The gradient of the output as autograd or a caller may hand it over: a slice that starts at an odd element, heads outermost,
    one row for all, one number for all."""
    from flashdeberta_b200 import backward, ops
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    g = torch.Generator().manual_seed(9)
    make = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)

    def grad(*shape):
        n = shape.numel() if isinstance(shape, torch.Size) else torch.Size(shape).numel()
        if form == "offset":
            return make(n + 3)[3:].view(shape)
        if form == "transposed":
            return make(*shape[::-1]).permute(*range(len(shape) - 1, -1, -1))
        return make(1, 1, *shape[2:]).expand(shape) if form == "expanded rows" else make(1).expand(shape)

    q, k, v = (make(2, 150, 2, 64) for _ in range(3))
    pk, pq = make(2, 64, 64), make(2, 64, 64)
    kw = dict(max_seqlen=150, position_buckets=32, max_relative_positions=64)
    dout = grad(2, 150, 2, 64)
    want = _run_op(q, k, v, pk, pq, dout.clone(memory_format=torch.contiguous_format), **kw)
    for a, b in zip(_run_op(q, k, v, pk, pq, dout, **kw), want):
        assert torch.equal(a, b)
    with torch.no_grad():  # and the function itself, with every tensor off its boundary
        out, lse = ops.disentangled_attention(q, k, v, pk, pq, return_lse=True, **kw)
        odd = lambda t: torch.cat((t.new_zeros(3), t.flatten()))[3:].view(t.shape)
        got = backward.attention_backward(dout, *(odd(t) for t in (q, k, v, pk, pq, out)), odd(lse), sm_scale=1 / (64 * 3) ** 0.5, **kw)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    module = FlashDisentangledSelfAttention(_small_config("b200")).to(DEV).bfloat16().train()
    x, rel, dout = make(2, 150, 256).requires_grad_(True), make(512, 256), grad(2, 150, 256)
    run = lambda d: torch.autograd.grad(module(x, None, rel_embeddings=rel)[0], [x, *module.parameters()], d)
    for a, b in zip(run(dout), run(dout.clone(memory_format=torch.contiguous_format))):
        assert torch.equal(a, b)
    ops.check_status()


@pytest.mark.parametrize("rows", [0, 1, 300])
@pytest.mark.parametrize("terms", [True, False])
def test_no_sequence_gives_zero_gradients(rows, terms):
    """Offsets that name no sequence: every row is outside, every gradient zero whatever the memory held before.  (The library's entry
    point is called itself for no rows at all, which the Python side answers alone.)"""
    import ctypes as C
    from flashdeberta_b200 import _lib, backward, ops
    g = torch.Generator().manual_seed(9)
    q, k, v, out, dout = (torch.randn(max(rows, 1), 2, 64, generator=g).bfloat16().to(DEV)[:rows] for _ in range(5))
    pk, pq = (torch.randn(2, 64, 64, generator=g).bfloat16().to(DEV) for _ in range(2)) if terms else (None, None)
    cu = torch.zeros(1, dtype=torch.int32, device=DEV)
    kw = dict(cu_seqlens=cu, max_seqlen=128, sm_scale=0.1, position_buckets=32, max_relative_positions=64)
    for _ in range(2):
        junk = [torch.full((n,), float("nan"), dtype=torch.bfloat16, device=DEV) for n in (rows * 128, 8192, 64 * 128, 1 << 20) for _ in range(4)]
        del junk
        got = backward.attention_backward(dout, q, k, v, pk, pq, out, torch.zeros(rows, 2, device=DEV), **kw)
        for t, like in zip(got, (q, k, v, pk, pq)):
            assert (t is None) == (like is None) and (t is None or (t.shape == like.shape and torch.count_nonzero(t) == 0))
    if rows == 0 and terms:
        d = torch.full((2, 2, 64, 64), float("nan"), dtype=torch.bfloat16, device=DEV)
        one = torch.zeros(1, 2, 64, dtype=torch.bfloat16, device=DEV)
        p, keep = ops._fill_params(one, one, one, pk, pq, cu, None, 128, 0.1, 32, 64, one, torch.zeros(1, 2, device=DEV))
        p.total_rows = 0
        b = backward.BwdParams()
        b.struct_bytes, b.fwd, b.dpos_key, b.dpos_query = C.sizeof(b), C.pointer(p), d[0].data_ptr(), d[1].data_ptr()
        _lib.check(_lib.load().fdb_attn_bwd(C.byref(b), C.c_void_p(ops.raw_stream(q.device))))
        assert torch.count_nonzero(d) == 0
    ops.check_status()


def test_heads_in_groups_give_the_same_gradients():
    """More bucket sums than the workspace holds at a time: three heads of 720000 rows go in a group of two and one.  Against the heads
    by themselves (one group each): equal but for the order in which the tables' gradients are summed."""
    from flashdeberta_b200 import backward, ops
    g = torch.Generator(device=DEV).manual_seed(9)
    n, H, L = 5625, 3, 128
    make = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.bfloat16)
    q, k, v, dout = (make(n * L + 7, H, 64) for _ in range(4))
    pk, pq = make(H, 512, 64), make(H, 512, 64)
    cu = torch.arange(0, n * L + 1, L, dtype=torch.int32, device=DEV) + 3  # rows outside on both ends
    kw = dict(cu_seqlens=cu, max_seqlen=L, sm_scale=0.07, position_buckets=256, max_relative_positions=512)
    with torch.no_grad():
        out, lse = ops.disentangled_attention(q, k, v, pk, pq, return_lse=True, **kw)
    got = backward.attention_backward(dout, q, k, v, pk, pq, out, lse, **kw)
    for h in range(H):
        one = lambda t: t[:, h:h + 1]
        want = backward.attention_backward(one(dout), one(q), one(k), one(v), pk[h:h + 1], pq[h:h + 1], one(out), one(lse), **kw)
        for a, b in zip(got[:3], want[:3]):
            assert torch.equal(one(a), b)
        for a, b in zip(got[3:], want[3:]):  # fp32 sums in two orders, then rounded: one bf16 step where they fall on either side
            assert ((a[h:h + 1].float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 1e-4 * b.float().abs().max()).all()
    ops.check_status()

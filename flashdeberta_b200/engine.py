"""Inference of the whole encoder through one call into libfdb_b200.so (``fdb_encoder_forward``).

The modules of model.py stay the interface and the owner of every parameter; this walks them once, hands their addresses to
the library, and from then on a forward of the backbone is one C call instead of a dozen torch operators per layer
(src/flashdeberta/model.py:275-310 of the reference is the module walk it stands for).  What it relies on is looked
at again on every call — parameters replaced or moved, modules swapped, the modules' own settings, hooks, training mode — and
whatever it does not cover goes through the modules as before.  As in the modules' caches, a parameter counts as unchanged while its
address and version counter are: a write that bypasses the counter (through ``.data``, a raw kernel) to one behind the position
tables is not seen.
"""
from __future__ import annotations

import ctypes as C
import math
import threading
from typing import Optional

import torch
from torch import nn

from . import _lib, bucket, ops


class EncoderLayer(C.Structure):
    """Mirror of ``fdb_encoder_layer`` (include/fdb_b200.h)."""

    _fields_ = [(n, C.c_void_p) for n in (
        "wq", "bq", "wk", "bk", "wv", "bv", "wo", "bo", "ln1_gamma", "ln1_beta", "wi", "bi", "wd", "bd", "ln2_gamma",
        "ln2_beta", "exp_key", "exp_query")] + [("ln1_eps", C.c_float), ("ln2_eps", C.c_float)]


class EncoderCall(C.Structure):
    """Mirror of ``fdb_encoder_call`` (include/fdb_b200.h)."""

    _fields_ = [
        ("struct_bytes", C.c_uint32), ("mask_type", C.c_int32), ("plan", C.c_void_p), ("ids", C.c_void_p), ("mask", C.c_void_p),
        ("cu_seqlens", C.c_void_p), ("batch", C.c_int32), ("max_seqlen", C.c_int32), ("total_rows", C.c_int32),
        ("position_buckets", C.c_int32), ("max_relative_positions", C.c_int32), ("lut_d_min", C.c_int32), ("lut_len", C.c_int32),
        ("lut", C.c_void_p), ("sm_scale", C.c_float), ("emb_eps", C.c_float), ("emb_table", C.c_void_p), ("emb_gamma", C.c_void_p),
        ("emb_beta", C.c_void_p), ("emb_rows", C.c_int64), ("out", C.c_void_p), ("workspace", C.c_void_p),
        ("workspace_bytes", C.c_uint64), ("status", C.c_void_p), ("attn_events", C.c_void_p), ("launches", C.c_int32),
    ]


#: settings of the modules that a plan copies or that decide whether it covers the model
_SETTINGS = ("attn_fp8", "num_attention_heads", "attention_head_size", "pos_att_type", "relative_attention", "position_buckets",
             "max_relative_positions", "pos_ebd_size", "share_att_key", "eps", "_erf_gelu", "norm_rel_ebd", "max_norm", "position_biased_input")


class _Tables:
    """The projected position tables of every layer, gathered through the bucket index.  The lock covers everything but ``data``: a
    thread that finds ``versions`` up to date also finds the event that its stream has to wait for."""

    def __init__(self, shape, device, params):
        self.params = params             # held, so that nothing else gets their identities
        with ops.on_device(device):
            self.data = torch.empty(shape, dtype=torch.bfloat16, device=device)
            self.streams = {ops.raw_stream(device)}  # those that the allocator knows to read `data`
        self.captured = False            # a graph may read `data`
        self.lock = threading.Lock()
        self.versions = None             # of the parameters that `data` was gathered from
        self.stream = self.event = None  # the stream it was gathered on; the end of it, until that is known to be reached


class _Plan:
    """What one walk over the model found: the library's plan, the objects it was made from (to notice a change) and the
    position tables gathered for every layer."""

    def __init__(self, model, kept=()):
        """``kept``: (key, tables) to take over where they are of the same parameters."""
        from .attention import FlashDisentangledSelfAttention
        from . import model as M
        enc, emb, cfg = model.encoder, model.embeddings, model.config
        modules = [enc, *(m for m in enc.modules() if m is not enc), *emb.modules()]
        self.ok = False
        self.handle, self.destroy = C.c_void_p(None), _lib.load().fdb_encoder_destroy
        self.module_dicts = [m._modules for m in modules]
        self.param_dicts = [m._parameters for m in modules if m._parameters]
        self.hooks = [h for m in modules for h in (m._forward_hooks, m._forward_pre_hooks)]
        self.attrs = [m.__dict__ for m in modules]
        self.module_ids = [id(v) for d in self.module_dicts for v in d.values()]
        self.params = [v for d in self.param_dicts for v in d.values() if v is not None]
        self.param_ids = [id(v) for d in self.param_dicts for v in d.values()]
        self.addresses = [p.data_ptr() for p in self.params]
        self.owner = (enc, emb)
        self.keep = modules
        self.setting_of = [(d, name) for d in self.attrs for name in _SETTINGS if name in d]
        self.settings = [list(v) if isinstance(v, list) else v for v in (d[name] for d, name in self.setting_of)]  # (lists may be written to)
        if type(enc) is not M.FlashDebertaV2Encoder or enc.conv is not None or not enc.relative_attention or len(enc.layer) == 0 or type(emb) is not M.FlashDebertaV2Embeddings:
            return
        if emb.position_embeddings is not None or emb.position_biased_input or emb.token_type_embeddings is not None or emb.embed_proj is not None:
            return
        if not self.params or any(type(p) is not nn.Parameter for p in self.params):
            return  # (a subclass keeps its values elsewhere than where it points)
        hidden, heads = cfg.hidden_size, cfg.num_attention_heads
        ffn = enc.layer[0].intermediate.dense.out_features
        device = self.params[0].device
        if hidden != heads * 64 or hidden % 256 or hidden > 2048 or ffn % 64 or device.type != "cuda":
            return
        if any(p.dtype != torch.bfloat16 or p.device != device or not p.is_contiguous() or p.data_ptr() % 16 for p in self.params):
            return

        def own(m, *names):
            """Whether these tensors are the module's registered parameters: only those are compared from call to call (sharding
            wrappers and replicas set others, and set them anew)."""
            return all(n in m._parameters and n not in m.__dict__ for n in names)

        def linear(m, n, k):
            return type(m) is nn.Linear and m.out_features == n and m.in_features == k and own(m, "weight", "bias") and m.weight is not None

        def norm(m):
            return (type(m) is nn.LayerNorm and m.elementwise_affine and own(m, "weight", "bias") and m.bias is not None
                    and m.normalized_shape == (hidden,))

        if (not norm(emb.LayerNorm) or type(emb.word_embeddings) is not nn.Embedding or not own(emb.word_embeddings, "weight")
                or emb.word_embeddings.max_norm is not None):
            return
        if type(enc.rel_embeddings) is not nn.Embedding or not own(enc.rel_embeddings, "weight"):
            return
        if "layer_norm" in enc.norm_rel_ebd and not own(enc.LayerNorm, "weight", "bias"):
            return
        attn0 = enc.layer[0].attention.self
        for layer in enc.layer:
            a = layer.attention.self
            if (type(layer) is not M.FlashDebertaV2Layer or type(layer.attention) is not M.FlashDebertaV2Attention
                    or type(a) is not FlashDisentangledSelfAttention or a.attn_fp8 or a.attention_head_size != 64
                    or a.num_attention_heads != heads or a.pos_att_type != attn0.pos_att_type or not a.relative_attention
                    or (a.position_buckets, a.max_relative_positions) != (attn0.position_buckets, attn0.max_relative_positions)
                    or type(layer.attention.output) is not M.FlashDebertaV2SelfOutput or type(layer.output) is not M.FlashDebertaV2Output
                    or type(layer.intermediate) is not M.FlashDebertaV2Intermediate or not layer.intermediate._erf_gelu):
                return
            if not (all(linear(m, hidden, hidden) for m in (a.query_proj, a.key_proj, a.value_proj, layer.attention.output.dense))
                    and linear(layer.intermediate.dense, ffn, hidden) and linear(layer.output.dense, hidden, ffn)
                    and norm(layer.attention.output.LayerNorm) and norm(layer.output.LayerNorm)):
                return
            if not a.share_att_key and not all(type(m) is nn.Linear and own(m, "weight", "bias")
                                               for m in (getattr(a, n, None) for n in ("pos_key_proj", "pos_query_proj")) if m is not None):
                return
        self.device, self.hidden, self.heads = device, hidden, heads
        self.c2p, self.p2c = "c2p" in attn0.pos_att_type, "p2c" in attn0.pos_att_type
        self.sm_scale = 1.0 / math.sqrt(64 * (1 + int(self.c2p) + int(self.p2c)))
        self.buckets, self.max_rel = attn0.position_buckets, attn0.max_relative_positions
        self.attention = [layer.attention.self for layer in enc.layer]
        # the parameters that the gathered tables depend on
        table_params = [enc.rel_embeddings.weight, *(enc.LayerNorm.parameters() if "layer_norm" in enc.norm_rel_ebd else ())]
        for a in self.attention:
            names = ("key_proj", "query_proj") if a.share_att_key else ("pos_key_proj", "pos_query_proj")
            for name in names:
                m = getattr(a, name, None)
                if m is not None:
                    table_params += list(m.parameters())
        self.table_params = [p for p in table_params if not p.is_inference()]  # (those have no version counter)
        self.lut, self.d_min, self.tables = None, 0, None
        if self.c2p or self.p2c:
            self.lut, self.d_min = bucket.device_lut(self.buckets, self.max_rel, device)
            rows = _lib.load().fdb_expanded_rows(self.d_min, self.lut.numel())
            shape = (len(enc.layer), 2, heads, rows, 64)
            self.table_key = (device, shape, self.c2p, self.p2c, self.buckets, self.max_rel, getattr(enc, "LayerNorm", enc).__dict__.get("eps"), [(id(p), p.data_ptr()) for p in table_params])
            self.tables = next((t for key, t in kept if key == self.table_key), None) or _Tables(shape, device, table_params)
        self._create(enc)

    def _create(self, enc):
        n = len(enc.layer)
        descs = (EncoderLayer * n)()
        ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
        for i, layer in enumerate(enc.layer):
            a, o, d = layer.attention.self, layer.attention.output, descs[i]
            for name, m in (("q", a.query_proj), ("k", a.key_proj), ("v", a.value_proj), ("o", o.dense), ("i", layer.intermediate.dense),
                            ("d", layer.output.dense)):
                setattr(d, "w" + name, ptr(m.weight))
                setattr(d, "b" + name, ptr(m.bias))
            d.ln1_gamma, d.ln1_beta, d.ln1_eps = ptr(o.LayerNorm.weight), ptr(o.LayerNorm.bias), o.LayerNorm.eps
            d.ln2_gamma, d.ln2_beta, d.ln2_eps = ptr(layer.output.LayerNorm.weight), ptr(layer.output.LayerNorm.bias), layer.output.LayerNorm.eps
            d.exp_key = ptr(self.tables.data[i, 0]) if self.c2p else None
            d.exp_query = ptr(self.tables.data[i, 1]) if self.p2c else None
        ffn = enc.layer[0].intermediate.dense.out_features
        with ops.on_device(self.device):
            rc = _lib.load().fdb_encoder_create(C.byref(descs), n, self.hidden, self.heads, ffn, C.byref(self.handle))
        self.ok = rc == _lib.FDB_OK

    def __del__(self):
        if self.handle:
            self.destroy(self.handle)
            self.handle = None

    def current(self, model) -> bool:
        """Whether the model still is the one this plan was made from: same modules and settings, same parameters at the same
        addresses."""
        return (model.encoder is self.owner[0] and model.embeddings is self.owner[1]
                and [d.get(name) for d, name in self.setting_of] == self.settings
                and [id(v) for d in self.module_dicts for v in d.values()] == self.module_ids
                and [id(v) for d in self.param_dicts for v in d.values()] == self.param_ids
                and [p.data_ptr() for p in self.params] == self.addresses)

    def plain(self) -> bool:
        """No hooks, no module in training mode, no patched ``forward``: nothing a module walk would do beside the arithmetic."""
        return not any(self.hooks) and not ops.global_module_hooks() and not any([d["training"] or "forward" in d for d in self.attrs])

    def versions(self):
        """What the gathered tables depend on, as it is now."""
        return [p._version for p in self.table_params]

    def gather(self, encoder, stream) -> int:
        """Gathers the projected position tables of every layer, from the parameters alone: what the modules keep of them may be on
        its way on another stream.  Returns the kernels launched."""
        lib = _lib.load()
        rel = encoder.get_rel_embedding(keep=False)
        for i, a in enumerate(self.attention):
            pos_key, pos_query = a._position_tables(rel, torch.bfloat16, keep=False)
            any_table = pos_key if pos_key is not None else pos_query
            _lib.check(lib.fdb_expand_tables(
                pos_key.data_ptr() if self.c2p else None, pos_query.data_ptr() if self.p2c else None,
                self.tables.data[i, 0].data_ptr() if self.c2p else None, self.tables.data[i, 1].data_ptr() if self.p2c else None,
                self.heads, any_table.shape[1], self.lut.data_ptr(), self.d_min, self.lut.numel(), C.c_void_p(stream)))
        return len(self.attention)

    def refresh_tables(self, encoder, stream, device) -> int:
        """Gathers the tables again when a parameter behind them was written to, and lets this stream wait for a gathering on another
        one, until that is known to be over.  Returns the kernels launched."""
        t, launched = self.tables, 0
        if t is None:
            return 0
        versions = self.versions()
        with t.lock:
            if t.versions != versions:
                t.versions = None  # should anything below fail
                launched = self.gather(encoder, stream)
                event = torch.cuda.Event()
                event.record()
                t.versions, t.stream, t.event = versions, stream, event
            elif t.event is not None:
                if t.event.query():
                    t.event = None
                elif stream != t.stream:
                    torch.cuda.current_stream(device).wait_event(t.event)
            if stream not in t.streams:  # once freed, the memory may be another tensor's only behind this stream's calls
                t.data.record_stream(torch.cuda.current_stream(device))
                t.streams.add(stream)
        return launched


class EncoderEngine:
    """One per model; holds the plan of the model as it is now.  Copies and pickles of a model get an empty one."""

    def __init__(self):
        self.plan: Optional[_Plan] = None
        self.kept = []  # (key, tables) that graphs captured with earlier plans of the same weights read

    def _replace_plan(self, model) -> _Plan:
        """A plan of the model as it is now.  Tables that a captured graph reads stay until the weights, which it reads too, are
        others; a plan of the same parameters and bucket table takes its predecessor's over."""
        old, kept = self.plan, self.kept
        if old is not None and old.tables is not None:
            kept = kept + [(old.table_key, old.tables)]
        plan = _Plan(model, kept)
        same = old is not None and plan.addresses == old.addresses
        self.plan, self.kept = plan, [(key, t) for key, t in kept if same and t.captured and t is not plan.tables]
        return plan

    def __deepcopy__(self, memo):
        return EncoderEngine()

    def __reduce__(self):
        return (EncoderEngine, ())

    def forward(self, model, ids: torch.Tensor, mask: Optional[torch.Tensor], cu_seqlens: Optional[torch.Tensor],
                max_seqlen: int) -> Optional[torch.Tensor]:
        """Last hidden state of (B, L) ids with an optional (B, L) mask, or of (1, T) packed ids with ``cu_seqlens``.  None
        when the model or the call is not covered."""
        plan, capturing = self.plan, ops.capturing(ids)
        # What a captured call launches has not run when the call returns, so nothing that it sets up may be taken for done by
        # another call: where the plan or its tables are not up to date, a captured call makes its own, and its graph gathers
        # the tables whenever it is replayed.
        own = capturing and (plan is None or not plan.current(model) or (plan.ok and plan.tables is not None and plan.versions() != plan.tables.versions))
        if own:
            plan = _Plan(model)
        elif plan is None or not plan.current(model):
            plan = self._replace_plan(model)
        if not plan.ok or ids.device != plan.device or not plan.plain():
            return None
        device = plan.device
        lib = _lib.load()
        if ids.dtype != torch.int64 or not ids.is_contiguous():
            ids = ids.to(torch.int64).contiguous()
        p = EncoderCall()
        p.struct_bytes = C.sizeof(EncoderCall)
        p.plan = plan.handle
        p.ids = ids.data_ptr()
        if mask is not None:
            if mask.device != device:
                mask = mask.to(device, non_blocking=True)
            if mask.dtype not in ops.MASK_TYPES:
                mask = mask.to(torch.float32)
            mask = mask.contiguous()
            p.mask, p.mask_type = mask.data_ptr(), ops.MASK_TYPES[mask.dtype]
        if cu_seqlens is not None:
            p.cu_seqlens, p.batch = cu_seqlens.data_ptr(), cu_seqlens.numel() - 1
        else:
            p.batch = ids.shape[0]
        p.max_seqlen, p.total_rows = max_seqlen, ids.numel()
        p.position_buckets, p.max_relative_positions = plan.buckets, plan.max_rel
        if plan.lut is not None:
            p.lut, p.lut_d_min, p.lut_len = plan.lut.data_ptr(), plan.d_min, plan.lut.numel()
        emb = model.embeddings
        p.sm_scale, p.emb_eps = plan.sm_scale, emb.LayerNorm.eps
        table = emb.word_embeddings.weight
        p.emb_table, p.emb_rows = table.data_ptr(), table.shape[0]
        p.emb_gamma, p.emb_beta = emb.LayerNorm.weight.data_ptr(), emb.LayerNorm.bias.data_ptr()
        out = torch.empty(*ids.shape, plan.hidden, dtype=torch.bfloat16, device=device)
        p.out = out.data_ptr()
        p.status = ops._status_word(device).data_ptr()
        with ops.on_device(device):
            stream = ops.raw_stream(device)
            if own and plan.tables is not None:
                ops._launches += plan.gather(model.encoder, stream)
            elif not capturing:  # (a capture cannot wait for work outside it, and need not: it begins with a synchronisation)
                ops._launches += plan.refresh_tables(model.encoder, stream, device)
            elif plan.tables is not None:
                plan.tables.captured = True
            need = lib.fdb_encoder_workspace_bytes(C.byref(p))
            ws = torch.empty(need + 256, dtype=torch.uint8, device=device)
            p.workspace, p.workspace_bytes = (ws.data_ptr() + 255) & ~255, need
            events = None
            if ops.event_log is not None:
                events = [torch.cuda.Event(enable_timing=True) for _ in range(2 * len(plan.attention))]
                for e in events:
                    e.record()  # creates it
                handles = (C.c_void_p * len(events))(*[e.cuda_event for e in events])
                p.attn_events = C.cast(handles, C.c_void_p)
            _lib.check(lib.fdb_encoder_forward(C.byref(p), C.c_void_p(stream)))
            if events is not None:
                ops.event_log += list(zip(events[0::2], events[1::2]))
        ops._launches += p.launches
        return out

"""Training of the attention module as one autograd node: projections, position tables and attention.

Operator by operator the module's forward and backward are some forty autograd nodes and a hundred launches, which cost the host
more than the GPU needs for a batch of paragraphs.  Here the forward is one call into the library (``fdb_projected_forward``: the
three projections, the position tables through the same weights, the attention), and the backward is ``fdb_attn_bwd`` in the
projections' buffers with one GEMM each for the input and the weights, and one pass for the biases.

What it does not cover goes through the modules as before: see ``covers``.
"""
from __future__ import annotations

import ctypes as C
import math

import torch
from torch import nn

from . import _lib, backward, bucket, ops

def _plain_linear(m, w, b, device, n: int, k: int) -> bool:
    return (b is not None and w.shape == (n, k) and b.shape == (n,) and w.dtype == torch.bfloat16 and b.dtype == torch.bfloat16
            and w.device == device and b.device == device and w.is_contiguous() and (w.data_ptr() | b.data_ptr()) % 16 == 0
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks) and "forward" not in m.__dict__)


def covers(module, x, query_states, mask, rel):
    """The projections' weights and biases, [wq, bq, wk, bk, wv, bv], when a call is one that ``attention`` stands for: autograd recording, bf16 on the GPU, both position terms through the
    key and query projections themselves, self-attention over a dense batch, nothing between the operators (dropout, hooks,
    autocast, tracing); else False."""
    if torch.is_autocast_enabled("cuda") or ops.global_module_hooks():
        return False
    if not (torch.is_grad_enabled() and x.is_cuda and x.dtype == torch.bfloat16 and module.share_att_key
            and module.relative_attention and not module.attn_fp8 and module.attention_head_size == 64):
        return False
    if query_states is not None and query_states is not x:
        return False
    if rel is None or rel.dim() != 2 or rel.dtype != torch.bfloat16 or rel.device != x.device or x.numel() == 0:
        return False
    if x.dim() != 3 or rel.shape[1] != x.shape[2]:  # (from here on only addresses are handed on: every size is looked at)
        return False
    linears = (module.query_proj, module.key_proj, module.value_proj)
    if not (type(linears[0]) is type(linears[1]) is type(linears[2]) is nn.Linear):
        return False
    weights = [linears[0].weight, linears[0].bias, linears[1].weight, linears[1].bias, linears[2].weight, linears[2].bias]
    if ops.intercepted(x, rel, mask, *weights):
        return False
    if (x.data_ptr() | rel.data_ptr()) % 16:
        return False
    if "c2p" not in module.pos_att_type or "p2c" not in module.pos_att_type or not (mask is None or isinstance(mask, torch.Tensor)):
        return False
    if mask is not None and (mask.device != x.device or mask.dim() == 0 or mask.shape[0] != x.shape[0] or (mask.dim() > 1 and mask.shape[-1] != x.shape[1])):
        return False
    drop = module.pos_dropout
    if (drop.training and drop.p > 0) or drop._forward_hooks or drop._forward_pre_hooks:
        return False
    n, k, device = module.num_attention_heads * 64, x.shape[2], x.device
    if k % 64 or not all([_plain_linear(linears[i], weights[2 * i], weights[2 * i + 1], device, n, k) for i in range(3)]):
        return False
    if rel.shape[0] < 2 * module.pos_ebd_size or not backward.index_covered(module.position_buckets, module.max_relative_positions):
        return False
    return weights if ops.wants_grad(x, rel, *weights) else False


class _ProjectedParams(C.Structure):
    """Mirror of ``fdb_projected_params`` (include/fdb_b200.h)."""

    _fields_ = [("struct_bytes", C.c_uint32), ("in_features", C.c_int32), ("attn", C.POINTER(_lib.AttnParams)),
                ("table_row_stride", C.c_int64), ("table_head_stride", C.c_int64)] + [
        (n, C.c_void_p) for n in ("x", "rel", "wq", "bq", "wk", "bk", "wv", "bv")]


def _params(qkv, tables, out, lse, lens, B, L, heads, buckets, max_rel):
    """The attention call over the projections' buffers: qkv (rows, 3, heads, 64), tables (2*att_span, 2, heads, 64) with the
    queries' projection of the embeddings (the p2c table) first, the keys' (c2p) second."""
    inner = heads * 64
    lut, d_min = bucket.device_lut(buckets, max_rel, qkv.device)
    q, t = qkv.data_ptr(), tables.data_ptr()
    p = _lib.AttnParams(  # in the order of the fields
        C.sizeof(_lib.AttnParams), _lib.FDB_BF16, q, q + 2 * inner, q + 4 * inner, out.data_ptr(), 3 * inner, 64, 3 * inner, 64, 3 * inner, 64,
        inner, 64, t + 2 * inner, t, None, None if lens is None else lens.data_ptr(), B, L, B * L, heads, 64, buckets, max_rel,
        lut.data_ptr(), d_min, lut.shape[0], 1.0 / math.sqrt(64 * 3))
    p.lse, p.status = lse.data_ptr(), ops._status_word(qkv.device).data_ptr()
    return p


class _Projected(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, rel, wq, wk, wv, bq, bk, bv, lens, heads, buckets, max_rel):
        B, L, hidden = x.shape
        dev, inner, span2 = x.device, heads * 64, 2 * bucket.att_span(buckets, max_rel)
        x2, rel2 = x.reshape(B * L, hidden).contiguous(), rel.contiguous()
        qkv = torch.empty(B * L, 3 * inner, dtype=torch.bfloat16, device=dev)
        tables = torch.empty(span2, 2 * inner, dtype=torch.bfloat16, device=dev)
        out = torch.empty(B, L, inner, dtype=torch.bfloat16, device=dev)
        lse = torch.empty(B * L, heads, dtype=torch.float32, device=dev)
        p = _params(qkv, tables, out, lse, lens, B, L, heads, buckets, max_rel)
        lib = _lib.load()
        need = lib.fdb_attn_workspace_bytes(C.byref(p))
        ws = torch.empty(need + 256, dtype=torch.uint8, device=dev)
        p.workspace, p.workspace_bytes = (ws.data_ptr() + 255) & ~255, need
        c = _ProjectedParams(C.sizeof(_ProjectedParams), hidden, C.pointer(p), 2 * inner, 64, x2.data_ptr(), rel2.data_ptr(),
                             *(t.data_ptr() for t in (wq, bq, wk, bk, wv, bv)))
        with ops.on_device(dev):
            _lib.check(lib.fdb_projected_forward(C.byref(c), C.c_void_p(ops.raw_stream(dev))))
        ops._launches += 5
        ctx.save_for_backward(x2, rel2, wq, wk, wv, qkv, tables, out, lse, lens)
        ctx.fdb_args = (B, L, heads, buckets, max_rel)
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, grad):
        x2, rel, wq, wk, wv, qkv, tables, out, lse, lens = ctx.saved_tensors
        B, L, heads, buckets, max_rel = ctx.fdb_args
        inner, span2, dev = heads * 64, tables.shape[0], qkv.device
        operators = ops.intercepted(grad) or ops.batched(grad)
        if operators:
            d_qkv, d_tables = _backward_by_operators(grad, qkv, tables, out, lse, lens, *ctx.fdb_args)
        else:
            grad = grad.contiguous()
            if grad.data_ptr() % 16:
                grad = grad.clone()
            d_qkv, d_tables = torch.empty_like(qkv), torch.empty_like(tables)
            p = _params(qkv, tables, out, lse, lens, B, L, heads, buckets, max_rel)
            d, t = d_qkv.data_ptr(), d_tables.data_ptr()
            b = backward.BwdParams(C.sizeof(backward.BwdParams), 0, C.pointer(p), grad.data_ptr(), inner, 64, d, d + 2 * inner, d + 4 * inner,
                                   3 * inner, 64, t + 2 * inner, t, 2 * inner, 64)
            with ops.on_device(dev):
                backward.launch(b, dev)
        want = ctx.needs_input_grad
        grads = [None] * 8
        if want[0] or want[1]:
            w = torch.cat((wq, wk, wv))
            if want[0]:
                grads[0] = torch.mm(d_qkv, w).view(B, L, -1)
            if want[1]:
                d_rel = torch.mm(d_tables, w[:2 * inner])
                if rel.shape[0] != span2:
                    d_rel = torch.cat((d_rel, d_rel.new_zeros(rel.shape[0] - span2, rel.shape[1])))
                grads[1] = d_rel
        if want[2] or want[3] or want[4]:
            dw = torch.mm(d_qkv.t(), x2)
            if operators:
                dw = torch.cat((dw[:2 * inner] + torch.mm(d_tables.t(), rel[:span2]), dw[2 * inner:]))
            else:
                dw[:2 * inner].addmm_(d_tables.t(), rel[:span2])
            grads[2:5] = [g if n else None for g, n in zip(dw.split(inner), want[2:5])]
        if want[5] or want[6] or want[7]:
            if operators:
                db = d_qkv.sum(0, dtype=torch.float32)
                db = torch.cat((db[:2 * inner] + d_tables.sum(0, dtype=torch.float32), db[2 * inner:])).to(qkv.dtype)
            else:
                db = ops.column_sums(d_qkv, d_tables)
            grads[5:8] = [g if n else None for g, n in zip(db.split(inner), want[5:8])]
        return (*grads, None, None, None, None)


def _backward_by_operators(grad, qkv, tables, out, lse, lens, B, L, heads, buckets, max_rel):
    """Gradients of the projections' buffers through the custom operator, for gradients that have no address (``ops.intercepted``)."""
    inner, span2 = heads * 64, tables.shape[0]
    q, k, v = qkv.view(B, L, 3, heads, 64).unbind(2)
    pos_query, pos_key = (t.transpose(0, 1) for t in tables.view(span2, 2, heads, 64).unbind(1))
    dq, dk, dv, dpk, dpq = ops.attn_bwd_op(
        grad.reshape(B, L, heads, 64), q, k, v, pos_key, pos_query, out.view(B, L, heads, 64), lse, None, lens, L, 1.0 / math.sqrt(64 * 3),
        buckets, max_rel)
    return (torch.stack((dq, dk, dv), 2).reshape(B * L, 3 * inner),
            torch.stack((dpq, dpk), 0).permute(2, 0, 1, 3).reshape(span2, 2 * inner))


def attention(module, x: torch.Tensor, lens, rel: torch.Tensor, weights) -> torch.Tensor:
    """Context (B, L, hidden) of ``FlashDisentangledSelfAttention`` where ``covers`` gave these weights."""
    lens = None if lens is None else lens.contiguous()
    wq, bq, wk, bk, wv, bv = weights
    return _Projected.apply(x, rel, wq, wk, wv, bq, bk, bv, lens, module.num_attention_heads, module.position_buckets,
                            module.max_relative_positions)

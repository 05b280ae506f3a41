"""Training of the attention module as one autograd node: projections, position tables and attention.

Operator by operator the module's forward and backward are some forty autograd nodes and a hundred launches, which cost the host
more than the GPU needs for a batch of paragraphs.  Here the three projections are one GEMM over the concatenated weights, and
so are their gradients; the two position tables are a second one over the same weights (``share_att_key``); in between are
the fused attention and its backward (ops.py, backward.py), which read and write the GEMMs' buffers in place.

What it does not cover goes through the modules as before: see ``covers``.
"""
from __future__ import annotations

import math

import torch
from torch import nn
from torch.nn.modules import module as _nn_module

from . import backward, bucket, ops

_GLOBAL_HOOKS = ("_global_forward_hooks", "_global_forward_pre_hooks", "_global_backward_hooks", "_global_backward_pre_hooks")


def _plain_linear(m, device) -> bool:
    w, b = m.weight, m.bias
    return (type(m) is nn.Linear and b is not None and w.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and w.device == device
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks) and "forward" not in m.__dict__)


def covers(module, x, query_states, mask, rel) -> bool:
    """Whether a call is one that ``attention`` stands for: autograd recording, bf16 on the GPU, both position terms through the
    key and query projections themselves, self-attention over a dense batch, nothing between the operators (dropout, hooks,
    autocast, tracing)."""
    if not (torch.is_grad_enabled() and x.is_cuda and x.dtype == torch.bfloat16 and module.share_att_key and module.relative_attention
            and not module.attn_fp8 and module.attention_head_size == 64):
        return False
    if query_states is not None and query_states is not x:
        return False
    if rel is None or rel.dim() != 2 or rel.dtype != torch.bfloat16 or rel.device != x.device or x.numel() == 0:
        return False
    if "c2p" not in module.pos_att_type or "p2c" not in module.pos_att_type or not (mask is None or isinstance(mask, torch.Tensor)):
        return False
    drop = module.pos_dropout
    if (drop.training and drop.p > 0) or drop._forward_hooks or drop._forward_pre_hooks:
        return False
    if torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or any(getattr(_nn_module, h, None) for h in _GLOBAL_HOOKS):
        return False
    linears = (module.query_proj, module.key_proj, module.value_proj)
    if not all(_plain_linear(m, x.device) for m in linears):
        return False
    if rel.shape[0] < 2 * module.pos_ebd_size or not backward.index_covered(module.position_buckets, module.max_relative_positions):
        return False
    return ops.wants_grad(x, rel, *(t for m in linears for t in (m.weight, m.bias)))


class _Projected(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, rel, wq, wk, wv, bq, bk, bv, lens, heads, buckets, max_rel):
        B, L, hidden = x.shape
        span2 = 2 * bucket.att_span(buckets, max_rel)
        x2, rel2 = x.reshape(B * L, hidden), rel[:span2]
        w, b = torch.cat((wq, wk, wv)), torch.cat((bq, bk, bv))
        inner = heads * 64
        qkv = torch.addmm(b, x2, w.t())
        q, k, v = qkv.view(B, L, 3, heads, 64).unbind(2)
        # the queries' projection of the embeddings is the p2c table, the keys' the c2p one
        tables = torch.addmm(b[:2 * inner], rel2, w[:2 * inner].t()).view(span2, 2, heads, 64).permute(1, 2, 0, 3).contiguous()
        sm_scale = 1.0 / math.sqrt(64 * 3)
        out, lse = ops.disentangled_attention(q, k, v, tables[1], tables[0], seq_lens=lens, max_seqlen=L, sm_scale=sm_scale,
                                              position_buckets=buckets, max_relative_positions=max_rel, return_lse=True)
        ctx.save_for_backward(x2, rel, w, qkv, tables, out, lse, lens)
        ctx.fdb_args = (B, L, heads, sm_scale, buckets, max_rel)
        return out.view(B, L, inner)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, grad):
        x2, rel, w, qkv, tables, out, lse, lens = ctx.saved_tensors
        B, L, heads, sm_scale, buckets, max_rel = ctx.fdb_args
        span2, inner = tables.shape[2], heads * 64
        q, k, v = qkv.view(B, L, 3, heads, 64).unbind(2)
        d_qkv, d_tables = torch.empty_like(qkv), torch.empty_like(tables)
        backward._fused(grad.contiguous().view(B, L, heads, 64), q, k, v, tables[1], tables[0], out, lse, None, lens, L, sm_scale, buckets,
                        max_rel, d_qkv.view(B * L, 3, heads, 64), (d_tables[1], d_tables[0]))
        d_proj = d_tables.permute(2, 0, 1, 3).reshape(span2, 2 * inner)
        want = ctx.needs_input_grad
        grads = [None] * 8
        if want[0]:
            grads[0] = torch.mm(d_qkv, w).view(B, L, -1)
        if want[1]:
            d_rel = torch.mm(d_proj, w[:2 * inner])
            if rel.shape[0] != span2:
                d_rel = torch.cat((d_rel, d_rel.new_zeros(rel.shape[0] - span2, rel.shape[1])))
            grads[1] = d_rel
        if any(want[2:5]):
            dw = torch.mm(d_qkv.t(), x2)
            dw[:2 * inner].addmm_(d_proj.t(), rel[:span2])
            grads[2:5] = [g if n else None for g, n in zip(dw.split(inner), want[2:5])]
        if any(want[5:8]):
            db = ops.column_sums(d_qkv, d_proj)
            grads[5:8] = [g if n else None for g, n in zip(db.split(inner), want[5:8])]
        return (*grads, None, None, None, None)


def attention(module, x: torch.Tensor, lens, rel: torch.Tensor) -> torch.Tensor:
    """Context (B, L, hidden) of ``FlashDisentangledSelfAttention`` where ``covers`` holds."""
    q, k, v = module.query_proj, module.key_proj, module.value_proj
    return _Projected.apply(x, rel, q.weight, k.weight, v.weight, q.bias, k.bias, v.bias, lens, module.num_attention_heads,
                            module.position_buckets, module.max_relative_positions)

"""CPU-only checks of the C ABI: the library loads, exports what the header declares, the struct layouts agree,
the integer bucket table is bit-exact against the HuggingFace fixtures, and argument errors are reported before any
launch."""
import ctypes as C
import os
import re
import subprocess
import sys

import numpy as np
import pytest
import torch

from flashdeberta_b200 import _lib, bucket
from flashdeberta_b200.attention import lengths_from_mask
from tests._golden import load_bucket_golden

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "fdb_b200.h")


def test_library_loads_and_exports_every_declared_symbol():
    lib = _lib.load()
    text = open(HEADER).read()
    declared = set(re.findall(r"FDB_API[^;(]*?\b(fdb_[a-z0-9_]+)\s*\(", text))
    assert declared, "no declarations found in the header"
    assert declared == set(_lib.EXPORTS)
    for name in declared:
        assert hasattr(lib, name), name
    assert lib.fdb_abi_version() == _lib.ABI_VERSION


def test_struct_layout_matches_the_header(tmp_path):
    fields = [f[0] for f in _lib.AttnParams._fields_]
    src = tmp_path / "layout.c"
    body = "\n".join(f'  printf("{f} %zu\\n", offsetof(fdb_attn_params, {f}));' for f in fields)
    src.write_text(
        '#include <stdio.h>\n#include <stddef.h>\n#include "fdb_b200.h"\nint main(void) {\n'
        '  printf("sizeof %zu\\n", sizeof(fdb_attn_params));\n' + body + "\n  return 0;\n}\n")
    exe = tmp_path / "layout"
    subprocess.check_call(["gcc", "-std=c11", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    out = dict(line.split() for line in subprocess.check_output([str(exe)], text=True).splitlines())
    assert int(out["sizeof"]) == C.sizeof(_lib.AttnParams)
    for f in fields:
        assert int(out[f]) == getattr(_lib.AttnParams, f).offset, f


def test_backward_block_layout_matches_the_header(tmp_path):
    from flashdeberta_b200 import backward
    fields = [f[0] for f in backward.BwdBlock._fields_]
    src = tmp_path / "layout_bwd.c"
    body = "\n".join(f'  printf("{f} %zu\\n", offsetof(fdb_bwd_block, {f}));' for f in fields)
    src.write_text(
        '#include <stdio.h>\n#include <stddef.h>\n#include "fdb_b200.h"\nint main(void) {\n'
        '  printf("sizeof %zu\\n", sizeof(fdb_bwd_block));\n' + body + "\n  return 0;\n}\n")
    exe = tmp_path / "layout_bwd"
    subprocess.check_call(["gcc", "-std=c11", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    out = dict(line.split() for line in subprocess.check_output([str(exe)], text=True).splitlines())
    assert int(out["sizeof"]) == C.sizeof(backward.BwdBlock)
    for f in fields:
        assert int(out[f]) == getattr(backward.BwdBlock, f).offset, f


def test_backward_block_argument_errors():
    from flashdeberta_b200 import backward
    lib = _lib.load()
    p = backward.BwdBlock()
    assert lib.fdb_attn_bwd_probs(C.byref(p), None) == -1          # struct_bytes missing
    p.struct_bytes = C.sizeof(backward.BwdBlock)
    p.groups, p.heads, p.seqlen, p.row0, p.rows = 6, 4, 128, 0, 64  # groups not a multiple of heads
    assert lib.fdb_attn_bwd_probs(C.byref(p), None) == -1
    p.groups = 8
    p.row0 = 100                                                     # block reaches past the sequence
    assert lib.fdb_attn_bwd_probs(C.byref(p), None) == -1
    p.row0 = 0
    assert lib.fdb_attn_bwd_probs(C.byref(p), None) == -1          # tensors missing
    assert lib.fdb_attn_bwd_bucket_sums(C.byref(p), None) == -1    # no tables, no dscores
    assert lib.fdb_last_error().decode() != ""
    p.rows = 0
    p.scores = p.dprobs = p.lse = p.delta = p.probs = p.dscores = 0x1000
    assert lib.fdb_attn_bwd_probs(C.byref(p), None) == 0           # an empty block is a no-op


def _configs(g):
    for k in g:
        if k.startswith("idx_"):
            _, b, m = k.split("_")
            yield int(b), int(m)


def test_bucket_table_bit_exact_vs_hf_fixture():
    g = load_bucket_golden()
    d_lo, d_hi = int(g["d_lo"]), int(g["d_hi"])
    for buckets, max_rel in _configs(g):
        want = g[f"idx_{buckets}_{max_rel}"].astype(np.int64)
        tab, d_min = bucket.host_lut(buckets, max_rel)
        d = np.arange(d_lo, d_hi + 1)
        got = tab[np.clip(d - d_min, 0, len(tab) - 1)].astype(np.int64)
        assert np.array_equal(got, want), (buckets, max_rel)
        # the saturation claim: first/last entries hold beyond the table
        assert tab[0] == want[0] and tab[-1] == want[-1]
        for dist in (-40000, -513, -512, -129, -1, 0, 1, 128, 129, 505, 506, 40000):
            assert bucket.relative_index(dist, buckets, max_rel) == want[dist - d_lo]


def test_v3_table_shape():
    tab, d_min = bucket.host_lut(256, 512)
    assert (len(tab), d_min, int(tab[0]), int(tab[-1])) == (1019, -512, 0, 511)
    assert np.all(np.diff(tab.astype(np.int32)) >= 0)


def _params(**kw):
    p = _lib.AttnParams()
    p.struct_bytes = C.sizeof(_lib.AttnParams)
    p.dtype = _lib.FDB_BF16
    p.q = p.k = p.v = p.out = 0x1000
    for n in ("q", "k", "v"):
        setattr(p, n + "_row_stride", 128)
        setattr(p, n + "_head_stride", 64)
    p.out_row_stride, p.out_head_stride = 128, 64
    p.batch, p.max_seqlen, p.total_rows, p.heads, p.head_dim = 2, 64, 128, 2, 64
    p.sm_scale = 0.125
    for k, v in kw.items():
        setattr(p, k, v)
    return p


@pytest.mark.parametrize("change,code", [
    (dict(struct_bytes=8), -1),
    (dict(q=0), -1),
    (dict(head_dim=128), -2),
    (dict(dtype=_lib.FDB_FP32), -2),
    (dict(dtype=7), -1),
    (dict(q=0x1008), -3),
    (dict(q_row_stride=130), -3),
    (dict(total_rows=100), -1),
    (dict(sm_scale=0.0), -1),
    (dict(pos_key=0x2000), -1),       # tables without a bucket table
    (dict(seq_lens=0x10, cu_seqlens=0x10), -1),
    (dict(prepared=4), -1),           # unknown bit
])
def test_argument_errors_are_reported_before_any_launch(change, code):
    lib = _lib.load()
    p = _params(**change)
    assert lib.fdb_attn_fwd(C.byref(p), None) == code
    assert lib.fdb_last_error().decode() != ""
    with pytest.raises(_lib.FdbError):
        _lib.check(lib.fdb_attn_fwd(C.byref(p), None))


def test_missing_workspace_is_an_error():
    lib = _lib.load()
    p = _params()
    need = lib.fdb_attn_workspace_bytes(C.byref(p))
    assert need > 0 and need % 256 == 0
    assert lib.fdb_attn_fwd(C.byref(p), None) == -4


def test_lengths_from_every_mask_form():
    m2 = torch.tensor([[1, 1, 1, 0], [1, 0, 0, 0], [0, 0, 0, 0]])
    want = [3, 1, 0]
    assert lengths_from_mask(m2).tolist() == want
    ext = m2.unsqueeze(1).unsqueeze(2)
    m4 = ext * ext.squeeze(-2).unsqueeze(-1)
    assert lengths_from_mask(m4).tolist() == want
    assert lengths_from_mask(m4[:, 0]).tolist() == want
    assert lengths_from_mask(torch.tensor(want)).tolist() == want
    assert lengths_from_mask(None) is None


def test_ops_refuse_cpu_tensors():
    from flashdeberta_b200 import ops
    x = torch.zeros(1, 8, 1, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.disentangled_attention(x, x, x, None, None, max_seqlen=8)


@pytest.mark.parametrize("x,gamma,hidden,code", [
    (0, 0x1000, 768, -1),          # x NULL
    (0x1000, 0, 768, -1),          # gamma NULL
    (0x1000, 0x1000, 100, -2),     # hidden not a multiple of 256
    (0x1000, 0x1000, 4096, -2),    # hidden above 2048
    (0x1008, 0x1000, 768, -3),     # x not 16-byte aligned
])
def test_add_layernorm_argument_errors(x, gamma, hidden, code):
    lib = _lib.load()
    rc = lib.fdb_add_layernorm(x or None, None, gamma or None, 0x1000, 0x2000, 4, hidden, 1e-7, None)
    assert rc == code
    assert lib.fdb_last_error().decode() != ""


def test_add_layernorm_zero_rows_is_a_no_op():
    lib = _lib.load()
    assert lib.fdb_add_layernorm(0x1000, None, 0x1000, 0x1000, 0x2000, 0, 768, 1e-7, None) == 0


def test_layer_output_blocks_keep_transformers_parameter_names():
    """The blocks that call the fused add + LayerNorm are drop-in for transformers' (same state-dict keys), and fall back to
    transformers' own expression on CPU tensors."""
    from transformers.models.deberta_v2.configuration_deberta_v2 import DebertaV2Config
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Layer
    from flashdeberta_b200.model import FlashDebertaV2Layer
    cfg = DebertaV2Config(hidden_size=256, num_attention_heads=4, intermediate_size=512, num_hidden_layers=1,
                          relative_attention=True, position_buckets=32, max_relative_positions=64,
                          pos_att_type="c2p|p2c", share_att_key=True, vocab_size=100, type_vocab_size=0)
    cfg.attn_backend = "b200"
    torch.manual_seed(0)
    ours, theirs = FlashDebertaV2Layer(cfg).eval(), DebertaV2Layer(cfg).eval()
    assert set(ours.state_dict().keys()) == set(theirs.state_dict().keys())
    theirs.load_state_dict(ours.state_dict())
    h, x = torch.randn(2, 5, 512), torch.randn(2, 5, 256)
    with torch.no_grad():
        assert torch.equal(ours.output(h, x), theirs.output(h, x))
        assert torch.equal(ours.attention.output(x, x), theirs.attention.output(x, x))
        assert torch.equal(ours.intermediate(x), theirs.intermediate(x))


@pytest.mark.parametrize("x,rows,row_stride,head_stride,y,head_dim,code", [
    (0, 4, 768, 64, 0x2000, 64, -1),         # x NULL
    (0x1000, -1, 768, 64, 0x2000, 64, -1),   # negative row count
    (0x1000, 4, 768, 64, 0x2000, 60, -1),    # head_dim not a multiple of 8
    (0x1008, 4, 768, 64, 0x2000, 64, -3),    # x not 16-byte aligned
    (0x1000, 4, 768, 64, 0x2004, 64, -3),    # y not 8-byte aligned
    (0x1000, 4, 772, 64, 0x2000, 64, -3),    # row stride not a multiple of 8 elements
    (0x1000, 4, 768, 0, 0x2000, 64, -3),     # head stride not positive
])
def test_quantize_argument_errors(x, rows, row_stride, head_stride, y, head_dim, code):
    lib = _lib.load()
    rc = lib.fdb_quantize_e4m3(x or None, rows, row_stride, head_stride, 0x3000, 1, 12, head_dim, y, 0x4000, None)
    assert rc == code
    assert lib.fdb_last_error().decode() != ""


def test_quantize_zero_rows_is_a_no_op():
    lib = _lib.load()
    assert lib.fdb_quantize_e4m3(0x1000, 0, 768, 64, 0x3000, 1, 12, 64, 0x2000, 0x4000, None) == 0


@pytest.mark.parametrize("x,weight,k,n,code", [
    (0, 0x1000, 768, 3072, -1),        # x NULL
    (0x1000, 0, 768, 3072, -1),        # weight NULL
    (0x1000, 0x1000, 100, 3072, -2),   # in_features not a multiple of 64
    (0x1000, 0x1000, 768, 1000, -2),   # out_features not a multiple of 256
    (0x1008, 0x1000, 768, 3072, -3),   # x not 16-byte aligned
])
def test_linear_gelu_argument_errors(x, weight, k, n, code):
    lib = _lib.load()
    rc = lib.fdb_linear_gelu(x or None, weight or None, None, 0x2000, 4, k, n, None, None)
    assert rc == code
    assert lib.fdb_last_error().decode() != ""


def test_linear_gelu_zero_rows_is_a_no_op():
    lib = _lib.load()
    assert lib.fdb_linear_gelu(0x1000, 0x1000, None, 0x2000, 0, 768, 3072, None, None) == 0


@pytest.mark.parametrize("ids,table,rows_in_table,hidden,code", [
    (0, 0x1000, 100, 768, -1),         # ids NULL
    (0x1000, 0, 100, 768, -1),         # table NULL
    (0x1000, 0x1000, 0, 768, -1),      # empty table
    (0x1000, 0x1000, 100, 100, -2),    # hidden not a multiple of 256
    (0x1000, 0x1008, 100, 768, -3),    # table not 16-byte aligned
])
def test_embed_layernorm_argument_errors(ids, table, rows_in_table, hidden, code):
    lib = _lib.load()
    rc = lib.fdb_embed_layernorm(ids or None, table or None, rows_in_table, 0x1000, 0x1000, None, 0x2000, 4, hidden, 1e-7,
                                 None, None)
    assert rc == code
    assert lib.fdb_last_error().decode() != ""


def test_model_keeps_transformers_parameter_names():
    """Every block this package swaps in (embeddings, attention, intermediate and output blocks) keeps transformers'
    state-dict keys, so checkpoints load unchanged; on CPU tensors the blocks run transformers' own code."""
    from transformers.models.deberta_v2.configuration_deberta_v2 import DebertaV2Config
    from transformers.models.deberta_v2.modeling_deberta_v2 import DebertaV2Model
    from flashdeberta_b200 import FlashDebertaV2Model
    cfg = DebertaV2Config(hidden_size=256, num_attention_heads=4, intermediate_size=512, num_hidden_layers=2,
                          relative_attention=True, position_buckets=32, max_relative_positions=64,
                          pos_att_type="c2p|p2c", share_att_key=True, vocab_size=100, type_vocab_size=0,
                          position_biased_input=False, norm_rel_ebd="layer_norm")
    cfg.attn_backend = "b200"
    ours, theirs = FlashDebertaV2Model(cfg).eval(), DebertaV2Model(cfg).eval()
    assert set(ours.state_dict().keys()) == set(theirs.state_dict().keys())
    theirs.load_state_dict(ours.state_dict())
    ids, mask = torch.randint(1, 100, (2, 9)), torch.ones(2, 9)
    with torch.no_grad():
        assert torch.equal(ours.embeddings(input_ids=ids, mask=mask), theirs.embeddings(input_ids=ids, mask=mask))


def test_backward_workspace_is_bounded_beside_what_every_row_needs_once():
    """The bucket sums (2 bytes per row, head and table row) are kept for as many heads at a time as fit 2 GiB."""
    from flashdeberta_b200 import backward
    lib, lut = _lib.load(), 0x1000
    for rows, heads, buckets in [(1 << 20, 16, 256), (400000, 12, 256), (1 << 17, 16, 256), (1 << 20, 16, 1600), (4096, 12, 256)]:
        p = _params(batch=1, max_seqlen=rows, total_rows=rows, heads=heads, pos_key=0x1000, pos_query=0x1000, position_buckets=buckets,
                    max_relative_positions=2 * buckets, bucket_lut=lut, lut_d_min=-2 * buckets, lut_len=3000)
        for n in ("q", "k", "v"):
            setattr(p, n + "_row_stride", heads * 64)
        p.out_row_stride = heads * 64
        b = backward.BwdParams()
        b.struct_bytes, b.fwd = C.sizeof(b), C.pointer(p)
        need = lib.fdb_attn_bwd_workspace_bytes(C.byref(b))
        once = rows * heads * (64 * 4 + 4)                                  # dQ or dK in fp32, delta
        sums = min(rows * heads * 2 * buckets * 2, max(1 << 31, rows * 2 * buckets * 2))  # (one head at least)
        assert once < need <= once + sums + (128 << 20), (rows, heads, buckets, need)


def test_encoder_plan_of_too_many_layers_is_an_error():
    """Not an exception that leaves the C entry, and no allocation of that size."""
    from flashdeberta_b200 import engine
    lib, layer, plan = _lib.load(), engine.EncoderLayer(), C.c_void_p()
    for n in (4097, 2 ** 31 - 1):
        assert lib.fdb_encoder_create(C.byref(layer), n, 256, 4, 512, C.byref(plan)) == -6
    assert not plan.value and "layers" in lib.fdb_last_error().decode()


def _structs():
    from flashdeberta_b200 import backward, engine, projected
    return [("fdb_attn_bwd_params", backward.BwdParams), ("fdb_quantize_attn_params", _lib.QuantizeAttnParams),
            ("fdb_encoder_layer", engine.EncoderLayer), ("fdb_projected_params", projected._ProjectedParams),
            ("fdb_encoder_call", engine.EncoderCall)]


@pytest.mark.parametrize("name,struct", _structs(), ids=[n for n, _ in _structs()])
def test_other_struct_layouts_match_the_header(name, struct, tmp_path):
    """Size, order and offsets, of every field that the header declares."""
    text = open(HEADER).read()
    body = re.sub(r"/\*.*?\*/", "", re.search(r"typedef struct %s \{(.*?)\} %s;" % (name, name), text, re.S).group(1), flags=re.S)
    declared = [re.search(r"(\w+)$", part.strip()).group(1) for line in body.split(";") for part in line.split(",") if part.strip()]
    rename = {"fdb_quantize_attn_params": {"in": "input"}}.get(name, {})
    assert [rename.get(f, f) for f in declared] == [f[0] for f in struct._fields_]
    src, exe = tmp_path / "layout.c", tmp_path / "layout"
    src.write_text('#include <stdio.h>\n#include <stddef.h>\n#include "fdb_b200.h"\nint main(void) {\n  printf("%%zu", sizeof(%s));\n' % name
                   + "".join('  printf(" %%zu", offsetof(%s, %s));\n' % (name, f) for f in declared) + "  return 0;\n}\n")
    subprocess.check_call(["gcc", "-std=c11", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    out = [int(v) for v in subprocess.check_output([str(exe)], text=True).split()]
    assert out == [C.sizeof(struct)] + [getattr(struct, rename.get(f, f)).offset for f in declared]


def _with_tables(**kw):
    base = dict(pos_key=0x1000, pos_query=0x1000, position_buckets=256, max_relative_positions=512, bucket_lut=0x1000, lut_d_min=-512, lut_len=1019)
    base.update(kw)
    return _params(**base)


def _refused(rc, code):
    assert rc == code and _lib.load().fdb_last_error().decode() != ""


@pytest.mark.parametrize("change,code", [
    (dict(struct_bytes=0), -1), (dict(dout=None), -1), (dict(dq=None), -1), (dict(dpos_key=None), -1), (dict(dpos_query=None), -1),
    (dict(dout=0x1008), -3), (dict(dv=0x1002), -3), (dict(dout_row_stride=100), -3), (dict(grad_head_stride=0), -3),
    (dict(table_row_stride=4), -3), (dict(workspace=None), -4), (dict(workspace_bytes=16), -4), (dict(workspace=0x1010), -3),
])
def test_backward_argument_errors(change, code):
    from flashdeberta_b200 import backward
    p = _with_tables(lse=0x1000)
    b = backward.BwdParams(C.sizeof(backward.BwdParams), 0, C.pointer(p), 0x1000, 128, 64, 0x1000, 0x1000, 0x1000, 128, 64, 0x1000, 0x1000, 0, 0,
                           0x1000, 1 << 40)
    for k, v in change.items():
        setattr(b, k, v)
    _refused(_lib.load().fdb_attn_bwd(C.byref(b), None), code)


@pytest.mark.parametrize("change,code", [
    (dict(dtype=1), -2), (dict(head_dim=32), -2), (dict(position_buckets=255), -2), (dict(lut_len=4000), -6), (dict(lse=None), -1),
])
def test_backward_refuses_calls_it_is_not_for(change, code):
    from flashdeberta_b200 import backward
    p = _with_tables(lse=0x1000, **change) if "lse" not in change else _with_tables()
    b = backward.BwdParams(C.sizeof(backward.BwdParams), 0, C.pointer(p), 0x1000, 128, 64, 0x1000, 0x1000, 0x1000, 128, 64, 0x1000, 0x1000, 0, 0,
                           0x1000, 1 << 40)
    _refused(_lib.load().fdb_attn_bwd(C.byref(b), None), code)


@pytest.mark.parametrize("change,code", [
    (dict(struct_bytes=0), -1), (dict(input=None), -1), (dict(q=None), -1), (dict(pos_key=None), -1), (dict(k_scale=None), -1),
    (dict(v=0x1004), -3), (dict(pos_query=0x1001), -3), (dict(q_scale=0x1002), -3), (dict(amax=0x1001), -3), (dict(amax=None), -4), (dict(amax_bytes=8), -4),
])
def test_quantize_attn_argument_errors(change, code):
    p = _with_tables()
    q = _lib.QuantizeAttnParams(C.sizeof(_lib.QuantizeAttnParams), 0, C.pointer(p), *[0x1000] * 11, 1 << 20)
    for k, v in change.items():
        setattr(q, k, v)
    _refused(_lib.load().fdb_quantize_attn(C.byref(q), None), code)


def test_quantize_attn_without_rows_is_a_no_op():
    p = _with_tables(batch=0, total_rows=0)
    q = _lib.QuantizeAttnParams(C.sizeof(_lib.QuantizeAttnParams), 0, C.pointer(p))
    assert _lib.load().fdb_quantize_attn(C.byref(q), None) == 0


@pytest.mark.parametrize("change,code", [
    (dict(struct_bytes=0), -1), (dict(attn=None), -1), (dict(in_features=100), -2), (dict(x=None), -1), (dict(bv=None), -1),
    (dict(wk=0x1008), -3), (dict(rel=0x1008), -3), (dict(table_row_stride=64), -3), (dict(table_row_stride=132), -3), (dict(table_head_stride=128), -3),
])
def test_projected_forward_argument_errors(change, code):
    from flashdeberta_b200 import projected
    p = _with_tables(lse=0x1000, workspace=0x1000, workspace_bytes=1 << 40)
    c = projected._ProjectedParams(C.sizeof(projected._ProjectedParams), 128, C.pointer(p), 256, 64, *[0x1000] * 8)
    for k, v in change.items():
        setattr(c, k, v)
    _refused(_lib.load().fdb_projected_forward(C.byref(c), None), code)


@pytest.mark.parametrize("args,code", [
    ((None, 0, 2, 8, 8, 1, 0x1000, None), -1), ((0x1000, 0, 2, 8, 8, 1, None, None), -1), ((0x1000, 9, 2, 8, 8, 1, 0x1000, None), -1),
    ((0x1000, 0, -1, 8, 8, 1, 0x1000, None), -1), ((0x1002, 0, 2, 8, 8, 1, 0x1000, None), -3), ((0x1004, 1, 2, 8, 8, 1, 0x1000, None), -3),
    ((0x1001, 4, 2, 8, 8, 1, 0x1000, None), -3), ((0x1000, 3, 2, 8, 8, 1, 0x1002, None), -3), ((None, 0, 0, 8, 8, 1, None, None), 0),
])
def test_lengths_from_mask_argument_errors(args, code):
    assert _lib.load().fdb_lengths_from_mask(*args, None) == code


@pytest.mark.parametrize("args,code", [
    ((None, 8, 64, None, 0, 0, 0x1000, 0x1000, 1 << 20), -1), ((0x1000, 8, 64, None, 4, 64, 0x1000, 0x1000, 1 << 20), -1),
    ((0x1000, 8, 64, 0x1000, 4, 72, 0x1000, 0x1000, 1 << 20), -1), ((0x1000, 8, 60, None, 0, 0, 0x1000, 0x1000, 1 << 20), -3),
    ((0x1008, 8, 64, None, 0, 0, 0x1000, 0x1000, 1 << 20), -3), ((0x1000, 8, 64, None, 0, 0, 0x1001, 0x1000, 1 << 20), -3),
    ((0x1000, 8, 64, None, 0, 0, 0x1000, 0x1002, 1 << 20), -3), ((0x1000, 8, 64, None, 0, 0, 0x1000, None, 0), -4), ((0x1000, 8, 64, None, 0, 0, 0x1000, 0x1000, 8), -4),
])
def test_column_sums_argument_errors(args, code):
    _refused(_lib.load().fdb_column_sums(*args, None), code)


@pytest.mark.parametrize("args,code", [
    ((0x1000, None, None, None, 12, 512, 0x1000, -512, 1019), -1), ((0x1000, None, 0x1000, None, 12, 512, None, -512, 1019), -1),
    ((0x1000, None, 0x1000, None, 0, 512, 0x1000, -512, 1019), -1), ((0x1008, None, 0x1000, None, 12, 512, 0x1000, -512, 1019), -3),
    ((0x1000, None, 0x1008, None, 12, 512, 0x1000, -512, 1019), -3), ((None, 0x1000, None, 0x1002, 12, 512, 0x1000, -512, 1019), -3),
    ((0x1000, None, 0x1000, None, 12, 512, 0x1001, -512, 1019), -3), ((None, None, None, None, 12, 512, 0x1000, -512, 1019), 0),
])
def test_expand_tables_argument_errors(args, code):
    assert _lib.load().fdb_expand_tables(*args, None) == code


@pytest.mark.parametrize("change,sizes,code", [
    ({}, (256, 3, 512), -2), ({}, (192, 3, 512), -2), ({}, (256, 4, 500), -2), ({}, (4096, 64, 512), -2), (dict(wq=None), (256, 4, 512), -1),
    (dict(ln2_beta=None), (256, 4, 512), -1), (dict(wd=0x1008), (256, 4, 512), -3), (dict(ln1_gamma=0x1008), (256, 4, 512), -3),
    (dict(ln2_beta=0x1004), (256, 4, 512), -3), (dict(exp_query=0x1008), (256, 4, 512), -3),
])
def test_encoder_create_argument_errors(change, sizes, code):
    from flashdeberta_b200 import engine
    layer, plan = engine.EncoderLayer(*[0x1000] * 18, 1e-7, 1e-7), C.c_void_p()
    for k, v in change.items():
        setattr(layer, k, v)
    _refused(_lib.load().fdb_encoder_create(C.byref(layer), 1, *sizes, C.byref(plan)), code)
    assert not plan.value


@pytest.mark.parametrize("change,code", [
    (dict(struct_bytes=0), -1), (dict(plan=None), -1), (dict(ids=None), -1), (dict(out=None), -1), (dict(batch=-1), -1), (dict(emb_rows=0), -1),
    (dict(total_rows=99), -1), (dict(cu_seqlens=0x1000, mask=0x1000), -1), (dict(mask_type=7), -1), (dict(out=0x1008), -3), (dict(emb_table=0x1008), -3),
    (dict(emb_beta=0x1004), -3), (dict(ids=0x1004), -3), (dict(mask=0x1004, mask_type=1), -3), (dict(mask=0x1001, mask_type=4), -3), (dict(cu_seqlens=0x1002), -3),
])
def test_encoder_call_argument_errors(change, code):
    from flashdeberta_b200 import engine
    c = engine.EncoderCall()
    c.struct_bytes, c.plan, c.ids, c.out = C.sizeof(c), 0x1000, 0x1000, 0x1000
    c.emb_table = c.emb_gamma = c.emb_beta = 0x1000
    c.batch, c.max_seqlen, c.total_rows, c.emb_rows = 2, 50, 100, 1000
    for k, v in change.items():
        setattr(c, k, v)
    lib = _lib.load()
    _refused(lib.fdb_encoder_forward(C.byref(c), None), code)
    assert lib.fdb_encoder_workspace_bytes(C.byref(c)) == 0

"""GPU parity of the decode kernel (seqlen_q = 1, keys on the tensor-memory lanes)
against the CPU oracle, same tolerances as the tiled path."""
import numpy as np
import pytest
import torch

import gpu_util
import oracle_lib
from plan_util import plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("nk,splits", [(128, 1), (1000, 1), (4096, 16), (5000, 7), (32768, 16), (300, 8)])
def test_decode_plain(dtype, nk, splits):
    gpu_util.assert_close(gpu_util.run_case(2, 4, 1, nk, 128, dtype, seed=50, num_splits=splits), f"nk={nk} s={splits}")


@pytest.mark.parametrize("d", [64, 96, 128, 32])
def test_decode_head_dims(d):
    gpu_util.assert_close(gpu_util.run_case(2, 3, 1, 2000, d, "bfloat16", seed=51, num_splits=4), f"d={d}")


def test_decode_masks_and_bias():
    # the query sits at the end of the sequence (bottom-right causal), some keys lie after it
    gpu_util.assert_close(gpu_util.run_case(1, 4, 1, 3000, 128, "bfloat16", seed=52, causal=True, q_pos0=2500,
                                            num_splits=6), "causal q_pos0 (empty splits)")
    gpu_util.assert_close(gpu_util.run_case(1, 4, 1, 3000, 128, "bfloat16", seed=53, causal=True, q_pos0=2999,
                                            window=(700, 0), alibi=True, num_splits=4), "causal + window + alibi")
    gpu_util.assert_close(gpu_util.run_case(1, 2, 1, 1500, 128, "float16", seed=54, window=(100, 50), q_pos0=800,
                                            num_splits=3), "two-sided window")
    # nothing visible at all: O = 0, LSE = -inf
    gpu_util.assert_close(gpu_util.run_case(1, 2, 1, 600, 128, "bfloat16", seed=55, causal=True, k_pos0=10,
                                            num_splits=2), "fully masked row")


def test_decode_dropout_follows_the_reference_streams():
    gpu_util.assert_close(gpu_util.run_case(2, 4, 1, 2048, 128, "bfloat16", seed=56, p_dropout=0.2, drop_seed=11,
                                            num_splits=1), "dropout")
    gpu_util.assert_close(gpu_util.run_case(2, 4, 1, 4096, 128, "bfloat16", seed=57, p_dropout=0.1, drop_seed=42,
                                            num_splits=4, offset=8), "dropout split")


def test_decode_config4_shape_sampled_units():
    # bf16 B=64 H=32 q=1 kv=32768 d=128, 16 splits: every unit is computed, a sample is checked
    import flash_attn_b200 as fa
    B, H, Nk, d = 64, 32, 32768, 128
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    q = torch.randn((B, H, 1, d), generator=g, device="cuda").bfloat16()
    k = torch.randn((B, H, Nk, d), generator=g, device="cuda").bfloat16()
    v = torch.randn((B, H, Nk, d), generator=g, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    o, lse = fa.flash_attn_forward(q, k, v, num_splits=16, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for b, h in ((0, 0), (63, 31), (17, 5), (40, 20)):
        want_o, want_lse = oracle_lib.forward(q[b:b + 1, h:h + 1].float().cpu().numpy(), k[b:b + 1, h:h + 1].float().cpu().numpy(),
                                              v[b:b + 1, h:h + 1].float().cpu().numpy(), d ** -0.5)
        err = np.abs(o[b, h].float().cpu().numpy() - want_o[0, 0])
        assert err.max() <= gpu_util.O_MAX_ABS and err.mean() <= gpu_util.O_MEAN_ABS, (b, h, err.max())
        assert abs(lse[b, h, 0].item() - want_lse[0, 0, 0]) <= gpu_util.LSE_ABS


@pytest.mark.parametrize("H,Hk,Nq,nk,d,dtype,kw", [
    (8, 2, 1, 129, 128, "bfloat16", {}),                      # 4 columns; two tiles, the second with one key
    (8, 2, 1, 1023, 128, "float16", {}),                      # 8-CTA cluster, one tile each, the last ragged
    (8, 2, 1, 2100, 64, "bfloat16", {}),                      # 16-CTA cluster, uneven parts, 64-wide tiles
    (7, 1, 1, 4097, 128, "bfloat16", {}),                     # 8 columns, one unused
    (8, 2, 4, 3000, 128, "bfloat16", {}),                     # 16 columns: 4 heads x 4 rows
    (12, 1, 5, 2500, 64, "float16", dict(window=(700, 0))),   # 15 columns, four sub-groups of 3 heads, clipped tiles
    (4, 2, 8, 1500, 96, "bfloat16", dict(alibi=True)),        # 16 columns with a bias per head
    (2, 1, 3, 5000, 128, "bfloat16", dict(window=(100, 0))),  # few visible tiles in a long cache
    (4, 1, 1, 65500, 64, "bfloat16", dict(num_splits=0)),     # more parts than a cluster holds: the combine kernel
    (4, 1, 2, 900, 128, "float16", dict(p_dropout=0.2, num_splits=4)),   # the caller's splits, merged in the cluster
    (2, 2, 1, 900, 128, "float16", dict(p_dropout=0.2, num_splits=5)),   # ... and through the workspace
])
def test_parts_of_a_unit_and_query_columns(H, Hk, Nq, nk, d, dtype, kw):
    gpu_util.assert_close(gpu_util.run_case(1, H, Nq, nk, d, dtype, seed=58, causal=True, q_pos0=nk - Nq, heads_k=Hk, **kw),
                          f"{H}/{Hk} heads, {Nq} rows, {nk} keys, d={d} {kw}")


@pytest.mark.parametrize("H,Hk,Nq,nk,kw", [
    (8, 2, 4, 700, {}),                                   # 4 heads x 4 rows of a K/V head, a ragged last chunk
    (10, 2, 3, 300, dict(offset=6)),                      # 5 heads x 3 rows, draws that straddle two Philox blocks
    (2, 2, 6, 1100, dict(num_splits=3)),                  # one head's rows share their draws
    (16, 2, 1, 600, dict(num_splits=2, launch_index=3)),  # 8 heads, a later launch of a loop
])
def test_dropout_of_query_rows_and_heads_that_share_keys(H, Hk, Nq, nk, kw):
    gpu_util.assert_close(gpu_util.run_case(2, H, Nq, nk, 64, "bfloat16", seed=59, causal=True, q_pos0=nk - Nq, heads_k=Hk,
                                            p_dropout=0.25, drop_seed=7, **kw), f"{H}/{Hk} heads, {Nq} rows, {nk} keys {kw}")


@pytest.mark.parametrize("tiles", [2039, 2048])  # a prime number of key tiles, and one that splits in many ways
@pytest.mark.parametrize("d", [64, 60])        # 60: padded copies, which do need a workspace
def test_a_plan_of_many_parts_does_without_their_workspace(tiles, d):
    """num_splits = 0 leaves the count to the library: with no room for the partials of its plan the parts are as many as a
    cluster merges.  (The C entry point; the Python one always brings the workspace that was asked for.)"""
    import ctypes
    import flash_attn_b200 as fa
    from flash_attn_b200 import _lib
    L = _lib.load()
    H, Hk, Nk = 4, 1, 128 * tiles
    got = plan(1, H, 1, Nk, d, heads_k=Hk)
    assert got.parts > 16 and not got.merged
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    q, k, v = (torch.randn((1, h, n, d), generator=g, device="cuda").bfloat16() for h, n in ((H, 1), (Hk, Nk), (Hk, Nk)))
    want_o, want_lse = fa.flash_attn_forward(q, k, v, num_splits=0)
    p = _lib.FwdParams()
    p.q, p.k, p.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    p.dtype = p.o_dtype = _lib.FA_DTYPE_BF16
    p.batch, p.heads, p.heads_k, p.seqlen_q, p.seqlen_k, p.head_dim = 1, H, Hk, 1, Nk, d
    p.softmax_scale, p.window_left, p.window_right = d ** -0.5, -1, -1
    p.stream = torch.cuda.current_stream().cuda_stream
    o, lse = torch.zeros_like(want_o), torch.zeros_like(want_lse)
    p.o, p.lse = o.data_ptr(), lse.data_ptr()
    need = L.fa_fwd_workspace_bytes(ctypes.byref(p))
    p.num_splits = 1
    least = L.fa_fwd_workspace_bytes(ctypes.byref(p))  # of the padded copies alone
    p.num_splits = 0
    assert need > least and (least > 0) == (d == 60)
    ws = torch.empty(need, device="cuda", dtype=torch.uint8)
    p.workspace = ws.data_ptr() if least else None
    p.workspace_bytes = least
    assert L.fa_fwd(ctypes.byref(p)) == 0
    torch.cuda.synchronize()
    assert (o.float() - want_o.float()).abs().max() <= gpu_util.O_MAX_ABS
    assert (lse - want_lse).abs().max() <= gpu_util.LSE_ABS
    p.num_splits = 32  # a count of the caller's: its workspace is asked for, as ever
    assert L.fa_fwd(ctypes.byref(p)) == -3


@pytest.mark.parametrize("B,H,Hk,Nq,nk,d,kw,columns,parts", [
    (1, 12, 2, 3, 69, 128, {}, 4, 1),                 # a head's three rows a CTA: six CTAs per K/V head
    (2, 64, 8, 5, 1848, 128, {}, 8, 1),               # (window) five rows a CTA
    (1, 32, 8, 8, 590, 128, {}, 8, 4),
    (4, 28, 4, 2, 700, 64, {}, 4, 4),                 # sub-groups of two heads, one of one
    (16, 32, 8, 4, 4100, 128, {}, 16, 2),             # sixteen where CTAs are many
    (1, 4, 1, 1, 262000, 64, {}, 4, 64),              # more parts than a cluster holds: the combine kernel
])
def test_columns_and_parts_of_the_plan(B, H, Hk, Nq, nk, d, kw, columns, parts):
    kw = dict(kw)
    if nk == 1848:
        kw["window"] = (200, 0)
    got = plan(B, H, Nq, nk, d, heads_k=Hk, causal=True, q_pos0=nk - Nq, **kw)
    assert (got.columns, got.parts) == (columns, parts)
    import flash_attn_b200 as fa
    torch.manual_seed(60)
    q, k, v = (torch.randn(B, h, n, d, device="cuda", dtype=torch.bfloat16) for h, n in ((H, Nq), (Hk, nk), (Hk, nk)))
    o, lse = fa.flash_attn_forward(q, k, v, causal=True, q_pos0=nk - Nq, num_splits=0, **kw)
    torch.cuda.synchronize()
    units = sorted({0, H // Hk - 1, H // Hk % (B * H), B * H // 2, B * H - 1})
    gpu_util.assert_close(gpu_util.check_sampled_units(q, k, v, o, lse, units, lambda u: range(Nq), d ** -0.5, causal=True,
                                                       q_pos0=nk - Nq, **kw), str((B, H, Nq, nk, d, kw)))

"""Query blocks whose keys are shared out over the CTAs of a cluster, and grouped queries stacked into common query
tiles.  Same tolerances as the unsplit kernel.  (What a case is cut into is the plan's choice: the cases that name it check
it against the plan for a B200.)"""
import pytest
import torch

import gpu_util
from plan_util import plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    dict(H=8, heads_k=2, Nq=130, Nk=3000, d=128, causal=True, q_pos0=2870),                  # grouped, two query tiles a head
    dict(H=4, Nq=100, Nk=2000, d=64, dtype="float16"),                                       # one query tile a unit
    dict(H=6, heads_k=2, Nq=40, Nk=2500, d=128, causal=True, q_pos0=2460, window=(300, 0)),  # grouped, left window
    dict(H=6, heads_k=2, Nq=43, Nk=900, d=64, q_pos0=400, window=(100, 60)),                 # grouped, both windows
    dict(H=4, heads_k=2, Nq=300, Nk=2500, d=64, causal=True, q_pos0=2200, alibi=True),       # grouped, a slope per head
    dict(H=2, Nq=257, Nk=1500, d=96, dtype="float16", window=(200, 100), q_pos0=600),
    dict(H=8, heads_k=1, Nq=20, Nk=700, d=31, dtype="float16", out_dtype=torch.float32),     # padded rows, scalar stores
    dict(H=2, Nq=400, Nk=2000, d=128, causal=True, q_pos0=50),                               # most keys invisible
    dict(H=4, Nq=384, Nk=1100, d=128, num_splits=3),
    dict(H=16, heads_k=4, Nq=62, Nk=1300, d=128, causal=True, q_pos0=1238),                  # grouped, one tile a head
    dict(H=128, Nq=257, Nk=300, d=100, dtype="float16", out_dtype=torch.float32),            # padded rows, unsplit
    dict(H=2, Nq=9, Nk=1100, d=20, dtype="float16"),                                         # fewest rows, 4-byte rows of O
])
def test_split_and_stacked_blocks_match_the_oracle(case):
    case = dict(case)
    H, Nq, Nk, d = (case.pop(x) for x in ("H", "Nq", "Nk", "d"))
    case.setdefault("num_splits", 0)
    gpu_util.assert_close(gpu_util.run_case(1, H, Nq, Nk, d, seed=71, **case), str((H, Nq, Nk, d, case)))


@pytest.mark.parametrize("B,H,Hk,Nq,Nk,d,kw,parts,stacked", [
    (1, 32, 8, 300, 8492, 128, dict(causal=True, q_pos0=8192), 3, 300),                       # tiles across heads, and split
    (6, 32, 8, 62, 2419, 128, dict(causal=True, q_pos0=2357), 2, 62),
    (6, 32, 8, 62, 2419, 128, dict(causal=True, q_pos0=2357, fp32_out=True), 2, 62),
    (6, 32, 8, 62, 1300, 64, dict(causal=True, q_pos0=1238), 2, 62),
    (6, 32, 8, 62, 1300, 100, dict(causal=True, q_pos0=1238), 2, 62),                         # padded rows
    (12, 32, 8, 43, 1500, 128, dict(causal=True, q_pos0=1457, window=(300, 0)), 1, 43),       # stacked only
    (12, 32, 8, 43, 1500, 128, dict(q_pos0=700, window=(200, 100)), 1, 43),
    (12, 28, 4, 50, 700, 128, dict(causal=True, q_pos0=650), 1, 50),                          # seven heads a group
    (1, 2, 2, 200, 9000, 128, {}, 16, 0),
    (1, 3, 3, 300, 16000, 128, dict(causal=True, q_pos0=15700, fp32_out=True), 16, 0),
    (1, 1, 1, 100, 16000, 64, {}, 16, 0),                                                     # one query tile a CTA
    (1, 4, 4, 300, 2500, 64, dict(causal=True, q_pos0=2200, alibi=True, fp32_out=True), 8, 0),
])
def test_cut_as_the_plan_says_and_right(B, H, Hk, Nq, Nk, d, kw, parts, stacked):
    import flash_attn_b200 as fa
    import synth
    got = plan(B, H, Nq, Nk, d, heads_k=Hk, **kw)
    assert (got.parts, got.stacked_rows, got.staged) == (parts, stacked, 1)
    kw = dict(kw)
    fp32, alibi = kw.pop("fp32_out", False), kw.pop("alibi", False)
    torch.manual_seed(72)
    q, k, v = (torch.randn(B, h, n, d, device="cuda", dtype=torch.bfloat16) for h, n in ((H, Nq), (Hk, Nk), (Hk, Nk)))
    slopes = synth.alibi_slopes(H) if alibi else None
    o, lse = fa.flash_attn_forward(q, k, v, num_splits=0, out_dtype=torch.float32 if fp32 else None,
                                   alibi_slopes=None if slopes is None else torch.from_numpy(slopes), **kw)
    torch.cuda.synchronize()
    edges = [0, 1, Nq // 2, Nq - 1] + [x for t in range(128, Nq, 128) for x in (t - 1, t)]
    units = sorted({0, 1 % (B * H), H // Hk - 1, B * H // 2, B * H - 2, B * H - 1} & set(range(B * H)))
    rows = lambda u: edges + [(128 * t - (u % (H // Hk)) * Nq + x) % Nq for t in range(1, 4) for x in (-1, 0)]  # (the tiles' edges)
    gpu_util.assert_close(gpu_util.check_sampled_units(q, k, v, o, lse, units, rows, d ** -0.5, causal=kw.get("causal", False),
                                                       window=kw.get("window", (-1, -1)), slopes=slopes,
                                                       q_pos0=kw.get("q_pos0", 0)), str((B, H, Nq, Nk, d, kw)))


@pytest.mark.parametrize("Nq,Nk", [(1, 2000), (4, 2000), (40, 2000), (300, 2000)])
def test_nan_in_a_value_reaches_every_row_that_sees_it(Nq, Nk):
    import flash_attn_b200 as fa
    torch.manual_seed(5)
    q, k, v = (torch.randn(1, 2, n, 128, device="cuda", dtype=torch.bfloat16) for n in (Nq, Nk, Nk))
    v[0, 1, 700] = float("nan")
    assert plan(1, 2, Nq, Nk, 128).merged == 1
    o, _ = fa.flash_attn_forward(q, k, v, num_splits=0)
    assert torch.isnan(o[0, 1]).all() and torch.isfinite(o[0, 0]).all()


@pytest.mark.parametrize("Nq,Nk", [(1, 2000), (4, 2000), (40, 2000), (300, 2000)])
def test_nan_reaches_its_rows_through_the_merge(Nq, Nk):
    import flash_attn_b200 as fa
    torch.manual_seed(5)
    q, k, v = (torch.randn(1, 2, n, 128, device="cuda", dtype=torch.bfloat16) for n in (Nq, Nk, Nk))
    q[0, 1, Nq - 1] = float("nan")
    o, _ = fa.flash_attn_forward(q, k, v, num_splits=0)
    assert torch.isnan(o[0, 1, Nq - 1]).all()
    assert torch.isfinite(o[0, 0]).all() and torch.isfinite(o[0, 1, : Nq - 1]).all()


@pytest.mark.parametrize("B,H,Hk,Nq,Nk,window,poisoned,rows", [
    (1, 32, 8, 300, 8492, (-1, -1), slice(8448, 8492), slice(0, 256)),  # keys that only the last query tile of a head reaches
    (8, 64, 8, 140, 1000, (300, 0), slice(0, 640), slice(128, 140)),    # ... that only the first one reaches
])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_masked_values_stay_out_of_query_tiles_that_do_not_reach_them(B, H, Hk, Nq, Nk, window, poisoned, rows, value):
    """V rows that are not finite (an unused part of a cache) reach the 128-row query tiles of a head that walk their KV
    tile, as P = 0 times them, and no others, however the launch is cut."""
    import flash_attn_b200 as fa
    torch.manual_seed(6)
    q, k, v = (torch.randn(B, h, n, 128, device="cuda", dtype=torch.bfloat16) for h, n in ((H, Nq), (Hk, Nk), (Hk, Nk)))
    call = lambda: fa.flash_attn_forward(q, k, v, causal=True, window=window, q_pos0=Nk - Nq, num_splits=0)[0][:, :, rows]
    clean = call()
    v[:, :, poisoned] = value
    assert torch.equal(call(), clean)


@pytest.mark.parametrize("num_splits", [0, 32])
def test_host_call_keeps_no_room_for_partials_that_nobody_writes(num_splits):
    from flash_attn_b200 import _lib, api
    L = _lib.load()
    H, Hk, Nq, Nk, d = 32, 8, 300, 8492, 128  # (partials of 32 and more splits: 158 MB and more; a slot's tensors: 20 MB)
    q, k, v = (torch.randn(1, h, n, d).bfloat16().pin_memory() for h, n in ((H, Nq), (Hk, Nk), (Hk, Nk)))
    api.flash_attn_forward_host(q, k, v, num_splits=1)  # (kernels and streams are in place)
    L.fa_fwd_host_release()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    o, _ = api.flash_attn_forward_host(q, k, v, num_splits=num_splits)
    held = before - torch.cuda.mem_get_info()[0]
    L.fa_fwd_host_release()
    assert 0 < held < 100 << 20, held
    import flash_attn_b200 as fa
    want = fa.flash_attn_forward(q.cuda(), k.cuda(), v.cuda())[0].cpu()
    assert (o.float() - want.float()).abs().max() <= gpu_util.O_MAX_ABS

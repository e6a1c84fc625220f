"""Query blocks whose keys are shared out over the CTAs of a cluster, and grouped queries stacked into common query
tiles: few query blocks against many keys, so that every case is split.  Same tolerances as the unsplit kernel."""
import pytest
import torch

import gpu_util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    dict(H=8, heads_k=2, Nq=130, Nk=3000, d=128, causal=True, q_pos0=2870),                  # stacked, tiles across heads
    dict(H=4, Nq=100, Nk=2000, d=64, dtype="float16"),                                       # one query tile a unit
    dict(H=6, heads_k=2, Nq=40, Nk=2500, d=128, causal=True, q_pos0=2460, window=(300, 0)),  # stacked, left window
    dict(H=6, heads_k=2, Nq=43, Nk=900, d=64, q_pos0=400, window=(100, 60)),                 # stacked, both windows
    dict(H=4, heads_k=2, Nq=300, Nk=2500, d=64, causal=True, q_pos0=2200, alibi=True),       # slopes go by head: not stacked
    dict(H=2, Nq=257, Nk=1500, d=96, dtype="float16", window=(200, 100), q_pos0=600),
    dict(H=8, heads_k=1, Nq=20, Nk=700, d=31, dtype="float16", out_dtype=torch.float32),     # padded rows, scalar stores
    dict(H=2, Nq=400, Nk=2000, d=128, causal=True, q_pos0=50),                               # parts without a visible key
    dict(H=4, Nq=384, Nk=1100, d=128, num_splits=3),
    dict(H=16, heads_k=4, Nq=62, Nk=1300, d=128, causal=True, q_pos0=1238),                  # two stacked tiles, one pair
    dict(H=128, Nq=257, Nk=300, d=100, dtype="float16", out_dtype=torch.float32),            # padded rows, unsplit
    dict(H=2, Nq=9, Nk=1100, d=20, dtype="float16"),                                         # fewest rows, 4-byte rows of O
])
def test_split_and_stacked_blocks_match_the_oracle(case):
    case = dict(case)
    H, Nq, Nk, d = (case.pop(x) for x in ("H", "Nq", "Nk", "d"))
    case.setdefault("num_splits", 0)
    gpu_util.assert_close(gpu_util.run_case(1, H, Nq, Nk, d, seed=71, **case), str((H, Nq, Nk, d, case)))


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

"""The give-up path of the kernels' bounded waits, exercised on a GPU without faulting, trapping or
hanging anything: a test build of the library (-DFA_TEST_SHORT_WAIT: waits give up after about 2 ms)
whose TMA producer is told to leave out the loads of a KV tile and of those behind it.  The MMA warp's wait for that tile
runs out, the kernel records 100 + n in the status word, drains, frees its tensor memory and returns;
the host-buffer entry point turns the word into FA_ERR_DEVICE_TIMEOUT; the next ordinary launch on
the same device and context is correct."""
import ctypes
import os

import numpy as np
import pytest
import torch

import gpu_util
import oracle_lib
import synth
from plan_util import plan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def test_lib():
    from flash_attn_b200 import _lib, build
    path = build.TEST_LIB
    if not os.path.exists(path):
        path = build.build_test_variant()
    L = ctypes.CDLL(path)
    pp = ctypes.POINTER(_lib.FwdParams)
    for name in ("fa_fwd", "fa_fwd_host"):
        getattr(L, name).argtypes = [pp]
        getattr(L, name).restype = ctypes.c_int
    for name in ("fa_test_skip_kv_tile", "fa_test_skip_decode_tile"):
        getattr(L, name).argtypes = [ctypes.c_int]
        getattr(L, name).restype = ctypes.c_int
    L.fa_fwd_workspace_bytes.argtypes = [pp]
    L.fa_fwd_workspace_bytes.restype = ctypes.c_size_t
    return L


def _params(q, k, v, o, lse, status=None):
    from flash_attn_b200 import _lib
    B, H, N, d = q.shape
    p = _lib.FwdParams()
    p.q, p.k, p.v, p.o, p.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr()
    p.dtype = p.o_dtype = _lib.FA_DTYPE_BF16
    p.batch, p.heads, p.seqlen_q, p.seqlen_k, p.head_dim = B, H, N, k.shape[2], d
    p.softmax_scale = d ** -0.5
    p.window_left = p.window_right = -1
    p.num_splits = 1
    if status is not None:
        p.status = status.data_ptr()
    if q.is_cuda:
        p.stream = torch.cuda.current_stream().cuda_stream
    return p


def test_a_wait_that_runs_out_is_reported_and_the_device_stays_usable(test_lib):
    L = test_lib
    B, H, N, d = 1, 2, 256, 128
    qh, kh, vh = synth.qkv(40, B, H, N, N, d, "bfloat16")
    q, k, v = (gpu_util.to_dev(x, "bfloat16") for x in (qh, kh, vh))
    o = torch.empty_like(q)
    lse = torch.empty((B, H, N), device="cuda", dtype=torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        assert L.fa_test_skip_kv_tile(1) == 0  # the second KV tile of every CTA never arrives
        assert L.fa_fwd(ctypes.byref(_params(q, k, v, o, lse, status))) == 0  # the launch itself succeeds
        torch.cuda.synchronize()  # ... and the kernel returns by itself
        code = int(status.item())
        assert 100 < code < 200, code  # a wait of the tiled kernel gave up
        # the synchronous host-buffer entry point reads the word itself
        pin = lambda x: torch.from_numpy(x).bfloat16().pin_memory()
        hq, hk, hv = pin(qh), pin(kh), pin(vh)
        ho = torch.empty((B, H, N, d), dtype=torch.bfloat16).pin_memory()
        hl = torch.empty((B, H, N), dtype=torch.float32).pin_memory()
        assert L.fa_fwd_host(ctypes.byref(_params(hq, hk, hv, ho, hl))) == -5  # FA_ERR_DEVICE_TIMEOUT
    finally:
        assert L.fa_test_skip_kv_tile(-1) == 0
    # same device, same context, same library: an ordinary launch is correct again
    status.zero_()
    assert L.fa_fwd(ctypes.byref(_params(q, k, v, o, lse, status))) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want_o, want_lse = oracle_lib.forward(qh, kh, vh, d ** -0.5)
    err = np.abs(o.float().cpu().numpy() - want_o)
    assert err.max() <= gpu_util.O_MAX_ABS and err.mean() <= gpu_util.O_MEAN_ABS
    assert np.abs(lse.cpu().numpy() - want_lse).max() <= gpu_util.LSE_ABS
    assert L.fa_fwd_host(ctypes.byref(_params(hq, hk, hv, ho, hl))) == 0
    assert np.abs(ho.float().numpy() - want_o).max() <= gpu_util.O_MAX_ABS


@pytest.mark.parametrize("skip,H,Hk,Nq,Nk,d", [
    ("fa_test_skip_kv_tile", 8, 8, 256, 2400, 128),     # the parts of a query block, merged in their cluster
    ("fa_test_skip_kv_tile", 8, 8, 100, 2400, 64),
    ("fa_test_skip_decode_tile", 2, 2, 1, 1100, 128),   # decode: eight parts in a cluster, of which one gives up
    ("fa_test_skip_decode_tile", 4, 1, 1, 262244, 64),   # ... and parts that the combine kernel merges
])
def test_a_part_that_gave_up_leaves_no_plausible_row(test_lib, skip, H, Hk, Nq, Nk, d):
    """The other parts of the keys are complete, so only the part that gave up can keep the merged rows from looking
    like a result: its sum is NaN."""
    from flash_attn_b200 import _lib
    L = test_lib
    qh, kh, vh = synth.qkv(41, 1, H, Nq, Nk, d, "bfloat16")
    kh, vh = np.ascontiguousarray(kh[:, :Hk]), np.ascontiguousarray(vh[:, :Hk])
    q, k, v = (gpu_util.to_dev(x, "bfloat16") for x in (qh, kh, vh))
    o = torch.zeros_like(q)
    lse = torch.zeros((1, H, Nq), device="cuda", dtype=torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = _params(q, k, v, o, lse, status)
    p.heads_k, p.num_splits = Hk, 0
    need = L.fa_fwd_workspace_bytes(ctypes.byref(p))
    ws = torch.empty(max(need, 16), device="cuda", dtype=torch.uint8)
    p.workspace, p.workspace_bytes = ws.data_ptr(), need
    # a KV tile (decode: a slot of the K/V stream) that only the longest parts have
    parts, tiles = plan(1, H, Nq, Nk, d, heads_k=Hk).parts, (Nk + 127) // 128
    assert parts > 1 and tiles % parts != 0
    tile = tiles // parts if skip == "fa_test_skip_kv_tile" else 3 if Nk == 1100 else 65
    try:
        assert getattr(L, skip)(tile) == 0
        assert L.fa_fwd(ctypes.byref(p)) == 0
        torch.cuda.synchronize()
        code = int(status.item())
        assert (100 < code < 200) if Nq > 8 else (200 < code < 300), code
        assert torch.isnan(o).all() and not torch.isfinite(lse).any()
    finally:
        assert getattr(L, skip)(-1) == 0
    status.zero_()
    assert L.fa_fwd(ctypes.byref(p)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want_o, want_lse = oracle_lib.forward(qh, np.repeat(kh, H // Hk, 1), np.repeat(vh, H // Hk, 1), d ** -0.5)
    assert np.abs(o.float().cpu().numpy() - want_o).max() <= gpu_util.O_MAX_ABS
    assert np.abs(lse.cpu().numpy() - want_lse).max() <= gpu_util.LSE_ABS


@pytest.mark.parametrize("H,Nq,d,skip,causal,out_dtype,p_dropout", [
    (160, 256, 128, 1, False, torch.bfloat16, 0.0),  # (two query tiles a CTA)
    (120, 300, 64, 0, True, torch.float32, 0.0),     # (a CTA whose second query tile does not exist; the first tile of the walk)
    (3, 300, 128, 1, False, torch.float32, 0.0),     # (one query tile a CTA, a ring of one stage)
    (3, 300, 96, 1, False, torch.bfloat16, 0.1),
])
def test_a_block_that_gave_up_leaves_no_running_result(test_lib, H, Nq, d, skip, causal, out_dtype, p_dropout):
    """The block before it is complete, and so are the ones behind it: neither may make its rows look like a result."""
    from flash_attn_b200 import _lib
    L = test_lib
    Nk = 500
    assert plan(1, H, Nq, Nk, d, causal=causal, q_pos0=3 * Nk, p_dropout=p_dropout, num_splits=1, accum=True).columns == (128 if H == 3 else 256)
    qh, kh, vh = synth.qkv(42, 1, 3, Nq, 4 * Nk, d, "bfloat16")  # (the oracle's heads, again and again)
    q, k, v = (gpu_util.to_dev(x, "bfloat16")[:, torch.arange(H) % 3].contiguous() for x in (qh, kh, vh))
    acc = (torch.empty((1, H, Nq, d), device="cuda"), torch.empty((1, H, Nq), device="cuda"))
    o = torch.zeros((1, H, Nq, d), device="cuda", dtype=out_dtype)
    lse = torch.zeros((1, H, Nq), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def block(i, first, final):
        kb, vb = (x[:, :, i * Nk:(i + 1) * Nk].contiguous() for x in (k, v))
        p = _params(q, kb, vb, o, lse, status)
        p.o_dtype = _lib.FA_DTYPE_FP32 if out_dtype is torch.float32 else _lib.FA_DTYPE_BF16
        p.p_dropout, p.seed = p_dropout, 3
        p.is_causal, p.q_pos0, p.k_pos0 = int(causal), 3 * Nk, i * Nk  # (with a causal mask no query sees the fourth block's end)
        p.accum_o, p.accum_lse = acc[0].data_ptr(), acc[1].data_ptr()
        p.accum_flags = (_lib.FA_ACCUM_FIRST if first else 0) | (_lib.FA_ACCUM_FINAL if final else 0)
        assert L.fa_fwd(ctypes.byref(p)) == 0
        torch.cuda.synchronize()

    def gives_up(i, first, final):
        status.zero_()
        try:
            assert L.fa_test_skip_kv_tile(skip) == 0
            block(i, first, final)
        finally:
            assert L.fa_test_skip_kv_tile(-1) == 0
        assert 100 < int(status.item()) < 200

    for first in (False, True):  # a block in the middle, the first one, and what the launches behind it make of the pair
        if not first:
            block(0, True, False)
            assert torch.isfinite(acc[0]).all() and torch.isfinite(acc[1]).all()
        gives_up(1, first, False)
        assert torch.isnan(acc[0]).all() and torch.isnan(acc[1]).all()
        status.zero_()
        block(2, False, False)
        assert torch.isnan(acc[0]).all() and torch.isnan(acc[1]).all()
        block(3, False, True)
        assert torch.isnan(o).all() and torch.isnan(lse).all() and int(status.item()) == 0
    block(0, True, False)
    gives_up(1, False, True)  # the last block
    assert torch.isnan(o).all() and torch.isnan(lse).all() and torch.isnan(acc[1]).all()
    status.zero_()
    for i in range(4):
        block(i, i == 0, i == 3)
    want_o, want_lse = oracle_lib.forward(qh, kh, vh, d ** -0.5, causal=causal, q_pos0=3 * Nk)
    assert int(status.item()) == 0
    if p_dropout > 0.0:  # (each block's launch has a mask of its own)
        assert torch.isfinite(o).all()
        return
    assert np.abs(o[:, :3].float().cpu().numpy() - want_o).max() <= gpu_util.O_MAX_ABS
    assert np.abs(lse[:, :3].cpu().numpy() - want_lse).max() <= gpu_util.LSE_ABS


@pytest.mark.parametrize("H,Hk,Nq,Nk,d,causal", [
    (4, 4, 300, 300, 31, False),     # padded rows
    (300, 300, 200, 300, 31, False),  # ... in CTAs of two query tiles
    (512, 64, 48, 546, 128, True),   # stacked heads
])
def test_an_unsplit_staged_launch_that_gave_up_leaves_no_plausible_row(test_lib, H, Hk, Nq, Nk, d, causal):
    """Each warp finishes its own rows behind its own waits; those that ran out make them NaN."""
    L = test_lib
    got = plan(1, H, Nq, Nk, d, heads_k=Hk, causal=causal, q_pos0=Nk - Nq if causal else 0)
    assert got.parts == 1 and got.staged and bool(got.stacked_rows) == (Hk < H)
    qh, kh, vh = synth.qkv(43, 1, 4, Nq, Nk, d, "bfloat16")
    q = gpu_util.to_dev(qh, "bfloat16")[:, torch.arange(H) % 4].contiguous()
    k, v = (gpu_util.to_dev(x, "bfloat16")[:, torch.arange(Hk) % 4].contiguous() for x in (kh, vh))
    o = torch.zeros_like(q)
    lse = torch.zeros((1, H, Nq), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = _params(q, k, v, o, lse, status)
    p.heads_k, p.num_splits, p.is_causal, p.q_pos0 = Hk, 0, int(causal), Nk - Nq if causal else 0
    need = L.fa_fwd_workspace_bytes(ctypes.byref(p))
    ws = torch.empty(max(need, 16), device="cuda", dtype=torch.uint8)
    p.workspace, p.workspace_bytes = ws.data_ptr(), need
    try:
        assert L.fa_test_skip_kv_tile(1) == 0
        assert L.fa_fwd(ctypes.byref(p)) == 0
        torch.cuda.synchronize()
        assert 100 < int(status.item()) < 200
        assert torch.isnan(o).all() and not torch.isfinite(lse).any()
    finally:
        assert L.fa_test_skip_kv_tile(-1) == 0
    status.zero_()
    assert L.fa_fwd(ctypes.byref(p)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and torch.isfinite(o).all()
    want_o, want_lse = oracle_lib.forward(qh[:, :1], kh[:, :1], vh[:, :1], d ** -0.5, causal=causal, q_pos0=Nk - Nq if causal else 0)
    assert np.abs(o[:, :1].float().cpu().numpy() - want_o).max() <= gpu_util.O_MAX_ABS
    assert np.abs(lse[:, :1].cpu().numpy() - want_lse).max() <= gpu_util.LSE_ABS

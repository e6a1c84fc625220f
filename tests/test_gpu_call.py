"""The native call path of flash_attn_forward: what it accepts and refuses, against the C ABI called through ctypes."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv(d=64, dtype=torch.float16, nq=40, hk=2):
    g = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randn(1, h, n, d, device="cuda", dtype=torch.float32, generator=g).to(dtype) for h, n in ((4, nq), (hk, 300), (hk, 300))]


def _by_ctypes(q, k, v, o, lse, **kw):
    from flash_attn_b200 import _lib
    L = _lib.load()
    p = _lib.FwdParams(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), o=o.data_ptr(), lse=lse.data_ptr(),
                       dtype=1 if q.dtype is torch.bfloat16 else 0, o_dtype={torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}[o.dtype],
                       batch=q.shape[0], heads=q.shape[1], heads_k=k.shape[1], seqlen_q=q.shape[2], seqlen_k=k.shape[2],
                       head_dim=q.shape[3], softmax_scale=q.shape[3] ** -0.5, window_left=-1, window_right=-1, num_splits=1)
    for name, x in kw.items():
        setattr(p, name, x)
    need = L.fa_fwd_workspace_bytes(ctypes.byref(p))
    room = torch.empty(max(need, 16), device="cuda", dtype=torch.uint8)
    p.workspace, p.workspace_bytes, p.stream = room.data_ptr(), room.numel(), torch.cuda.current_stream().cuda_stream
    assert L.fa_fwd(ctypes.byref(p)) == 0
    torch.cuda.synchronize()
    return o, lse


@pytest.mark.parametrize("d,args,fields", [
    (64, dict(), dict()),
    (64, dict(softmax_scale=np.float64(0.25), causal=1, window=[np.int64(50), 0], q_pos0=np.int32(200)),
     dict(softmax_scale=0.25, is_causal=1, window_left=50, window_right=0, q_pos0=200)),
    (64, dict(causal=True, window=torch.tensor([50, -1])), dict(is_causal=1, window_left=50)),
    (64, dict(window={0: 20, 1: 30}), dict(window_left=20, window_right=30)),
    (128, dict(p_dropout=0.25, seed=-3, offset=2 ** 64 + 8, launch_index=1), dict(p_dropout=0.25, seed=2 ** 64 - 3, offset=8, launch_index=1)),
    (128, dict(p_dropout=0.5, seed=7, num_splits=2, unit0=5), dict(p_dropout=0.5, seed=7, num_splits=2, unit0=5)),
    (50, dict(out_dtype=torch.float32, num_splits=0), dict(num_splits=0)),
])
def test_arguments_reach_the_library_as_they_are(d, args, fields):
    import flash_attn_b200 as fa
    q, k, v = _qkv(d)
    o, lse = fa.flash_attn_forward(q, k, v, **args)
    want_o, want_lse = _by_ctypes(q, k, v, torch.empty_like(o), torch.empty_like(lse), **fields)
    assert torch.equal(o, want_o) and torch.equal(lse, want_lse)
    mine = torch.empty_like(o)
    again = fa.flash_attn_forward(q, k, v, out=mine, return_lse=False, **args)
    assert again[0] is mine and again[1] is None and torch.equal(mine, o)


def test_slopes_of_another_kind_stream_and_status():
    import flash_attn_b200 as fa
    q, k, v = _qkv(64, torch.bfloat16)
    slopes = [0.5, 0.25, 0.125, 0.0625]
    status = torch.zeros(1, device="cuda", dtype=torch.int32)
    o = fa.flash_attn_forward(q, k, v, alibi_slopes=torch.tensor(slopes, dtype=torch.float64), status=status)[0]
    dev = torch.tensor(slopes, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        assert torch.equal(o, fa.flash_attn_forward(q, k, v, alibi_slopes=dev)[0])
    torch.cuda.current_stream().wait_stream(s)
    assert int(status) == 0


@pytest.mark.parametrize("change,error", [
    (lambda q, k, v: dict(q=q.cpu()), ValueError),
    (lambda q, k, v: dict(q=q[0]), ValueError),
    (lambda q, k, v: dict(k=k[:, :, :8]), ValueError),
    (lambda q, k, v: dict(q=q.float()), ValueError),
    (lambda q, k, v: dict(v=v.bfloat16()), ValueError),
    (lambda q, k, v: dict(q=q.transpose(1, 2)), ValueError),
    (lambda q, k, v: dict(q=q[:, :3].contiguous()), ValueError),
    (lambda q, k, v: dict(out=torch.empty(q.shape, device="cuda", dtype=torch.float64)), KeyError),
    (lambda q, k, v: dict(accum=(torch.empty(q.shape, device="cuda", dtype=q.dtype), torch.empty(q.shape[:3], device="cuda"))), ValueError),
    (lambda q, k, v: dict(accum=(torch.empty(q.shape, device="cuda"),)), ValueError),
    (lambda q, k, v: dict(window=(1,)), IndexError),
    (lambda q, k, v: dict(p_dropout="much"), ValueError),
    (lambda q, k, v: dict(p_dropout=1.5), RuntimeError),
    (lambda q, k, v: dict(softmax_scale=-1.0), RuntimeError),
])
def test_what_was_refused_stays_refused(change, error):
    import flash_attn_b200 as fa
    q, k, v = _qkv()
    with pytest.raises(error):
        fa.flash_attn_forward(**{**dict(q=q, k=k, v=v), **change(q, k, v)})


# what lies outside a tensor, or in memory that the device does not reach, must not come to a kernel: nothing is launched here
@pytest.mark.parametrize("change", [
    lambda q, k, v: dict(out=torch.empty(q.numel() - 1, device="cuda", dtype=q.dtype)),
    lambda q, k, v: dict(out=torch.empty(q[:, :2].shape, device="cuda", dtype=q.dtype)),
    lambda q, k, v: dict(out=torch.empty(q.shape, dtype=q.dtype)),
    lambda q, k, v: dict(k=k.cpu()),
    lambda q, k, v: dict(v=v.cpu()),
    lambda q, k, v: dict(alibi_slopes=torch.ones(3)),
    lambda q, k, v: dict(status=torch.zeros(0, device="cuda", dtype=torch.int32)),
    lambda q, k, v: dict(status=torch.zeros(1, device="cuda", dtype=torch.int16)),
    lambda q, k, v: dict(status=torch.zeros(8, device="cuda", dtype=torch.int8)[1:]),
    lambda q, k, v: dict(status=torch.zeros(1, dtype=torch.int32)),
    lambda q, k, v: dict(num_splits=2, workspace=torch.empty(1 << 24, dtype=torch.uint8)),
    lambda q, k, v: dict(accum=(torch.empty(q.shape), torch.empty(q.shape[:3], device="cuda")), accum_first=True),
    lambda q, k, v: dict(accum=(torch.empty(q.shape, device="cuda"), torch.empty(q.shape[:3])), accum_first=True),
])
def test_memory_that_a_kernel_may_not_touch_is_refused(change):
    import flash_attn_b200 as fa
    q, k, v = _qkv()
    with pytest.raises(ValueError):
        fa.flash_attn_forward(**{**dict(q=q, k=k, v=v), **change(q, k, v)})


def test_memory_of_another_shape_or_place_that_serves_is_taken():
    import flash_attn_b200 as fa
    q, k, v = _qkv()
    want = fa.flash_attn_forward(q, k, v)[0]
    flat = torch.full((q.numel() + 8,), 7.0, device="cuda", dtype=q.dtype)
    assert fa.flash_attn_forward(q, k, v, out=flat)[0] is flat
    assert torch.equal(flat[:-8].view_as(q), want) and bool((flat[-8:] == 7.0).all())
    status = torch.zeros(1, dtype=torch.int32).pin_memory()
    assert torch.equal(fa.flash_attn_forward(q, k, v, status=status)[0], want)
    slopes = torch.full((4,), 0.25)
    assert torch.equal(*(fa.flash_attn_forward(q, k, v, alibi_slopes=x)[0] for x in (slopes, torch.cat([slopes, slopes]))))
    split = fa.flash_attn_forward(q, k, v, num_splits=2)[0]
    for room in (torch.empty(1, device="cuda").expand(1 << 22), torch.empty(4)):  # (no room: the call takes its own)
        assert torch.equal(fa.flash_attn_forward(q, k, v, num_splits=2, workspace=room)[0], split)
    torch.cuda.synchronize()
    assert int(status) == 0


def test_host_buffers_too_small_for_the_call_are_refused():
    import flash_attn_b200 as fa
    q, k, v = (x.cpu() for x in _qkv())
    for bad in (dict(out=torch.empty(q.numel() - 1, dtype=q.dtype)), dict(alibi_slopes=torch.ones(3))):
        with pytest.raises(ValueError):
            fa.flash_attn_forward_host(q, k, v, **bad)

"""fa_fwd_plan for a shape, as a FwdPlan: how the library would cut the call on a B200 (148 SMs unless told otherwise)."""
import ctypes

from flash_attn_b200 import _lib

# clusters of 0, 1, ... 16 CTAs that a B200 holds at once, one CTA an SM (as its runtime reports them)
B200_CLUSTERS = (0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7)


def plan(B, H, Nq, Nk, d, heads_k=0, causal=False, window=(-1, -1), alibi=False, p_dropout=0.0, num_splits=0, q_pos0=0,
         k_pos0=0, fp32_out=False, accum=False, sms=148, clusters=B200_CLUSTERS):
    p = _lib.FwdParams()
    p.q = p.k = p.v = p.o = 4096  # (not followed)
    p.batch, p.heads, p.heads_k, p.seqlen_q, p.seqlen_k, p.head_dim = B, H, heads_k, Nq, Nk, d
    p.dtype = _lib.FA_DTYPE_BF16
    p.o_dtype = _lib.FA_DTYPE_FP32 if fp32_out else p.dtype
    p.softmax_scale, p.is_causal, p.window_left, p.window_right = d ** -0.5, int(causal), *window
    p.alibi_slopes = 4096 if alibi else None
    p.p_dropout, p.num_splits, p.q_pos0, p.k_pos0 = p_dropout, num_splits, q_pos0, k_pos0
    if accum:
        p.accum_o = p.accum_lse = 4096
        p.accum_flags = _lib.FA_ACCUM_FIRST | _lib.FA_ACCUM_FINAL
    out = _lib.FwdPlan()
    rc = _lib.load().fa_fwd_plan(ctypes.byref(p), sms, (ctypes.c_int * 17)(*clusters), ctypes.byref(out))
    assert rc == 0, _lib.strerror(rc)
    return out

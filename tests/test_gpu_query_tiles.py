"""One query tile a CTA or two: the launch takes either by its size, with the same bits.  A launch of many units runs two tiles a
CTA, each of its units alone one; ragged rows and keys, odd numbers of tiles, masks, dropout streams, and the oracle on one unit."""
import numpy as np
import pytest
import torch

import gpu_util
import oracle_lib
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nq,Nk,d,dtype,kw", [
    (257, 257, 64, "float16", dict()),
    (300, 700, 128, "bfloat16", dict(causal=True, q_pos0=400)),
    (384, 384, 96, "bfloat16", dict(causal=True)),
    (640, 129, 128, "float16", dict()),
    (513, 1000, 64, "bfloat16", dict(window=(200, 30), q_pos0=300)),
    (400, 400, 32, "float16", dict(causal=True, p_dropout=0.2, seed=9)),
    (260, 520, 128, "bfloat16", dict(p_dropout=0.1, seed=4)),
    (900, 900, 128, "bfloat16", dict(causal=True, window=(250, 0), p_dropout=0.5, seed=1)),
])
def test_units_of_a_large_launch_equal_the_same_units_alone(Nq, Nk, d, dtype, kw):
    import flash_attn_b200 as fa
    heads = 2 * 148 // ((Nq + 127) // 128) + 1  # more tiles than one a CTA would have resident
    g = torch.Generator(device="cuda").manual_seed(7)
    dt = getattr(torch, dtype)
    q, k, v = (torch.randn(1, heads, n, d, device="cuda", generator=g).to(dt) for n in (Nq, Nk, Nk))
    q0, k0, v0 = synth.qkv(70, 1, 1, Nq, Nk, d, dtype, 0.7)
    for x, x0 in ((q, q0), (k, k0), (v, v0)):
        x[0, 0] = gpu_util.to_dev(x0, dtype)[0, 0]
    o, lse = fa.flash_attn_forward(q, k, v, **kw)
    for u in (0, 1, heads // 2, heads - 1):
        qu, ku, vu = (x[:, u:u + 1].contiguous() for x in (q, k, v))
        acc = (torch.empty(qu.shape, device="cuda"), torch.empty(qu.shape[:3], device="cuda"))  # (such a launch is never split)
        ou, lu = fa.flash_attn_forward(qu, ku, vu, unit0=u, accum=acc, accum_first=True, accum_final=True, **kw)
        assert torch.equal(ou[0, 0], o[0, u]) and torch.equal(lu[0, 0], lse[0, u]), u
    opts = {n: x for n, x in kw.items()}
    if "p_dropout" in opts:
        opts["p_dropout"] = float(np.float32(opts["p_dropout"]))
    want_o, want_lse = oracle_lib.forward(q0, k0, v0, d ** -0.5, **opts)
    assert np.abs(o[:, :1].float().cpu().numpy() - want_o).max() <= gpu_util.O_MAX_ABS
    fin = np.isfinite(want_lse)
    assert np.abs(lse[:, :1].cpu().numpy()[fin] - want_lse[fin]).max() <= gpu_util.LSE_ABS

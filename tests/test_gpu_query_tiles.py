"""One query tile a CTA or two: the launch takes either by its size, without ALiBi with the same bits (with it, two-tile CTAs add
the bias in the tensor core).  A launch of many units runs two tiles a CTA, each of its units alone one; ragged rows and keys,
odd numbers of tiles, masks, dropout streams, and the oracle on one unit."""
import numpy as np
import pytest
import torch

import gpu_util
import oracle_lib
import synth
from plan_util import plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nq,Nk,d,dtype,kw", [
    (257, 257, 64, "float16", dict()),
    (300, 300, 128, "bfloat16", dict(causal=True, q_pos0=100)),
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
    cut = dict(num_splits=1, **{n: x for n, x in kw.items() if n != "seed"})
    assert plan(1, heads, Nq, Nk, d, **cut).columns == 256 and plan(1, 1, Nq, Nk, d, accum=True, **cut).columns == 128
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


def test_alibi_in_ctas_of_one_tile_and_of_two():
    import flash_attn_b200 as fa
    Nq, Nk, d, heads = 300, 400, 64, 99
    assert plan(1, heads, Nq, Nk, d, num_splits=1, causal=True, alibi=True).columns == 256
    assert plan(1, 3, Nq, Nk, d, num_splits=1, causal=True, alibi=True, accum=True).columns == 128
    q0, k0, v0 = synth.qkv(71, 1, 3, Nq, Nk, d, "bfloat16", 0.7)
    q, k, v = (gpu_util.to_dev(x, "bfloat16") for x in (q0, k0, v0))
    slopes = torch.tensor([0.5, 0.0625, 1.5], device="cuda")
    acc = (torch.empty(q.shape, device="cuda"), torch.empty(q.shape[:3], device="cuda"))
    alone = fa.flash_attn_forward(q, k, v, causal=True, alibi_slopes=slopes, accum=acc, accum_first=True, accum_final=True)
    many = fa.flash_attn_forward(*(x.repeat(1, heads // 3, 1, 1) for x in (q, k, v)), causal=True, alibi_slopes=slopes.repeat(heads // 3))
    want_o, want_lse = oracle_lib.forward(q0, k0, v0, d ** -0.5, causal=True, alibi_slopes=slopes.cpu().numpy())
    for o, lse in (alone, (many[0][:, -3:], many[1][:, -3:])):
        assert np.abs(o.float().cpu().numpy() - want_o).max() <= gpu_util.O_MAX_ABS
        assert np.abs(lse.cpu().numpy() - want_lse).max() <= gpu_util.LSE_ABS

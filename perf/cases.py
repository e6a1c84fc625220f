"""What the speed of the forward pass is measured on: the calls that programs make of this package, from a
single small launch to long sequences, with their work, their tolerances and a generator of more of the same.

A case is a plain dict:
  kind   "forward": one flash_attn_forward on device tensors
         "blocks":  the key blocks of one long sequence arriving one launch at a time, merged into a running result
         "host":    flash_attn_forward_host on pinned host tensors
  dtype  of Q, K, V;  out_fp32: O in fp32 instead
  B, H, Hk, Nq, Nk, d;  causal, window_left, window_right, alibi, p_dropout, splits, q_pos0 as in flash_attn_forward
  blocks number of key blocks ("blocks" only; Nk is the length of one)
  sigma  standard deviation of the inputs
"""
import math

import numpy as np
import torch

import flash_attn_b200 as fa
from flash_attn_b200 import api

_BASE = dict(kind="forward", dtype="bfloat16", out_fp32=False, B=1, H=1, Hk=1, Nq=1, Nk=1, d=128, causal=False,
             window_left=-1, window_right=-1, alibi=False, p_dropout=0.0, splits=1, q_pos0=0, blocks=1, sigma=1.0)


def _case(**kw):
    c = dict(_BASE)
    c.update(kw)
    if "Hk" not in kw:
        c["Hk"] = c["H"]
    return c


# ------------------------------------------------------------------ the families
# Each family is one use; `r` (a random.Random) varies it over its range.
def _log_int(r, lo, hi):
    return int(round(math.exp(r.uniform(math.log(lo), math.log(hi)))))


def _small(r):
    return _case(dtype=r.choice(["float16", "bfloat16"]), B=r.randint(1, 4), H=r.choice([4, 8, 12, 16]),
                 Nq=(n := _log_int(r, 16, 512)), Nk=n, d=r.choice([32, 64, 64, 96, 128]), causal=r.random() < 0.5)


def _dropout(r):
    n = _log_int(r, 256, 4096)
    return _case(dtype=r.choice(["bfloat16", "bfloat16", "float16"]), B=max(1, min(16, _log_int(r, 2048, 16384) // n)),
                 H=r.choice([8, 12, 16]), Nq=n, Nk=n, d=r.choice([64, 128, 128]), causal=r.random() < 0.75,
                 p_dropout=r.choice([0.1, 0.1, 0.2, 0.5]))


def _local(r):
    n = _log_int(r, 1024, 8192)
    return _case(B=r.randint(1, 4), H=r.choice([16, 32]), Nq=n, Nk=n, d=r.choice([64, 128, 128]), causal=True,
                 window_left=_log_int(r, 128, 2048), window_right=0, alibi=r.random() < 0.75)


def _decode(r):
    nk = _log_int(r, 1024, 32768)
    b = max(1, min(64, _log_int(r, 16384, 524288) // nk))
    return _case(dtype=r.choice(["bfloat16", "bfloat16", "float16"]), B=b, H=r.choice([16, 32]), Nq=1, Nk=nk,
                 d=r.choice([64, 128, 128]), splits=r.choice([16, 16, 8, 0]))


def _decode_gqa(r):
    nk = _log_int(r, 512, 32768)
    h, hk = r.choice([(32, 8), (32, 8), (64, 8), (32, 4), (28, 4)])
    return _case(dtype=r.choice(["bfloat16", "bfloat16", "float16"]), B=max(1, min(64, _log_int(r, 8192, 524288) // nk)),
                 H=h, Hk=hk, Nq=1, Nk=nk, d=r.choice([64, 128, 128]), causal=True, q_pos0=nk - 1, splits=r.choice([0, 0, 1]),
                 window_left=r.choice([-1, -1, -1, 1024]))


def _decode_one(r):
    nk = _log_int(r, 64, 4096)
    h, hk = r.choice([(8, 8), (16, 16), (32, 32), (32, 8)])
    return _case(dtype=r.choice(["bfloat16", "float16"]), B=1, H=h, Hk=hk, Nq=1, Nk=nk, d=r.choice([64, 128]),
                 splits=r.choice([0, 0, 1]))


def _short_query(r):
    nk = _log_int(r, 512, 16384)
    nq = r.randint(2, 8)
    h, hk = r.choice([(32, 8), (32, 8), (32, 32), (16, 4), (64, 8)])
    return _case(dtype=r.choice(["bfloat16", "bfloat16", "float16"]), B=max(1, min(32, _log_int(r, 8192, 131072) // nk)),
                 H=h, Hk=hk, Nq=nq, Nk=nk, d=r.choice([64, 128, 128]), causal=True, q_pos0=nk - nq, splits=0)


def _prefill_64(r):
    n = _log_int(r, 512, 8192)
    h, hk = r.choice([(16, 16), (16, 16), (32, 8), (12, 12)])
    return _case(dtype=r.choice(["float16", "bfloat16"]), B=max(1, min(16, _log_int(r, 4096, 32768) // n)), H=h, Hk=hk,
                 Nq=n, Nk=n, d=64, causal=r.random() < 0.7)


def _odd_head_dim(r):
    n = _log_int(r, 129, 2048)
    return _case(dtype=r.choice(["float16", "float16", "bfloat16"]), out_fp32=r.random() < 0.75, B=r.randint(1, 4), H=8,
                 Nq=n, Nk=n, d=r.choice([20, 31, 31, 50, 100, 125]), causal=r.random() < 0.4, splits=r.choice([1, 1, 0]))


def _chunk(r):
    nq = _log_int(r, 16, 1024)
    nk = nq + _log_int(r, 1024, 32768)
    h, hk = r.choice([(32, 8), (32, 8), (32, 32), (64, 8)])
    return _case(dtype=r.choice(["bfloat16", "bfloat16", "float16"]), B=max(1, min(8, _log_int(r, 4096, 65536) // nk)),
                 H=h, Hk=hk, Nq=nq, Nk=nk, d=r.choice([64, 128, 128]), causal=True, q_pos0=nk - nq, splits=r.choice([0, 0, 1]))


def _blocks(r):
    c = _log_int(r, 1024, 8192)
    h, hk = r.choice([(32, 32), (32, 8), (16, 16)])
    n = r.randint(2, 3)
    return _case(kind="blocks", B=1, H=h, Hk=hk, Nq=c, Nk=c, d=r.choice([64, 128, 128]), causal=True, blocks=n,
                 q_pos0=(n - 1) * c, sigma=0.5)


def _host(r):
    n = _log_int(r, 256, 2048)
    return _case(kind="host", dtype=r.choice(["bfloat16", "float16"]), B=max(1, min(8, _log_int(r, 1024, 16384) // n)),
                 H=r.choice([8, 16]), Nq=n, Nk=n, d=r.choice([64, 128]), causal=True, p_dropout=r.choice([0.0, 0.1]))


_FAMILIES = [_small, _dropout, _local, _decode, _decode_gqa, _decode_one, _short_query, _prefill_64, _odd_head_dim,
             _chunk, _blocks, _host]


def listed():
    return [
        # the smallest ordinary call: a test-sized layer, all latency and launch cost
        _case(name="small_fp16", dtype="float16", H=4, Nq=256, Nk=256, d=64),
        # a training forward: causal with dropout on the attention weights
        _case(name="causal_dropout", B=8, H=16, Nq=2048, Nk=2048, causal=True, p_dropout=0.1),
        # sliding-window layers with ALiBi
        _case(name="local_alibi", B=4, H=32, Nq=8192, Nk=8192, causal=True, window_left=1024, window_right=0, alibi=True),
        # decoding a full batch against long caches, a K/V head per query head, the caller's own split count
        _case(name="decode_long", B=16, H=32, Nq=1, Nk=32768, splits=16),
        # a serving step: grouped-query decode of a medium batch, ragged cache length, the library's split count
        _case(name="decode_gqa", B=16, H=32, Hk=8, Nq=1, Nk=4097, causal=True, q_pos0=4096, splits=0),
        # one user, short cache: the shortest decode step
        _case(name="decode_one", B=1, H=32, Hk=8, Nq=1, Nk=1000, splits=0),
        # the verification step of speculative decoding: a few query rows at the end of the cache
        _case(name="verify_gqa", B=8, H=32, Hk=8, Nq=4, Nk=8000, causal=True, q_pos0=7996, splits=0),
        # prefill of a model with 64-wide heads
        _case(name="prefill_d64", dtype="float16", B=4, H=16, Nq=4096, Nk=4096, d=64, causal=True),
        # head dimension and length of no round size, fp16 in and fp32 out
        _case(name="odd_fp32_out", dtype="float16", out_fp32=True, B=1, H=8, Nq=1021, Nk=1021, d=31),
        # chunked prefill: a chunk of new rows against a cache that is already there
        _case(name="chunk_gqa", B=1, H=32, Hk=8, Nq=300, Nk=8492, causal=True, q_pos0=8192, splits=0),
        # a long sequence whose key blocks come one launch at a time (the diagonal block, then the ones before it)
        _case(name="key_blocks", kind="blocks", B=1, H=32, Nq=8192, Nk=8192, causal=True, blocks=3, q_pos0=16384, sigma=0.5),
        # the same work on host memory: transfers and kernels pipelined
        _case(name="host_buffers", kind="host", B=8, H=16, Nq=2048, Nk=2048, causal=True, p_dropout=0.1),
    ]


_MOST_FLOPS, _MOST_BYTES = 8.0e11, 4.0e9  # bounds of a drawn case; the largest listed ones are beyond both


def draw(rng):
    while True:
        c = rng.choice(_FAMILIES)(rng)
        w = work(c)
        if w["flops"] <= _MOST_FLOPS and w["bytes"] <= _MOST_BYTES:
            return c


# ------------------------------------------------------------------ what a program has in hand, and the call
def _slopes(h):
    return torch.tensor([2.0 ** (-8.0 * (i + 1) / h) for i in range(h)], dtype=torch.float32, device="cuda")


def prepare(case, seed):
    dt = getattr(torch, case["dtype"])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def make(b, h, n):
        x = torch.empty((b, h, n, case["d"]), device="cuda", dtype=dt)
        return x.normal_(0.0, case["sigma"], generator=g)

    B, H, Hk, Nq, Nk, d = (case[x] for x in ("B", "H", "Hk", "Nq", "Nk", "d"))
    st = dict(case=case, q=make(B, H, Nq), k=[make(B, Hk, Nk) for _ in range(case["blocks"])],
              v=[make(B, Hk, Nk) for _ in range(case["blocks"])], slopes=_slopes(H) if case["alibi"] else None)
    if case["kind"] == "blocks":
        st["acc"] = (torch.empty((B, H, Nq, d), device="cuda", dtype=torch.float32),
                     torch.empty((B, H, Nq), device="cuda", dtype=torch.float32))
    elif case["kind"] == "host":
        for x in ("q", "k", "v"):
            t = st[x] if x == "q" else st[x][0]
            st[x] = torch.empty(t.shape, dtype=dt, pin_memory=True)
            st[x].copy_(t)
        st["out"] = torch.empty((B, H, Nq, d), dtype=dt, pin_memory=True)
    return st


def run(state):
    c = state["case"]
    opts = dict(causal=c["causal"], window=(c["window_left"], c["window_right"]), p_dropout=c["p_dropout"], seed=42)
    if c["kind"] == "host":
        return api.flash_attn_forward_host(state["q"], state["k"], state["v"], num_splits=c["splits"], out=state["out"], **opts)
    if c["kind"] == "blocks":
        # the diagonal block first, then the earlier ones, as a key/value ring brings them
        n = c["blocks"]
        res = None
        for i in range(n):
            res = fa.flash_attn_forward(state["q"], state["k"][i], state["v"][i], q_pos0=c["q_pos0"], k_pos0=(n - 1 - i) * c["Nk"],
                                        accum=state["acc"], accum_first=i == 0, accum_final=i == n - 1, **opts)
        return res
    return fa.flash_attn_forward(state["q"], state["k"][0], state["v"][0], alibi_slopes=state["slopes"], q_pos0=c["q_pos0"],
                                 num_splits=c["splits"], out_dtype=torch.float32 if c["out_fp32"] else None, **opts)


# ------------------------------------------------------------------ work and tolerance
def _visible(case, k_pos0):
    """(unmasked (query, key) pairs of a unit, keys that any query sees) for one key block at k_pos0."""
    q = case["q_pos0"] + np.arange(case["Nq"], dtype=np.int64)
    lo = np.full_like(q, k_pos0)
    hi = np.full_like(q, k_pos0 + case["Nk"] - 1)
    if case["causal"]:
        hi = np.minimum(hi, q)
    if case["window_right"] >= 0:
        hi = np.minimum(hi, q + case["window_right"])
    if case["window_left"] >= 0:
        lo = np.maximum(lo, q - case["window_left"])
    n = np.maximum(0, hi - lo + 1)
    keys = int(hi[n > 0].max() - lo[n > 0].min() + 1) if (n > 0).any() else 0
    return int(n.sum()), keys


def work(case):
    pairs = keys = 0
    for i in range(case["blocks"]):
        p, k = _visible(case, i * case["Nk"])
        pairs += p
        keys += k
    units, rows = case["B"] * case["H"], case["B"] * case["H"] * case["Nq"]
    bytes_ = rows * case["d"] * (2 + (4 if case["out_fp32"] else 2)) + rows * 4 + 2 * case["B"] * case["Hk"] * keys * case["d"] * 2
    if case["alibi"]:
        bytes_ += 4 * case["H"]
    return {"bytes": bytes_, "flops": 4 * case["d"] * units * pairs}


def tolerance(case):
    # Against a 64-bit evaluation, over these cases and 36 drawn ones: the rounding of P and O to the 16-bit type
    # shows as 2.7e-3 (bf16) and 3.1e-4 (fp16, with O in fp32 too) in the 2-norm, and as at most 2.4e-2 / 4.8e-3 of a
    # row set's root mean square in the worst element; LSE stays below both.  Four times that:
    if case["dtype"] == "bfloat16":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 1.25e-3, "max": 0.02}

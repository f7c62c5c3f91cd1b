"""The work that is timed: batched big-integer operations through the library's Python front end.

A case is one operation over a batch (`op`, element width `w`, limbs per
operand, instances `n`) or one uneven batch (`op` = "batch").  Sizes are those
of the repository's benchmark and tests (2048-bit products of 32-bit words, the
multiply sweep 64..2048 limbs, divisions of 2m by m limbs, the mixed batch of
256..65536-bit instances) plus odd sizes that fall on no tile's edge.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "big-int_gb300"))
import bigint_gb300 as B  # noqa: E402
from bigint_gb300 import workloads  # noqa: E402

# Bounds of the drawn cases (64-bit limbs): elements moved by add/sub, limb
# products of a multiply (the 1024-limb listed case has 2^32) and of a division.
MAX_LIMBS = 1 << 24
MAX_MUL_PRODUCTS = 1 << 32
MAX_DIV_PRODUCTS = 1 << 31


def listed():
    return [
        # one caller, one pair of 4096-bit integers: what a single call costs
        {"name": "add one pair", "op": "add", "w": 64, "m": 64, "n": 1},
        # a size of the add sweep, operands larger than L2, one fifth carry chains
        {"name": "add 65536 bit", "op": "add", "w": 64, "m": 1024, "n": 16384},
        # the 32-bit layout at an odd size: rows start on no wide boundary
        {"name": "sub odd words", "op": "sub", "w": 32, "m": 1001, "n": 32000},
        # 4096 pairs of 2048-bit integers in 32-bit words, one tenth all ones
        {"name": "mulfull 2048 bit", "op": "mulfull", "w": 32, "m": 64, "n": 4096},
        # the multiply sweep's small end, a batch that fills the GPU
        {"name": "mulfull 64 limbs", "op": "mulfull", "w": 64, "m": 64, "n": 65536},
        # the multiply sweep's large operands
        {"name": "mulfull 1024 limbs", "op": "mulfull", "w": 64, "m": 1024, "n": 4096},
        # the reference's truncated product, at a size between its own
        {"name": "mul 250 limbs", "op": "mul", "w": 64, "m": 250, "n": 16000},
        # many small divisions (1024-bit by 512-bit)
        {"name": "div 16 by 8", "op": "div", "w": 64, "m": 16, "mb": 8, "n": 262144},
        # a handful of large divisions at once: a serving program's slowest requests
        {"name": "div few 512 by 256", "op": "div", "w": 64, "m": 512, "mb": 256, "n": 8},
        # batches of medium and large divisions (2m by m limbs)
        {"name": "div 256 by 128", "op": "div", "w": 64, "m": 256, "mb": 128, "n": 16384},
        {"name": "div 2048 by 1024", "op": "div", "w": 64, "m": 2048, "mb": 1024, "n": 2048},
        # mixed operations and sizes in one plan (256..65536 bits)
        {"name": "uneven batch", "op": "batch", "w": 64, "m": 0, "n": 20000},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], spread evenly over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["add", "sub", "mul", "mulfull", "mulfull", "div", "div", "batch"])
    if op == "batch":
        return {"op": op, "w": 64, "m": 0, "n": _log_int(rng, 500, 20000)}
    w = rng.choice([64, 64, 32])
    per = 64 // w                      # elements per 64-bit limb
    if op in ("add", "sub"):
        m = _log_int(rng, 1, 4096 * per)
        n = _log_int(rng, 1, max(1, MAX_LIMBS * per // m))
        return {"op": op, "w": w, "m": m, "n": n}
    if op in ("mul", "mulfull"):
        m = _log_int(rng, 4 * per, 2048 * per)
        limbs = -(-m // per)
        most = min(MAX_LIMBS // limbs, MAX_MUL_PRODUCTS // limbs ** 2)
        return {"op": op, "w": w, "m": m, "n": _log_int(rng, min(16, most), most)}
    mb = _log_int(rng, per, 1024 * per)
    m = mb + rng.choice([mb, mb, rng.randint(0, 2 * mb)])
    limbs, limbs_b = -(-m // per), -(-mb // per)
    most = min((1 << 22) // limbs, MAX_DIV_PRODUCTS // (limbs_b * (limbs - limbs_b + 1)))
    return {"op": op, "w": w, "m": m, "mb": mb, "n": _log_int(rng, 1, max(1, most))}


def _random(g, n, m, w):
    if w == 64:
        return torch.randint(-(1 << 63), (1 << 63) - 1, (n, m), generator=g, device="cuda", dtype=torch.int64)
    return torch.randint(-(1 << 31), (1 << 31) - 1, (n, m), generator=g, device="cuda", dtype=torch.int32)


def _batch(n, seed):
    """The benchmark's uneven batch of n instances (the sizes depend on n alone), its operands drawn from `seed`."""
    descs, arena, out_limbs, nflags = workloads.uneven_batch(n=n)
    g = torch.Generator(device="cuda").manual_seed(seed)
    arena_in = _random(g, 1, arena.size, 64)[0].contiguous()
    div = descs[descs["op"] == B.OP_DIV]
    top = torch.from_numpy((div["b"] + div["mb"] - 1).astype(np.int64)).cuda()
    arena_in[top] |= 1                 # a divisor's top limb is not zero
    return descs, arena_in, out_limbs, nflags


def prepare(case, seed):
    op, n, m, w = case["op"], case["n"], case["m"], case["w"]
    if op == "batch":
        descs, arena_in, out_limbs, nflags = _batch(n, seed)
        arena_out = torch.zeros(out_limbs, dtype=torch.int64, device="cuda")
        flags = torch.zeros(nflags, dtype=torch.uint8, device="cuda")
        plan = B.Plan(descs, arena_in.numel(), out_limbs, nflags)
        return {"case": case, "plan": plan, "in": arena_in, "out": arena_out, "flags": flags}
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = _random(g, n, m, w)
    b = _random(g, n, case.get("mb", m), w)
    if op in ("add", "sub"):
        # one instance in five has a long run of all-ones (add) or zero (sub)
        # limbs, so that a carry (borrow) runs through it
        chain = torch.rand(n, generator=g, device="cuda") < 0.2
        length = m // 2 + torch.randint(0, m - m // 2 + 1, (n,), generator=g, device="cuda")
        run = chain[:, None] & (torch.arange(m, device="cuda")[None, :] < length[:, None])
        a.masked_fill_(run, -1 if op == "add" else 0)
        if op == "sub":
            b.masked_fill_(chain[:, None], 0)
        b[:, 0] |= 1
    elif op in ("mul", "mulfull"):
        ones = torch.rand(n, generator=g, device="cuda") < 0.1
        a.masked_fill_(ones[:, None], -1)
        b.masked_fill_(ones[:, None], -1)
    else:
        b[:, -1] |= 1                  # the divisor's top limb is not zero
    return {"case": case, "a": a, "b": b}


def run(state):
    op = state["case"]["op"]
    if op == "batch":
        state["plan"].execute(state["in"], state["out"], state["flags"])
        return [state["out"], state["flags"]]
    if op == "add":
        return B.add(state["a"], state["b"])
    if op == "sub":
        return list(B.sub(state["a"], state["b"]))
    if op == "mul":
        return B.mul(state["a"], state["b"])
    if op == "mulfull":
        return B.mulfull(state["a"], state["b"])
    return list(B.div(state["a"], state["b"]))


def _batch_work(case):
    """Bytes and 32-bit word products of an uneven batch, from its size distribution's means."""
    # sizes log-uniform over 4..1024 limbs; 20 % add, 20 % sub, 40 % full products, 20 % 2m-by-m divisions
    lo, hi = math.log(4.0), math.log(1024.0)
    m1 = (1024.0 - 4.0) / (hi - lo)
    m2 = (1024.0 ** 2 - 4.0 ** 2) / 2 / (hi - lo)
    limbs = case["n"] * m1 * (0.4 * 3 + 0.4 * 4 + 0.2 * 6)
    products = case["n"] * m2 * 0.6
    return 8 * limbs, 4 * products


def work(case):
    """Bytes: operands read and results written once.  Flops: two for each
    32-by-32-bit word product of the schoolbook method (add, sub: one a word)."""
    op, n, m, size = case["op"], case["n"], case["m"], case["w"] // 8
    if op == "batch":
        bytes_, words = _batch_work(case)
        return {"bytes": bytes_, "flops": 2 * words}
    words = (size / 4) ** 2
    if op in ("add", "sub"):
        return {"bytes": 3 * n * m * size + (n if op == "sub" else 0), "flops": n * m * size / 4}
    if op == "mul":
        return {"bytes": 3 * n * m * size, "flops": 2 * words * n * m * (m + 1) / 2}
    if op == "mulfull":
        return {"bytes": 4 * n * m * size, "flops": 2 * words * n * m * m}
    mb = case["mb"]
    return {"bytes": n * (2 * m + 2 * mb) * size + n, "flops": 2 * words * n * mb * (m - mb + 1)}


def _ints(t, w):
    raw = t.cpu().numpy().tobytes()
    step = t.shape[1] * w // 8
    return [int.from_bytes(raw[i:i + step], "little") for i in range(0, len(raw), step)]


def _limbs(values, m, w):
    raw = b"".join(v.to_bytes(m * w // 8, "little") for v in values)
    return torch.from_numpy(np.frombuffer(raw, dtype=np.int64 if w == 64 else np.int32).reshape(len(values), m).copy())


def exact(case, seed):
    """The same results in Python's integers."""
    op, n, m, w = case["op"], case["n"], case["m"], case["w"]
    if op == "div" and n * case["mb"] * (m - case["mb"] + 1) * (w / 30) ** 2 > 1.2e10:
        return None
    if op == "batch":
        descs, arena, out_limbs, nflags = _batch(n, seed)
        raw = arena.cpu().numpy().tobytes()
        out = bytearray(8 * out_limbs)
        flags = np.zeros(nflags, np.uint8)

        def put(at, v, limbs):
            out[8 * at:8 * (at + limbs)] = v.to_bytes(8 * limbs, "little")

        for d in descs:
            k, ma, mb, a0, b0, r0, r2 = (int(d[f]) for f in ("op", "m", "mb", "a", "b", "r", "r2"))
            x = int.from_bytes(raw[8 * a0:8 * (a0 + ma)], "little")
            y = int.from_bytes(raw[8 * b0:8 * (b0 + mb)], "little")
            if k == B.OP_ADD:
                put(r0, (x + y) % (1 << 64 * ma), ma)
            elif k == B.OP_SUB:
                put(r0, abs(x - y), ma)
                flags[int(d["flag"])] = x < y
            elif k == B.OP_MULFULL:
                put(r0, x * y, 2 * ma)
            else:
                q, r = divmod(x, y)
                put(r0, q, ma)
                put(r2, r, mb)
        return [torch.from_numpy(np.frombuffer(bytes(out), dtype=np.int64).copy()), torch.from_numpy(flags)]
    state = prepare(case, seed)
    x, y = _ints(state["a"], w), _ints(state["b"], w)
    mod = 1 << (w * m)
    if op == "add":
        return _limbs([(p + q) % mod for p, q in zip(x, y)], m, w)
    if op == "sub":
        return [_limbs([abs(p - q) for p, q in zip(x, y)], m, w),
                torch.tensor([p < q for p, q in zip(x, y)], dtype=torch.uint8)]
    if op == "mul":
        return _limbs([p * q % mod for p, q in zip(x, y)], m, w)
    if op == "mulfull":
        return _limbs([p * q for p, q in zip(x, y)], 2 * m, w)
    qr = [divmod(p, q) for p, q in zip(x, y)]
    return [_limbs([q for q, _ in qr], m, w), _limbs([r for _, r in qr], case["mb"], w),
            torch.zeros(n, dtype=torch.uint8)]

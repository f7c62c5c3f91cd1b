"""Uneven batches whose divisions run in blocks on the tensor cores: divisors
on both sides of every class, short and long quotients, 32-bit-word and
64-bit-limb descriptors, zero divisors and divisors with leading zero limbs,
against Python integers, from a plan and without allocation."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _val(arena, off, n, w):
    v = arena.view(np.uint32 if w == 32 else np.uint64)[off:off + n]
    return int.from_bytes(v.tobytes(), "little")


def _divisions(B, seed):
    rng = random.Random(seed)
    sizes = [(mb + dq, mb) for mb in (128, 129, 223, 224, 479, 480, 991, 992, 1247, 1248, 2015, 2016) for dq in (0, 40, 300)]
    descs, words, out = [], [], 0
    for k, (m, mb) in enumerate(sizes):
        for w in (64, 32):
            e = 64 // w
            mm, mmb = (m * e - (w == 32), mb * e - (w == 32))
            mm = max(mm, mmb)
            v = rng.getrandbits(mmb * w) | 1 << (mmb * w - 1)
            if k % 7 == 3:
                v >>= rng.randrange(mmb * w)
            if k % 11 == 5:
                v = 0
            u = (1 << (mm * w)) - 1 if k % 5 == 4 else rng.getrandbits(mm * w)
            a = 2 * len(words)                                   # in 32-bit words, whole limbs
            words += list(np.frombuffer(u.to_bytes((mm * w + 63) // 64 * 8, "little"), np.uint64))
            b = 2 * len(words)
            words += list(np.frombuffer(v.to_bytes((mmb * w + 63) // 64 * 8, "little"), np.uint64))
            r = 2 * out
            out += (mm * w + 63) // 64
            r2 = 2 * out
            out += (mmb * w + 63) // 64
            s = 1 if w == 32 else 2
            descs.append((B.OP_DIV, mm, mmb, w, a // s, b // s, r // s, r2 // s, len(descs)))
    return np.array(descs, dtype=B.DESC_DTYPE), np.array(words, dtype=np.uint64), out


def _check(arena_in, d, arena_out, flags):
    for k, x in enumerate(d):
        w = int(x["width"])
        u, v = _val(arena_in, int(x["a"]), int(x["m"]), w), _val(arena_in, int(x["b"]), int(x["mb"]), w)
        got = (_val(arena_out, int(x["r"]), int(x["m"]), w), _val(arena_out, int(x["r2"]), int(x["mb"]), w), int(flags[k]))
        assert got == ((0, 0, 1) if v == 0 else (*divmod(u, v), 0)), tuple(x)


@pytest.mark.parametrize("copies", [1, 12])
def test_division_classes(bigint, copies):
    import torch

    B = bigint
    one, words, out = _divisions(B, 11)
    d = np.concatenate([one] * copies)                           # the same operands, other results
    for c in range(copies):
        part = d[c * len(one):(c + 1) * len(one)]
        e = np.where(part["width"] == 32, 2, 1)
        part["r"] += (c * out * e).astype(np.uint64)
        part["r2"] += (c * out * e).astype(np.uint64)
        part["flag"] += c * len(one)
    ain = B.to_device(words)
    aout = torch.zeros(out * copies, dtype=torch.int64, device="cuda")
    fl = torch.full((len(d),), 9, dtype=torch.uint8, device="cuda")
    plan = B.Plan(d, ain.numel(), aout.numel(), fl.numel())
    for _ in range(2):
        plan.execute(ain, aout, fl)
    torch.cuda.synchronize()
    _check(words, d, B.to_host(aout, np.uint64), fl.cpu().numpy())
    plan.close()
    aout.zero_()
    fl.fill_(9)
    st = B.lib().bi_batch_run_noalloc(d.ctypes.data, len(d), ain.data_ptr(), ain.numel(), aout.data_ptr(), aout.numel(),
                                      fl.data_ptr(), fl.numel(), None)
    assert st == 0
    _check(words, d, B.to_host(aout, np.uint64), fl.cpu().numpy())


@pytest.mark.parametrize("n", [40, 600])
def test_multiply_classes(bigint, n):
    """Full and truncated products on both sides of each tensor-core class,
    largest and smallest in one launch, so that a buffer holds a smaller operand
    after a larger one."""
    import torch

    B = bigint
    rng = random.Random(n)
    edges = [150, 159, 160, 161, 207, 208, 256, 257, 300, 512, 513, 700, 1024, 1025, 2048]
    descs, nin, nout = [], 0, 0
    for k in range(n):
        full = k % 3 != 2
        w = 32 if k % 4 == 3 else 64
        m = edges[k % len(edges)] if k < 2 * len(edges) else rng.randint(140, 700)
        e = 64 // w
        mm = m * e - (w == 32 and k % 8 == 3)
        rl = (2 if full else 1) * m
        descs.append((B.OP_MULFULL if full else B.OP_MUL, mm, mm, w, nin * e, (nin + m) * e, nout * e, 0, 0))
        nin += 2 * m
        nout += rl
    d = np.array(descs, dtype=B.DESC_DTYPE)
    words = np.random.default_rng(n).integers(0, 1 << 64, nin, dtype=np.uint64)
    words[: nin // 8] = np.uint64(0xFFFFFFFFFFFFFFFF)
    ain = B.to_device(words)
    aout = torch.zeros(nout, dtype=torch.int64, device="cuda")
    plan = B.Plan(d, nin, nout)
    for _ in range(2):
        plan.execute(ain, aout)
    torch.cuda.synchronize()
    out = B.to_host(aout, np.uint64)
    for x in d:
        w, m, full = int(x["width"]), int(x["m"]), int(x["op"]) == B.OP_MULFULL
        u, v = _val(words, int(x["a"]), m, w), _val(words, int(x["b"]), m, w)
        k = 2 * m if full else m
        assert _val(out, int(x["r"]), k, w) == u * v % (1 << (w * k)), tuple(x)
    plan.close()

"""The digits and order sums of the FP64-width tensor pass (tensor64.cu), at
the ends of their ranges.

On the CPU: the state's digits as bytes 128 too large against the operator's
balanced digits, with starting sums that take the excess off, give the exact
order sums; every partial sum, whatever the order of the terms, stays where an
FP32 accumulator near 0.75 with units of 2^-24 is exact; and the combination
of the sums' bits is the exact product to three bits below the old unit.

On the GPU: operators and states whose terms all add up with full digits, so
that one rounded product or sum would show at 2^-24 of the result."""
import random
import struct
from fractions import Fraction

import numpy as np
import pytest

BIAS = 0x0080808080808080
M64 = (1 << 64) - 1
ACC0, PAIR = 0x3F400000, 0x7F400000


def raw_digits(v):
    """store_digits: bytes of v + BIAS, the most significant (9 bits) first."""
    u = v + BIAS
    assert 0 <= u < 1 << 57
    return [u >> 48] + [(u >> (8 * (6 - j))) & 255 for j in range(1, 7)]


def combine(bits):
    """combine_orders, in 64-bit arithmetic."""
    r12, r34, r56 = (((bits[i] << 8) + bits[i + 1]) & 0xFFFFFFFF for i in (1, 3, 5))
    const = (ACC0 << 43) + (PAIR << 27) + (PAIR << 11) + (PAIR >> 5) + (ACC0 >> 13)
    acc = r34 * 2048 + (r56 >> 5) + (bits[7] >> 13) + (r12 << 27) + (((bits[0] * 2048) & 0xFFFFFFFF) << 32) - const
    acc &= M64
    return acc - (1 << 64) if acc >> 63 else acc


def f16(x):
    b = struct.pack("<e", float(x))
    assert Fraction(struct.unpack("<e", b)[0]) == x  # exact in FP16
    return x


@pytest.mark.parametrize("kind", ["random", "largest", "mixed", "zero"])
def test_order_sums_are_exact(kind):
    rng = random.Random(kind)
    top = 1 << 55
    pick = {"random": lambda: rng.randint(-top, top), "largest": lambda: rng.choice([-top, top]),
            "mixed": lambda: rng.choice([-top, top, 0, 1, -1, top - 1, 0x7F7F7F7F7F7F7F, -0x80808080808080]),
            "zero": lambda: 0}[kind]
    for _ in range(40):
        w, v = [pick() for _ in range(32)], [pick() for _ in range(32)]
        wd = [[d - 128 for d in raw_digits(t)] for t in w]
        vd = [raw_digits(t) for t in v]
        assert all(abs(d) <= 128 for r in wd for d in r)
        sums = []
        for o in range(8):
            pairs = [(o - j, j) for j in range(7) if 0 <= o - j <= 6]
            C = sum(wd[k][j] for _, j in pairs for k in range(32))
            c1 = (C + 128) >> 8
            c0 = C - 256 * c1
            start = f16(Fraction(3, 4)) - f16(Fraction(c1, 512)) - f16(Fraction(c0, 1 << 17))
            terms = [vd[k][i] * wd[k][j] for i, j in pairs for k in range(32)]
            rng.shuffle(terms)
            s = start * (1 << 24)
            for t in terms:
                s += t
                assert 1 << 23 <= s < 1 << 24  # FP32 in [1/2, 1): units of 2^-24
            assert s == 3 * (1 << 22) + sum((vd[k][i] - 128) * wd[k][j] for i, j in pairs for k in range(32))
            f = struct.unpack("<I", struct.pack("<f", float(s / (1 << 24))))[0]
            assert f == ACC0 + int(s) - 3 * (1 << 22)
            sums.append(f)
        # the orders that are left out reach 5 * 32 * 2^14 units of 2^-64 of order 0's
        exact = Fraction(sum(a * b for a, b in zip(w, v)), 1 << 53)
        if abs(exact) < 1 << 63:
            assert -2 - Fraction(5 * 32 * (1 << 14) * 258, 256 ** 4) * 8 <= combine(sums) - exact <= Fraction(5 * 32 * (1 << 14) * 258, 256 ** 4) * 8


FULL = 0x7F7F7F7F7F7F7F / 2.0 ** 55  # every digit 127


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,x,s", [(6, 4, 1 - 2.0 ** -40, 1 - 2.0 ** -53), (6, 4, FULL, FULL), (7, 4, FULL, 1 - 2.0 ** -53),
                                     (7, 4, 0.75 + 2.0 ** -52, FULL), (6, 3, FULL, FULL),
                                     (7, 3, 0.5 + 2.0 ** -53, 2.0 ** -30 * FULL)])
def test_full_digits_on_the_gpu(engine, n, k, x, s):
    """U = x (1 + i) everywhere on k qubits, rho = s (1 - i) with |s| < 1 in
    each half: every output is a sum of 2^(2k) equal terms, known exactly.
    Two steps of at most 2^-54 of the column's largest value times the row's
    1-norm (equal to the result here), and the rounding of the result."""
    one = np.array([[1, 1], [1, 1]], dtype=complex)
    dim = 1 << n
    re, im = np.full(dim * dim, s), np.full(dim * dim, -s)
    with engine.Simulation(n, mode="fused", tensor="all") as sim:
        sim.append_c1(0, (x + 1j * x) * one)
        for q in range(1, k):
            sim.append_c1(q, one)
        sim.upload()
        sim.set_option(engine.OPT_RECORD, 1)
        sim.set_dm(re, im)
        sim.run()
        rec = sim.pass_records()
        gr, gi = sim.get_dm()
    assert rec[:, 8].sum() == 1 and rec[0, 0] == k
    # sum over 2^k kets of x(1+i) s(1-i) = 2 x s each, then over 2^k bras of x(1-i)
    want = Fraction(2 * 4 ** k) * Fraction(x) ** 2 * Fraction(s)
    got = np.unique(np.concatenate([gr, -gi]))
    err = max(abs(Fraction(float(g)) - want) / want for g in got)
    assert err <= Fraction(3, 1 << 53), float(err)

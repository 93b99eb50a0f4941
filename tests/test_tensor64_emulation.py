"""The arithmetic of the FP64-width tensor pass (tensor64.cu) as it stands, with
Python integers: values aligned to their column's grid (three of four rounded by
a conversion, the fourth truncated), digits as biased bytes, exact order sums,
their combination from the accumulators' bits, the bra columns' keys and shifts,
and the one rounding to FP64.

On the CPU against exact rational arithmetic, within a bound that is derived
below; on the GPU the kernel's outputs bit for bit.

The bound, for D = 2^K, one output of one step: a column's largest value X has at
least 2^54 units on its grid and an operator row's largest entry w_max at least
2^54 on the row's, so
  * the column's values are off by one unit each at most: 2^-54 X |w|_1;
  * the row's 2 D entries by half a unit each: D 2^-54 w_max X;
  * the sums leave out orders 8 to 12, below 2 D 5.02 2^14 256^4 products of
    the two units, and floor the orders below 0 and 7 once each; one unit of the
    combination is 2^53 of those products: (2 D 5.02 / 128 + 2) 2^-55 w_max X.
Together 2^-54 X (|w|_1 + (1.04 D + 1) w_max), then one rounding, 2^-53, of the
result of the second step."""
from fractions import Fraction as F

import numpy as np
import pytest

import dmsim_workloads as W
from test_tensor64_digits import ACC0, BIAS, combine, raw_digits
from test_tensor64_numerics import bits_f64, digits, f64_bits

M64 = (1 << 64) - 1
C2 = 65  # the planner's id of an arbitrary 2-qubit gate (gates.h)


def rint(x):
    """x (Fraction) to the nearest integer, ties to even."""
    return round(x)


def host_rows(m):
    """build_tc64_k: rows 0..D-1 [Ur, -Ui] and D..2D-1 [Ui, Ur] as (exponent, digits);
    the digits of a negated entry are the entry's negated."""
    d, top, low = m.shape[0], [], []
    for a in range(d):
        mx = max(np.abs(m[a].real).max(), np.abs(m[a].imag).max())
        e = int(np.frexp(mx)[1])
        part = lambda z: [digits(int(np.rint(np.ldexp(v, 55 - e))) if mx > 0 else 0) for v in z]
        re, im = part(m[a].real), part(m[a].imag)
        top.append((e - 55 if mx > 0 else 0, re + [[-x for x in t] for t in im]))
        low.append((top[-1][0], im + re))
    return top + low


def align(xs):
    """align_fp64 on one column (2 D values): exponent field and integers."""
    bits = [f64_bits(x) for x in xs]
    e = max(max((b >> 52) & 0x7FF for b in bits), 64)
    d = len(xs) // 2
    out = []
    for i, b in enumerate(bits):
        ex, frac, neg = (b >> 52) & 0x7FF, b & ((1 << 52) - 1), b >> 63
        if (i % d) & 3 != 3 and e < 1077:  # one conversion, the significand with its leading 1 even at exponent 0
            v = rint(F((1 << 52) | frac) * F(2) ** (ex + 1077 - e - 1075))
        else:
            v = (((1 << 52) | frac) << 2) >> (e - ex)
        assert v <= 1 << 55
        out.append(-v if neg else v)
    return e, out


def product(row, values):
    """One output's accumulators and their combination, as a signed 64-bit integer."""
    digits = [[b - 128 for b in raw_digits(v)] for v in values]
    acc = []
    for o in range(8):
        s = sum(digits[k][i] * row[k][o - i] for i in range(7) if 0 <= o - i <= 6 for k in range(len(values)))
        assert abs(s) < 1 << 22
        acc.append(ACC0 + s)
    return combine(acc)


def leading_bit(hi):
    hi = hi - (1 << 32) if hi >> 31 else hi
    return (hi if hi >= 0 else ~hi).bit_length() - 1


def to_fp64(y, p, near):
    b = f64_bits(float(y))
    if near:
        h = b >> 32
        return bits_f64((((h + (p << 20)) & 0xFFFFFFFF if h else 0) << 32) | (b & 0xFFFFFFFF))
    return bits_f64((b + ((p & M64) << 52)) & M64) if y != 0 and ((b >> 52) & 0x7FF) + p > 0 else 0.0


def emulate(u, v, x):
    """out[a][b] = sum U[a][c] V[b][e] x[c][e] as the kernel computes it."""
    d = u.shape[0]
    ru, rv = host_rows(u), host_rows(v)
    Y, E = [[0] * d for _ in range(2 * d)], []
    for b in range(d):
        e, vals = align(list(x[:, b].real) + list(x[:, b].imag))
        E.append(e)
        for n in range(2 * d):
            Y[n][b] = product(ru[n][1], vals)
    out = np.zeros((d, d), complex)
    ewmin = min(r[0] for r in rv[:d])
    shifted_left = False
    for a in range(d):
        ys = [Y[a][b] for b in range(d)] + [Y[a + d][b] for b in range(d)]
        es = E + E
        key = max([0] + [e + leading_bit((y & M64) >> 32) for y, e in zip(ys, es)])
        vals = []
        for y, e in zip(ys, es):
            s = key - 22 - e
            shifted_left |= s < 0 and y != 0
            w = y >> s if s >= 0 else y << -s
            assert abs(w) <= 1 << 55
            vals.append(w)
        pa = key + ru[a][0] - 993
        for n in range(2 * d):
            b = n % d
            r = to_fp64(product(rv[n][1], vals), pa + rv[b][0], pa + ewmin >= -1022)
            out[a, b] += r if n < d else 1j * r
    return out, shifted_left


def cmul(p, q):
    return p[0] * q[0] - p[1] * q[1], p[0] * q[1] + p[1] * q[0]


def check_bound(u, v, x, got):
    """Every output within the docstring's bound of the exact one."""
    d = u.shape[0]
    ex = [[(F(z.real), F(z.imag)) for z in row] for row in x]
    eu = [[(F(z.real), F(z.imag)) for z in row] for row in u]
    ev = [[(F(z.real), F(z.imag)) for z in row] for row in v]
    slack = F(104 * d, 100) + 1
    norm1 = lambda row: sum(abs(z[0]) + abs(z[1]) for z in row)
    big = lambda zs: max(max(abs(z[0]), abs(z[1])) for z in zs)
    unit = F(1, 1 << 54)
    T = [[None] * d for _ in range(d)]
    err = [[None] * d for _ in range(d)]
    for a in range(d):
        for b in range(d):
            z = [cmul(eu[a][c], ex[c][b]) for c in range(d)]
            T[a][b] = (sum(t[0] for t in z), sum(t[1] for t in z))
            X = max(big([ex[c][b] for c in range(d)]), F(1, 1 << 958))  # grids end at exponent field 64
            err[a][b] = unit * X * (norm1(eu[a]) + slack * big(eu[a]))
    worst = 0.0
    for a in range(d):
        X = max(big(T[a]) + max(err[a]), F(1, 1 << 1000))
        for b in range(d):
            z = [cmul(ev[b][c], T[a][c]) for c in range(d)]
            want = (sum(t[0] for t in z), sum(t[1] for t in z))
            tol = sum((abs(ev[b][c][0]) + abs(ev[b][c][1])) * err[a][c] for c in range(d))
            tol += unit * X * (norm1(ev[b]) + slack * big(ev[b]))
            for w, g in zip(want, (got[a, b].real, got[a, b].imag)):
                e = abs(F(float(g)) - w)
                assert e <= tol + abs(w) * F(1, 1 << 53) + F(1, 1 << 1022), (a, b, float(e), float(tol))
                worst = max(worst, float(e / tol) if tol else 0.0)
    return worst


def unitary(rng, d):
    return np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))[0]


def inputs(kind, d, rng):
    u = unitary(rng, d)
    x = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
    if kind == "skewed":  # one entry near 1, the rest tiny and not on the row's grid
        u = (rng.uniform(1, 2, (d, d)) + 1j * rng.uniform(1, 2, (d, d))) * 2.0 ** -50 / 3
        u[np.arange(d), rng.permutation(d)] = 1 - 2.0 ** -53
        x = np.full((d, d), 1 - 2.0 ** -53) * (1 + 1j)
    elif kind == "sizes":
        x *= 10.0 ** rng.uniform(-280, 12, size=(1, d))
    elif kind == "large":  # grids at and above 2^1077: shifted, not converted
        x *= 10.0 ** rng.uniform(10, 100, size=(1, d))
    elif kind == "zeros":
        x[:, 1:] = 0
        x[3, 0] = 0
        u[2] = 0
    elif kind == "cancelled":  # ket outputs far below what their inputs could give
        s = 1.0 / np.sqrt(d)
        u = np.array([[s * (-1) ** bin(i & j).count("1") for j in range(d)] for i in range(d)], complex)
        x = np.ones((d, 1)) * x[:1] + 2.0 ** -40 * x
    elif kind == "density":
        x = x @ x.conj().T
        x /= np.trace(x).real
    return u, x


@pytest.mark.parametrize("d", [8, 16])
@pytest.mark.parametrize("kind", ["random", "skewed", "sizes", "large", "zeros", "cancelled", "density"])
def test_within_the_derived_bound(kind, d):
    rng = np.random.default_rng([d, len(kind), ord(kind[0])])
    u, x = inputs(kind, d, rng)
    got, shifted_left = emulate(u, u.conj(), x)
    check_bound(u, u.conj(), x, got)
    if kind == "cancelled":
        assert shifted_left


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["random", "sizes", "large", "zeros", "cancelled", "density"])
@pytest.mark.parametrize("n,qubits", [(6, (0, 1, 2, 3)), (6, (5, 2, 0, 3)), (7, (6, 1, 4, 3)), (6, (0, 2, 5)), (7, (6, 4, 3))])
def test_kernel_equals_the_emulation(engine, kind, n, qubits):
    """One dense pass on the GPU: three groups of every column bit for bit."""
    k, dim = len(qubits), 1 << n
    rng = np.random.default_rng([n, k, len(kind), ord(kind[0])])
    gates = [(None, (qubits[i], qubits[(i + 1) % k]), 0, 0, 0, unitary(rng, 4)) for i in range(k)]
    if kind == "cancelled":
        gates = [(W.OP["H"], (q,), 0, 0, 0) for q in qubits]
    with engine.Simulation(n, mode="fused", max_k=k, tensor="all") as s:
        for g in gates:
            s.append_c2(*g[1], g[5]) if g[0] is None else s.append(*g)
        plan = engine.plan_inspect(n, [(C2 if g[0] is None else g[0],) + tuple(g[1:]) for g in gates], max_k=k)
        s.upload()
        s.set_option(engine.OPT_RECORD, 1)
        assert len(plan) == 1 and plan[0]["K"] == k
        q, u, v = plan[0]["qubits"], plan[0]["U"], plan[0]["V"]
        state = np.zeros((dim, dim), complex)  # [ket][bra]
        rest = [b for b in range(n) if b not in q]
        spread = lambda i, bits: sum(((i >> t) & 1) << b for t, b in enumerate(bits))
        kets = [[spread(a, q) | spread(o, rest) for a in range(1 << k)] for o in range(1 << len(rest))]
        for rows in kets:
            for cols in kets:
                state[np.ix_(rows, cols)] = inputs(kind, 1 << k, rng)[1]
        A = state.T
        s.set_dm(A.real.reshape(-1), A.imag.reshape(-1))
        s.run()
        assert s.pass_records()[0, 8] == 1
        got = s.rho()
    for r, c in ((0, 0), (len(kets) - 1, 1), (1, len(kets) - 1)):
        want, _ = emulate(u, v, state[np.ix_(kets[r], kets[c])])
        block = got[np.ix_(kets[r], kets[c])]
        assert np.array_equal(block.real, want.real) and np.array_equal(block.imag, want.imag)

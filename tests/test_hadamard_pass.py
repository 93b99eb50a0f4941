"""1-qubit passes whose real operator has four entries of size sqrt(1/2) (H and
its sign variants): sums, differences and exact halves, so the same in numpy
bit for bit -- normal numbers, zeros, numbers whose half is subnormal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
S = np.sqrt(0.5)
SIGNS = [(1, 1, 1, -1), (1, -1, 1, 1), (-1, 1, 1, 1), (1, 1, -1, 1), (-1, -1, 1, -1)]


def butterfly(x, q, n, u):
    """Half of (signs of u) on the ket and the bra bit q of A[bra][ket], in the kernel's order of additions."""
    x = x.reshape(1 << (n - 1 - q), 2, 1 << q, 1 << (n - 1 - q), 2, 1 << q)  # bra high, bit, low; ket high, bit, low
    z = {}
    for j in (0, 1):  # ket sums and differences of either bra value
        a, b = x[:, j, :, :, 0], x[:, j, :, :, 1]
        z[j] = (a + b, a - b)
    both = {(i, j): 0.5 * ((z[0][i] + z[1][i]) if j == 0 else (z[0][i] - z[1][i])) for i in (0, 1) for j in (0, 1)}
    out = np.empty_like(x)
    for a in (0, 1):
        for b in (0, 1):
            sign = u[2 * a] * u[2 * b]
            out[:, b, :, :, a] = sign * both[int(u[2 * a] * u[2 * a + 1] < 0), int(u[2 * b] * u[2 * b + 1] < 0)]
    return out.reshape(-1)


@pytest.mark.parametrize("u", SIGNS)
@pytest.mark.parametrize("n,q", [(2, 0), (2, 1), (5, 2), (8, 7), (9, 0)])
def test_hadamard_pass(engine, n, q, u):
    rng = np.random.default_rng(n + 10 * q)
    N = 1 << (2 * n)
    parts = []
    for _ in range(2):
        x = rng.standard_normal(N)
        x[rng.random(N) < 0.2] = 0.0
        tiny = rng.random(N) < 0.2
        x[tiny] = rng.integers(-7, 8, tiny.sum()) * 2.0 ** -1074
        tiny = rng.random(N) < 0.1
        x[tiny] = rng.choice([1.0, 1.5, -1.25], tiny.sum()) * 2.0 ** -1022
        parts.append(x)
    with engine.Simulation(n, mode="plain") as s:
        s.append_c1(q, np.array(u).reshape(2, 2) * S)
        s.upload()
        s.set_dm(*parts)
        s.run()
        got = s.get_dm()
    for x, g in zip(parts, got):
        assert np.array_equal(g, butterfly(x, q, n, u))


def test_near_hadamard_is_not_one(engine):
    """Entries off by 1e-12 keep their own multiply-adds."""
    n, q = 3, 1
    rng = np.random.default_rng(1)
    x, y = rng.standard_normal((2, 64))
    m = np.array([[S * (1 + 1e-12), S], [S, -S]])
    full = np.kron(np.kron(np.eye(2), m), np.eye(2))
    a = (x + 1j * y).reshape(8, 8).T
    want = full @ a @ full.T
    with engine.Simulation(n, mode="plain") as s:
        s.append_c1(q, m)
        s.upload()
        s.set_dm(x, y)
        s.run()
        got = s.rho()
    # 16 products below 4 each way at 2^-53
    assert np.abs(got - want).max() <= 1e-14

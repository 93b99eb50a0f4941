"""Channels whose superoperators hold zero, real and complex terms, at the
smallest states and tile edges, on both 1-qubit kernels, against numpy."""
import numpy as np
import pytest

from test_noise import embed


def kraus_set(kind, nq, rng):
    d = 1 << nq
    if kind == "dense":  # every term nonzero and complex
        v = rng.standard_normal((3 * d, d)) + 1j * rng.standard_normal((3 * d, d))
        q, _ = np.linalg.qr(v)
        return [q[i * d:(i + 1) * d] for i in range(3)]
    if kind == "phases":  # diagonal: one complex term a row
        return [np.diag(np.exp(1j * rng.uniform(0, 6, d)))]
    p = 0.3  # damping of the last basis state into the first: real rows of one and two terms
    k0 = np.eye(d, dtype=complex)
    k0[-1, -1] = np.sqrt(1 - p)
    k1 = np.zeros((d, d), complex)
    k1[0, -1] = np.sqrt(p)
    return [k0, k1]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "phases", "damping"])
@pytest.mark.parametrize("n,qubits", [(1, (0,)), (2, (1,)), (5, (0,)), (6, (5,)), (7, (3,)), (2, (1, 0)), (3, (0, 2)),
                                      (5, (4, 1)), (7, (0, 1)), (7, (6, 3))])
@pytest.mark.parametrize("direct1", [True, False])
def test_channel_terms(engine, kind, n, qubits, direct1):
    rng = np.random.default_rng(5)
    kraus = kraus_set(kind, len(qubits), rng)
    d = 1 << n
    a = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))) / d
    # a 2-qubit matrix's index is 2 bit(qubits[1]) + bit(qubits[0]) as the engine takes it
    ops = [embed(k, qubits[::-1], n) for k in kraus]
    want = sum(k @ a @ k.conj().T for k in ops)
    with engine.Simulation(n, mode="plain", direct1=direct1) as s:
        s.set_dm(a.T.real.reshape(-1), a.T.imag.reshape(-1))
        s.append_channel(qubits, kraus)
        s.upload()
        s.run()
        got = s.rho()
    # 16 products of entries below 1 each way, 2^-53 apiece, and the host's own superoperator sums
    assert np.abs(got - want).max() <= 1e-14

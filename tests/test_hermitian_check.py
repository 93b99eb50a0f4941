"""What a run pays for asking whether a written state is Hermitian."""
import time

import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,passes", [(11, 4), (11, 6), (12, 6)])
def test_check_is_cheap_on_arbitrary_states(engine, n, passes):
    """Short plans on a state without the symmetry: with half-range passes
    planned, a run takes no more than 8 % longer than without them."""
    d = 1 << n
    x = np.random.default_rng(1).standard_normal(d * d) / d
    best = {}
    for hermitian in (0, 1):
        with engine.Simulation(n, mode="plain") as s:
            s.set_option(engine.OPT_HERMITIAN, hermitian)
            for i in range(passes):
                s.append(W.OP["CX"], (i % n, (i + 3) % n))
            s.upload()
            s.set_dm(x, x)
            times = []
            for _ in range(60):
                t = time.perf_counter()
                s.run()
                times.append(time.perf_counter() - t)
            best[hermitian] = min(times)
    assert best[1] <= 1.08 * best[0], best


@pytest.mark.parametrize("where", ["first", "last", "inside", "diagonal"])
def test_one_different_entry_is_found(engine, where):
    """A Hermitian state but for one entry: the run is the whole one (chained
    passes on arbitrary states are linear: compare with the option off)."""
    n = 11
    d = 1 << n
    rng = np.random.default_rng(2)
    a = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))) / d
    a = (a + a.conj().T) / 2
    i, j = {"first": (0, 1), "last": (d - 1, d - 2), "inside": (d // 2 + 33, 700), "diagonal": (77, 77)}[where]
    a[i, j] += 0.25j if where == "diagonal" else 0.25
    circ = W.table_mix(n, 40, seed=5)
    out = []
    for hermitian in (1, 0):
        with engine.Simulation(n, mode="fused") as s:
            s.set_option(engine.OPT_HERMITIAN, hermitian)
            s.extend(circ)
            s.upload()
            s.set_dm(a.T.real.reshape(-1), a.T.imag.reshape(-1))
            s.run()
            out.append(s.rho())
    assert np.abs(out[0] - out[1]).max() <= 1e-12
    assert np.abs(out[0] - out[0].conj().T).max() > 1e-4

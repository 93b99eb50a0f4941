"""3- and 4-qubit sparse operators of complex64 states on the dense FP32 kernel:
what an earlier kernel left in shared memory does not reach the state, although
the pass leaves runs out that only zeros of the operator would read."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu
OP = W.OP


def controlled(control, targets, rng):
    """Rotations of the targets under one control: rows of the identity where it is 0."""
    out = []
    for t in targets:
        out.append((OP["CRY"], (control, t), *rng.uniform(0.3, 2.5, 3)))
        out.append((OP["CU3"], (control, t), *rng.uniform(0.3, 2.5, 3)))
    return out


@pytest.mark.parametrize("n,control,targets", [(7, 6, (0, 1)), (9, 8, (1, 2)), (9, 0, (7, 8)), (10, 9, (5, 7)),
                                               (8, 7, (0, 1, 2)), (10, 9, (0, 4, 8))])
def test_unloaded_runs_are_zeros(engine, oracle, n, control, targets):
    rng = np.random.default_rng(n)
    circ = [(OP["U3"], (q,), *rng.uniform(0.3, 2.5, 3)) for q in range(n)]
    half = controlled(control, targets, rng)
    k = 1 + len(targets)
    # fill every SM's shared memory with NaN: dense tiles of an all-NaN state
    with engine.Simulation(10, mode="fused", max_k=4, precision="c64", tensor=False, renorm=0) as s:
        s.extend(W.layered_u3_cx(10, 60, seed=1))
        s.upload()
        bad = np.full(1 << 20, np.nan)
        s.set_dm(bad, bad)
        s.run()
    with engine.Simulation(n, mode="fused", max_k=k, precision="c64", tensor=False, direct1=False, renorm=0) as s:
        s.extend(half)
        s.upload()
        s.set_option(engine.OPT_RECORD, 1)
        re, im = oracle.dm_sim(n, circ)
        s.set_dm(re, im)
        s.run()
        rec = s.pass_records()
        got = s.get_dm()
    assert len(rec) == 1 and rec[0, 0] == k and rec[0, 1] == 4  # one SPARSE pass
    want = oracle.dm_sim(n, half, re, im)
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= 1e-6  # two steps of at most 16 terms below 1, 2^-24 apiece

"""What a batch's wide circuits cost outside its graph, and how many narrow
circuits stay with the work queue by default."""
import time

import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


def make(engine, sizes, **opts):
    rng = np.random.default_rng(3)
    b = engine.Batch(sizes, **opts)
    for c, n in enumerate(sizes):
        b.extend(c, W.hea(n, 1, rng))
    b.upload()
    return b


def test_run_costs_no_copy_per_wide_circuit(engine):
    """256 wide circuits: the host's clock around run() is the graph's time, a
    launch and one 4-byte copy.  (A synchronous copy for every wide circuit took
    some 9 us each, 2.3 ms here.)"""
    with make(engine, [3] * 256, wide_qubits=3) as b:
        rest = []
        for _ in range(20):
            t = time.perf_counter()
            b.run()
            rest.append((time.perf_counter() - t) * 1e3 - b.stats()["ms"])
    assert np.median(rest) <= 0.5, rest


@pytest.mark.parametrize("mode,arith,n,few", [("fused", "fp64", 6, 8), ("fused", "fp64", 7, 32), ("plain", "fp64", 7, 8),
                                              ("fused", "df64", 8, 8)])
def test_many_narrow_circuits_go_to_the_queue(engine, mode, arith, n, few):
    for count in (few, few + 1):
        with make(engine, [n] * count, mode=mode, fused_arith=arith) as b:
            assert (b.stats()["items"] > 0) == (count > few)  # items: tiles of the queue
            b.run()
            assert abs(b.diag(count - 1).sum() - 1) <= 1e-9

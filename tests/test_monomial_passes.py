"""Monomial passes (MOVE, SIGNED, PHASE) of 2 to 4 qubits on states large
enough for the pipelined kernel (kernels_mono.cu), in all three arithmetics,
against the statevector oracle."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu
OP = W.OP

GATES = {"diagonal": ["Z", "S", "T", "U1", "CZ", "CU1", "CRZ", "RZZ"], "move": ["X", "CX", "SWAP", "CCX", "CSWAP"], "signed": ["X", "Y", "Z", "S", "CX", "CZ", "CY"],
         "phase": ["X", "T", "U1", "CX", "CU1", "CRZ", "RZZ", "CCX"]}


def circuit(n, kind, gates, rng):
    c = [(OP["U3"], (q,), *rng.uniform(0, 6, 3)) for q in range(n)]
    for _ in range(gates):
        op = rng.choice(GATES[kind])
        k = 3 if op in ("CCX", "CSWAP") else 1 if op in ("X", "Y", "Z", "S", "T", "U1") else 2
        # half of the gates on a few qubits, so that passes of all widths and positions come up
        pool = rng.permutation(n)[:5] if rng.random() < 0.5 else np.arange(n)
        c.append((OP[op], tuple(int(q) for q in rng.choice(pool, k, replace=False)), *rng.uniform(0, 6, 3)))
    return c


@pytest.mark.parametrize("kind", ["diagonal", "move", "signed", "phase"])
@pytest.mark.parametrize("n,max_k,precision,arith,tol", [
    (10, 2, "fp64", "fp64", 1e-13), (10, 4, "fp64", "fp64", 1e-13), (11, 3, "fp64", "fp64", 1e-13),
    (11, 4, "fp64", "df64", 1e-10), (10, 3, "fp64", "df64", 1e-10), (10, 2, "c64", "fp64", 1e-5),
    (11, 4, "c64", "fp64", 1e-5), (10, 3, "c64", "fp64", 1e-5)])
def test_monomial_passes(engine, oracle, kind, n, max_k, precision, arith, tol):
    """Tolerances: FP64 1e-13 (20 passes of a few roundings of values below
    1), double-float and complex64 those of the fused and complex64 tests."""
    c = circuit(n, kind, 80, np.random.default_rng(3 * n + max_k))
    sr, si = oracle.sv_sim(n, c)
    with engine.Simulation(n, mode="fused", max_k=max_k, precision=precision, fused_arith=arith) as s:
        s.extend(c)
        s.upload()
        s.set_option(engine.OPT_RECORD, 1)
        s.run()
        rec = s.pass_records()
        m = s.pure_metrics(sr + 1j * si)
    assert ((rec[:, 1] <= 2) & (rec[:, 0] >= 2)).sum() >= 1
    assert m["max_abs_err"] <= tol, m

"""The order of a 2-qubit channel's qubits, as the header and append_channel state
it: kron(A, B) is A on qubits[1] and B on qubits[0]."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu


def damping(p):
    return [np.array([[1, 0], [0, np.sqrt(1 - p)]], complex), np.array([[0, np.sqrt(p)], [0, 0]], complex)]


@pytest.mark.parametrize("n,qubits", [(2, (0, 1)), (2, (1, 0)), (5, (3, 1)), (5, (0, 4))])
def test_product_channel_is_its_factors(engine, n, qubits):
    a, b = damping(0.4), damping(0.1)
    circ = W.layered_u3_cx(n, 12, seed=2)
    out = []
    for product in (True, False):
        with engine.Simulation(n, mode="plain") as s:
            s.extend(circ)
            if product:
                s.append_channel(qubits, [np.kron(x, y) for x in a for y in b])
            else:
                s.append_channel((qubits[1],), a)
                s.append_channel((qubits[0],), b)
            s.upload()
            s.run()
            out.append(s.rho())
    # 16 products of entries below 1 each way, 2^-53 apiece, and the superoperators' own sums
    assert np.abs(out[0] - out[1]).max() <= 1e-14

"""Several narrow passes in one sweep (kernels_multi.cu) against the same passes
launched one by one (a recorded run does that): the same operations in the same
order, so the same state bit for bit."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu
OP = W.OP
ONE = ["U3", "U2", "U1", "X", "Y", "Z", "H", "S", "SDG", "T", "TDG", "RX", "RY", "RZ", "W", "R"]


def program(n, rng, noise):
    """Runs of gates and channels on one or two qubits, from anywhere."""
    out = []
    for _ in range(25):
        pair = [int(q) for q in rng.choice(n, 2, replace=False)]
        for _ in range(int(rng.integers(1, 20))):
            x = rng.random()
            if x < 0.35:
                c, t = pair if rng.random() < 0.5 else pair[::-1]
                out.append((OP["CX"], (c, t), 0.0, 0.0, 0.0))
            elif x < 0.42 and noise:
                out.append(("depolarizing2", tuple(pair if rng.random() < 0.5 else pair[::-1]), float(rng.uniform(0.01, 0.4))))
            elif x < 0.5 and noise:
                kind = str(rng.choice(["depolarizing", "amplitude_damping", "phase_damping", "bit_flip", "phase_flip"]))
                out.append((kind, (pair[int(rng.integers(2))],), float(rng.uniform(0.01, 0.4))))
            else:
                name = str(rng.choice(ONE[:-1] if rng.random() < 0.95 else ONE))
                out.append((OP[name], (pair[int(rng.integers(2))],), *rng.uniform(0.1, 1.2, 3)))
    return out


@pytest.mark.parametrize("precision,arith", [("fp64", "fp64"), ("fp64", "df64"), ("c64", "fp64")])
@pytest.mark.parametrize("n", [2, 3, 5, 9, 10, 11])
@pytest.mark.parametrize("noise", [False, True])
@pytest.mark.parametrize("mode", ["plain", "fused"])
def test_merged_equals_single(engine, n, precision, arith, noise, mode):
    rng = np.random.default_rng(100 * n + noise)
    prog = program(n, rng, noise)
    with engine.Simulation(n, mode=mode, max_k=1 if mode == "fused" else 4, precision=precision, plain_arith=arith,
                           fused_arith=arith, renorm=0) as s:
        for g in prog:
            s.append_noise(g[0], g[1], g[2]) if isinstance(g[0], str) else s.append(*g)
        s.upload()
        out = []
        for record in (0, 1):
            s.reset_dm()
            s.set_option(engine.OPT_RECORD, record)
            s.run()
            out.append(s.get_dm())
    assert np.abs(out[0][0]).max() > 0 and np.isfinite(out[0][0]).all()
    for a, b in zip(*out):
        assert np.array_equal(a, b)

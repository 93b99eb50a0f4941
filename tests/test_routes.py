"""That the special passes run where they should: half-range passes, merged
sweeps and pipelined monomial passes, seen in the bytes and blocks that a run
reports, and the branches between half-range and whole runs on one handle."""
import numpy as np
import pytest

import dmsim_workloads as W

pytestmark = pytest.mark.gpu
OP = W.OP


def sim(engine, n, circ, mode="fused", hermitian=1, **kw):
    s = engine.Simulation(n, mode=mode, **kw)
    s.set_option(engine.OPT_HERMITIAN, hermitian)
    s.extend(circ)
    s.upload()
    return s


def run_bytes(s):
    s.run()
    return s.last_timings()["bytes"]


def random_state(n, seed, hermitian):
    d = 1 << n
    rng = np.random.default_rng(seed)
    a = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))) / d
    if hermitian:
        a = (a + a.conj().T) / 2
    return a.T.real.reshape(-1), a.T.imag.reshape(-1)


# ---------------------------------------------------------------- which passes ran
@pytest.mark.parametrize("n", [6, 9, 10, 12, 13])
@pytest.mark.parametrize("mode,arith", [("fused", "fp64"), ("fused", "df64"), ("plain", "fp64")])
def test_half_range_from_ten_qubits_on(engine, n, mode, arith):
    circ = W.qft_then_layers(n, 40, seed=n) + W.table_mix(n, 30, seed=n)
    got = []
    for hermitian in (1, 0):
        with sim(engine, n, circ, mode, hermitian, fused_arith=arith) as s:
            s.set_option(engine.OPT_RECORD, 1)  # no merged sweeps
            got.append(run_bytes(s))
    assert (got[0] != got[1]) == (n >= 10)
    if n >= 12:  # at 10 qubits the mirrors may move as much as the passes save: what they take decides
        assert got[0] < 0.85 * got[1]


@pytest.mark.parametrize("precision,arith", [("fp64", "fp64"), ("fp64", "df64"), ("c64", "fp64")])
@pytest.mark.parametrize("n", [2, 5, 11])
@pytest.mark.parametrize("noise", [False, True])
def test_narrow_passes_are_merged(engine, n, precision, arith, noise):
    """Ten phase and CX gates on two qubits, and channels: one sweep's bytes (a
    recorded run launches them one by one)."""
    with engine.Simulation(n, mode="plain", precision=precision, plain_arith=arith, renorm=0) as s:
        for i in range(5):
            s.append(OP["T"], (i & 1,))
            s.append(OP["CX"], (0, 1) if i & 1 else (1, 0))
        if noise:
            s.append_noise("depolarizing2", (0, 1), 0.1)
            s.append_noise("phase_damping", (1,), 0.1)
        s.upload()
        merged = run_bytes(s)
        s.set_option(engine.OPT_RECORD, 1)
        single = run_bytes(s)
    assert merged < 0.7 * single


@pytest.mark.parametrize("n,merged", [(3, False), (8, False), (10, True)])
def test_double_float_channels_are_merged_where_it_pays(engine, n, merged):
    """A lone warp takes longer for them in a sweep than a pass by itself."""
    with engine.Simulation(n, mode="plain", plain_arith="df64") as s:
        for i in range(12):
            s.append_noise("depolarizing", (i & 1,), 0.1)
        s.upload()
        one = run_bytes(s)
        s.set_option(engine.OPT_RECORD, 1)
        assert (one < run_bytes(s)) == merged


@pytest.mark.parametrize("kind,gate", [("move", "CX"), ("signed", "CZ"), ("phase", "CU1")])
@pytest.mark.parametrize("n,precision,arith", [(10, "fp64", "fp64"), (11, "fp64", "df64"), (11, "c64", "fp64"), (12, "fp64", "fp64")])
@pytest.mark.parametrize("k", [2, 3, 4])
def test_monomial_passes_are_pipelined(engine, n, kind, gate, precision, arith, k):
    """A persistent grid: two blocks an SM, one for 4 qubits."""
    sms = pytest.importorskip("torch").cuda.get_device_properties(0).multi_processor_count
    circ = [(OP[gate], (i, i + 1), 0.3, 0.2, 0.1) for i in range(k - 1)]
    with sim(engine, n, circ, "fused", max_k=k, precision=precision, fused_arith=arith, renorm=0) as s:
        s.set_option(engine.OPT_RECORD, 1)
        s.run()
        rec = s.pass_records()
    rec = rec[rec[:, 0] == k]
    tiles = 4 ** n // (256 << k)
    blocks = sms * (1 if k == 4 else 2)
    assert len(rec) == 1 and rec[0, 1] <= 2 and tiles >= blocks and rec[0, 9] == blocks


# ---------------------------------------------------------------- half range and whole on one handle
def test_written_state_with_a_short_plan_runs_whole(engine):
    """A plan that saves less than the check costs: no check, the whole range,
    and the half range again once the state is known."""
    n = 11
    circ = [(OP["CX"], (i, i + 3), 0, 0, 0) for i in range(4)]
    with sim(engine, n, circ, "plain", 0) as s:
        whole = run_bytes(s)
    for hermitian in (True, False):
        x = random_state(n, 5, hermitian)
        with sim(engine, n, circ, "plain", 0) as s:
            s.set_dm(*x)
            s.run()
            want = s.get_dm()
        with sim(engine, n, circ, "plain") as s:
            s.set_option(engine.OPT_RECORD, 1)
            assert run_bytes(s) < whole  # known: half range
            s.set_dm(*x)
            assert run_bytes(s) == whole
            for a, b in zip(s.get_dm(), want):
                assert np.array_equal(a, b)  # CX moves entries
            s.reset_dm()
            assert run_bytes(s) < whole
            assert abs(s.get_diag()[0] - 1) == 0


def test_half_range_plan_after_an_srn_run(engine):
    """SRN leaves rho without the symmetry: the next circuit on the handle runs whole on it."""
    n = 10
    rng = np.random.default_rng(4)
    srn = [(OP["U3"], (q,), *rng.uniform(0, 6, 3)) for q in range(n)] + [(OP["SRN"], (3,), 0, 0, 0)]
    circ = W.table_mix(n, 40, seed=6)
    out, moved = [], []
    for hermitian in (1, 0):
        with sim(engine, n, srn, "fused", hermitian) as s:
            s.run()
            s.clear_circuit()
            rho = s.rho()
            s.extend(circ)
            s.upload()
            moved.append(run_bytes(s))
            out.append(s.rho())
    assert np.abs(rho - rho.conj().T).max() > 1e-3
    assert moved[0] == moved[1]
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * max(1.0, np.abs(out[1]).max())


@pytest.mark.parametrize("arith,tol", [("fp64", 1e-13), ("df64", 1e-11)])
def test_half_range_channels_with_complex_terms(engine, arith, tol):
    """1- and 2-qubit channels of dense complex superoperators, on high and low qubits."""
    n = 11
    rng = np.random.default_rng(9)

    def kraus(d):
        q, _ = np.linalg.qr(rng.standard_normal((3 * d, d)) + 1j * rng.standard_normal((3 * d, d)))
        return [q[i * d:(i + 1) * d] for i in range(3)]

    program = [((1, 0), kraus(4)), ((10, 3), kraus(4)), ((6,), kraus(2)), ((5, 9), kraus(4)), ((0,), kraus(2))]
    out, moved = [], []
    for hermitian in (1, 0):
        with engine.Simulation(n, mode="plain", plain_arith=arith) as s:
            s.set_option(engine.OPT_HERMITIAN, hermitian)
            for q in range(n):
                s.append(OP["U3"], (q,), 0.3 + q, 0.2, 0.7)
            for qubits, k in program:
                s.append_channel(qubits, k)
            s.upload()
            s.set_option(engine.OPT_RECORD, 1)
            moved.append(run_bytes(s))
            assert (s.pass_records()[:, 1] == 6).sum() == len(program)
            out.append(s.rho())
    assert moved[0] < 0.85 * moved[1]
    assert np.abs(out[0] - out[1]).max() <= tol

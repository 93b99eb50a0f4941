"""Half-range passes (one of every two Hermitian partners rho[r][c], rho[c][r]
is computed, the other copied): the tile enumeration on the CPU, and on the
GPU the same results as passes over the whole state, for Hermitian and for
arbitrary states."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import dmsim_workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dm-sim_gb300", "csrc")


def test_half_maps(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "half_map_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "half_map_check.cpp"), os.path.join(CSRC, "plan.cpp"),
                    os.path.join(CSRC, "gates.cpp"), "-o", exe], check=True, capture_output=True, text=True,
                   timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


def _sim(engine, n, circ, mode, arith, hermitian):
    s = engine.Simulation(n, mode=mode, fused_arith=arith, plain_arith=arith)
    s.set_option(engine.OPT_HERMITIAN, hermitian)
    s.extend(circ)
    s.upload()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "fused"])
@pytest.mark.parametrize("arith", ["fp64", "df64"])
@pytest.mark.parametrize("state", ["basis", "hermitian", "arbitrary", "pointers"])
def test_half_against_whole(engine, mode, arith, state):
    """One circuit twice in a row (chained) on 11 qubits.  An entry of either
    run is within the arithmetic's error of the exact one (2^-48 or 2^-53
    times the terms added, at most some thousands here), so the two differ by
    no more than twice that."""
    n = 11
    circ = W.table_mix(n, 60, seed=21) + W.qft(n)[:40]
    d = 1 << n
    tol = 2e-12 if arith == "fp64" else 2e-10
    runs = []
    for hermitian in (1, 0):
        with _sim(engine, n, circ, mode, arith, hermitian) as s:
            if state in ("hermitian", "arbitrary"):
                rng = np.random.default_rng(3)
                a = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))) / d
                if state == "hermitian":
                    a = (a + a.conj().T) / 2
                s.set_dm(a.T.real.reshape(-1), a.T.imag.reshape(-1))
            if state == "pointers":
                s.device_state()
            s.run()
            s.run()
            runs.append(s.rho())
    assert np.abs(runs[0] - runs[1]).max() <= tol * max(1.0, np.abs(runs[1]).max())
    if state in ("basis", "pointers"):
        assert abs(np.trace(runs[0]) - 1) <= 10 * tol
    if state == "arbitrary":  # nothing was made Hermitian
        assert np.abs(runs[0] - runs[0].conj().T).max() > 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 7, 8, 9, 10, 12, 13])
def test_half_sizes(engine, n):
    """|0..0> through QFT, layers and mixed gates, half against whole."""
    circ = W.qft_then_layers(n, 40, seed=n) + W.table_mix(n, 30, seed=n)
    out = []
    for hermitian in (1, 0):
        with _sim(engine, n, circ, "fused", "fp64", hermitian) as s:
            s.run()
            out.append(s.get_dm())
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("arith", ["fp64", "df64"])
def test_half_tiled_one_qubit_passes(engine, arith):
    """The tiled kernel's half-range instances of every 1-qubit class: at the
    smallest size that runs half, without the register kernel."""
    n = 10
    circ = W.table_mix(n, 20, seed=4) + W.layered_u3_cx(n, 30, seed=4)
    out = []
    for hermitian in (1, 0):
        with engine.Simulation(n, mode="plain", plain_arith=arith, direct1=False) as s:
            s.set_option(engine.OPT_HERMITIAN, hermitian)
            s.extend(circ)
            for q in range(n):
                s.append_noise("depolarizing", (q,), 0.01)
            s.upload()
            s.run()
            out.append(s.get_dm())
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= (1e-12 if arith == "fp64" else 1e-10)

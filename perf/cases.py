"""Timing cases of the density-matrix engine: what its users run, through its public entry points.

Three ways of use:
  * "run":   a ``Simulation`` handle whose circuit is uploaded once; a pass returns rho to |0..0><0..0|, runs the
             circuit and reads the probabilities.  rho itself stays on the device (its own buffers are returned).
  * "call":  a whole call from the drop-in module, as the reference's scripts do it: reset, append every gate, upload
             (planning), run, shots, and rho copied to the host.
  * "sweep": a ``Batch`` of uneven circuits, uploaded once; a pass runs it and reads every diagonal and <ZZ>.

``exact`` restates the circuits with plain torch in 64 bits (statevectors; density matrices where there is noise).
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PY = os.path.join(_ROOT, "dm-sim_gb300", "python")
if _PY not in sys.path:
    sys.path.insert(0, _PY)

import dmsim_gb300 as E  # noqa: E402
import dmsim_workloads as W  # noqa: E402
import libdmsim_py_nvgpu_omp as DM  # noqa: E402

OP = W.OP
SHOTS = 32


def listed():
    return [
        # the headline workload (14 qubits, gates of the mixed table), with fewer gates
        {"name": "fused14_table", "use": "run", "circuit": "table", "n": 14, "gates": 200, "mode": "fused",
         "precision": "fp64", "arith": "fp64"},
        # QFT followed by U3 + CX layers, the 16-qubit configuration one qubit narrower: the largest state
        {"name": "fused15_qft", "use": "run", "circuit": "qft", "n": 15, "gates": 150, "mode": "fused",
         "precision": "fp64", "arith": "fp64"},
        # a mid-size circuit whose state is a little larger than L2
        {"name": "fused12_table", "use": "run", "circuit": "table", "n": 12, "gates": 300, "mode": "fused",
         "precision": "fp64", "arith": "fp64"},
        # the 10-qubit configuration (200 gates of U3 / CX layers), fused: the state fits L2
        {"name": "fused10_layers", "use": "run", "circuit": "layers", "n": 10, "gates": 200, "mode": "fused",
         "precision": "fp64", "arith": "fp64"},
        # the same, gate by gate: the engine's default mode
        {"name": "plain10_layers", "use": "run", "circuit": "layers", "n": 10, "gates": 200, "mode": "plain",
         "precision": "fp64", "arith": "fp64"},
        # the mixed table gate by gate on a state in HBM (odd qubit count)
        {"name": "plain13_table", "use": "run", "circuit": "table", "n": 13, "gates": 40, "mode": "plain",
         "precision": "fp64", "arith": "fp64"},
        # complex64, the U3 / CX / CCX workload of the 17-qubit configuration on 15 qubits
        {"name": "c64_15_ccx", "use": "run", "circuit": "ccx", "n": 15, "gates": 100, "mode": "fused",
         "precision": "c64", "arith": "fp64"},
        # the double-float option
        {"name": "df64_13_table", "use": "run", "circuit": "table", "n": 13, "gates": 150, "mode": "fused",
         "precision": "fp64", "arith": "df64"},
        # a noisy ansatz: depolarising after every gate, amplitude damping after every layer
        {"name": "noise11_hea", "use": "run", "circuit": "noisy", "n": 11, "gates": 96, "mode": "fused",
         "precision": "fp64", "arith": "fp64"},
        # the parameter sweep (6 to 12 qubits, 4 to 10 ansatz layers), an eighth of its 512 circuits
        {"name": "sweep64", "use": "sweep", "circuits": 64, "nmin": 6, "nmax": 12, "lmin": 4, "lmax": 10,
         "shape": 4},
        # one step of a variational loop on 8 qubits, with new angles: the whole call, fused
        {"name": "call8_hea", "use": "call", "circuit": "hea", "n": 8, "gates": 184, "mode": "fused"},
        # the smallest: a short script on 5 qubits, gate by gate
        {"name": "call5_table", "use": "call", "circuit": "table", "n": 5, "gates": 20, "mode": "plain"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fused", "fused", "plain", "c64", "df64", "noise", "sweep", "call"])
    run = {"use": "run", "mode": "fused", "precision": "fp64", "arith": "fp64"}
    if kind in ("fused", "df64"):
        n = rng.randint(7, 14 if kind == "fused" else 13)
        gates = min(_log(rng, 20, 400), 200 * 4 ** (14 - n))
        return dict(run, circuit=rng.choice(["table", "layers", "qft", "ccx"]), n=n, gates=gates,
                    arith="df64" if kind == "df64" else "fp64")
    if kind == "plain":
        n = rng.randint(5, 13)
        return dict(run, circuit=rng.choice(["table", "layers", "ccx"]), n=n, mode="plain",
                    gates=min(_log(rng, 10, 300), 40 * 4 ** (13 - n)), arith=rng.choice(["fp64", "fp64", "df64"]))
    if kind == "c64":
        n = rng.randint(8, 15)
        return dict(run, circuit=rng.choice(["ccx", "layers"]), n=n, precision="c64",
                    gates=min(_log(rng, 20, 300), 100 * 4 ** (15 - n)))
    if kind == "noise":
        n = rng.randint(5, 11)
        return dict(run, circuit="noisy", n=n, gates=_log(rng, 20, 120))
    if kind == "sweep":
        nmin = rng.randint(4, 8)
        lmin = rng.randint(2, 6)
        return {"use": "sweep", "circuits": _log(rng, 6, 64), "nmin": nmin, "nmax": rng.randint(nmin, 12),
                "lmin": lmin, "lmax": lmin + rng.randint(0, 4), "shape": rng.randint(0, 999)}
    n = rng.randint(3, 9)
    return {"use": "call", "circuit": rng.choice(["table", "hea", "layers"]), "n": n, "gates": _log(rng, 10, 250),
            "mode": rng.choice(["plain", "fused"])}


# ---------------------------------------------------------------- inputs
def _circuit(case, seed):
    """[(op, qubits, theta, phi, lam)]; a channel is ("noise kind", qubits, strength)."""
    n, gates, kind = case["n"], case["gates"], case["circuit"]
    if kind == "table":
        return W.table_mix(n, gates, seed=seed)
    if kind == "layers":
        return W.layered_u3_cx(n, gates, seed=seed)
    if kind == "qft":
        return W.qft_then_layers(n, gates, seed=seed)
    if kind == "ccx":
        return W.u3_cx_ccx(n, gates, seed=seed)
    rng = np.random.default_rng(seed)
    hea = W.hea(n, -(-gates // (3 * n - 1)), rng)[:gates]
    if kind == "hea":
        return hea
    out = []
    for i, g in enumerate(hea):
        out.append(g)
        if len(g[1]) == 1:
            out.append(("depolarizing", g[1], float(rng.uniform(0.0, 0.02))))
        else:
            out.append(("depolarizing2", g[1], float(rng.uniform(0.0, 0.03))))
        if (i + 1) % (3 * n - 1) == 0:
            out += [("amplitude_damping", (q,), float(rng.uniform(0.0, 0.05))) for q in range(n)]
    return out


def _sweep(case, seed):
    """[(n, circuit)]: the case says how wide and deep each circuit is, the seed its angles."""
    shape, rng = np.random.default_rng(case["shape"]), np.random.default_rng(seed)
    sizes = [(int(shape.integers(case["nmin"], case["nmax"] + 1)), int(shape.integers(case["lmin"], case["lmax"] + 1)))
             for _ in range(case["circuits"])]
    return [(n, W.hea(n, layers, rng)) for n, layers in sizes]


class _Device:
    """One of rho's device arrays, as a tensor made without a copy; keeps its Simulation alive."""

    def __init__(self, sim, ptr, dtype):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (1 << (2 * sim.n),), "typestr": dtype, "data": (ptr, False),
                                         "version": 3, "strides": None}


def prepare(case, seed):
    if case["use"] == "sweep":
        circuits = _sweep(case, seed)
        b = E.Batch([n for n, _ in circuits])
        for c, (_, circ) in enumerate(circuits):
            b.extend(c, circ)
        b.upload()
        return case, b
    if case["use"] == "call":
        sim = DM.Simulation(case["n"], 1, mode=case["mode"])
        gates = [DM.Gate(g[0], *(list(g[1]) + [0] * (5 - len(g[1]))), g[2], g[3], g[4]) for g in _circuit(case, seed)]
        return case, sim, gates, np.random.default_rng(seed + 1).random(SHOTS)
    key = "fused_arith" if case["mode"] == "fused" else "plain_arith"
    sim = E.Simulation(case["n"], mode=case["mode"], precision=case["precision"], **{key: case["arith"]})
    for g in _circuit(case, seed):
        if isinstance(g[0], str):
            sim.append_noise(g[0], g[1], g[2])
        else:
            sim.append(*g)
    sim.upload()
    dtype = "<f4" if case["precision"] == "c64" else "<f8"
    re, im = (torch.as_tensor(_Device(sim, p, dtype), device="cuda") for p in sim.device_state())
    return case, sim, re, im


def run(state):
    use = state[0]["use"]
    if use == "sweep":
        b = state[1]
        b.run()
        return {"diag": np.concatenate([b.diag(c) for c in range(len(b.nq))]),
                "zz": np.concatenate([b.zz(c) for c in range(len(b.nq))])}
    if use == "call":
        _, sim, gates, uniforms = state
        sim.reset()
        for g in gates:
            sim.append(g)
        sim.upload()
        sim.run()
        shots = sim.measure(SHOTS, uniforms)
        re, im = sim.get_dm()
        return {"shots": np.array(shots, dtype=np.int64), "re": re, "im": im}
    _, sim, re, im = state
    sim.reset_dm()
    sim.run()
    return {"re": re, "im": im, "diag": sim.get_diag()}


def work(case):
    """The state once in and once out, and for every gate a row of the operator's nonzeros on either side."""
    if case["use"] == "sweep":
        circuits = _sweep(case, 0)
        return {"bytes": sum(32.0 * 4 ** n for n, _ in circuits),
                "flops": sum(4.0 ** n * 2 * 8 * sum(2 if len(g[1]) == 1 else 0 for g in c) for n, c in circuits)}
    per = {1: 2, 2: 2, 3: 1, 4: 1, 5: 2}  # nonzeros of a row, about
    flops = 0.0
    for g in _circuit(case, 0):
        if isinstance(g[0], str):
            flops += 4.0 ** case["n"] * 8 * 4
        else:
            flops += 4.0 ** case["n"] * 2 * 8 * per[len(g[1])]
    size = 8 if case.get("precision") == "c64" else 16
    return {"bytes": 2.0 * size * 4 ** case["n"], "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits, with torch
_S2 = math.sqrt(0.5)


def _u3(t, p, l):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return np.array([[c, -np.exp(1j * l) * s], [np.exp(1j * p) * s, np.exp(1j * (p + l)) * c]])


def _u1(l):
    return np.diag([1.0, np.exp(1j * l)])


def _rx(t):
    return np.array([[math.cos(t / 2), -1j * math.sin(t / 2)], [-1j * math.sin(t / 2), math.cos(t / 2)]])


_X = np.array([[0, 1], [1, 0]], dtype=complex)
_Y = np.array([[0, -1j], [1j, 0]])
_H = np.array([[_S2, _S2], [_S2, -_S2]], dtype=complex)


def _ctl(u, controls=1):
    """u on the last qubit of a list, under `controls` qubits before it (index: first qubit most significant)."""
    m = np.eye(2 << controls, dtype=complex)
    m[-2:, -2:] = u
    return m


def _pauli_rot(t, p):
    pp = np.kron(p, p)
    return math.cos(t / 2) * np.eye(4) - 1j * math.sin(t / 2) * pp


def _matrices(g):
    """A gate as [(matrix, qubits)], each up to a phase, in the engine's meaning of the gate."""
    op, q, th, ph, la = g
    name = W.OP_NAMES[op]
    one = {"U3": lambda: _u3(th, ph, la), "U2": lambda: _u3(math.pi / 2, ph, la), "U1": lambda: _u1(la),
           "RX": lambda: _rx(th), "RY": lambda: _u3(th, 0, 0), "RZ": lambda: _u1(ph), "H": lambda: _H,
           "S": lambda: _u1(math.pi / 2), "T": lambda: _u1(math.pi / 4), "X": lambda: _X, "Y": lambda: _Y,
           "Z": lambda: np.diag([1.0, -1.0]), "CX": lambda: _ctl(_X), "CY": lambda: _ctl(_Y),
           "CZ": lambda: _ctl(np.diag([1.0, -1.0])), "CH": lambda: _ctl(_H),
           "SWAP": lambda: np.eye(4)[[0, 2, 1, 3]],
           "CRX": lambda: _ctl(_rx(la)), "CRY": lambda: _ctl(_u3(la, 0, 0)),
           "CRZ": lambda: _ctl(np.diag([np.exp(-0.5j * la), np.exp(0.5j * la)])), "CU1": lambda: _ctl(_u1(la)),
           "CU3": lambda: _ctl(_u3(th, ph, la)), "RXX": lambda: _pauli_rot(th, _X), "RYY": lambda: _pauli_rot(th, _Y),
           "RZZ": lambda: _pauli_rot(th, np.diag([1.0, -1.0])), "CCX": lambda: _ctl(_X, 2),
           "CSWAP": lambda: np.eye(8)[[0, 1, 2, 3, 4, 6, 5, 7]], "C3X": lambda: _ctl(_X, 3)}
    if name in one:
        return [(one[name](), q)]
    assert name == "C4X"  # the engine's C4X is a sequence of its own, not a 4-controlled X
    a, b, c, d, e = q
    root = 0.5 * np.array([[1 - 1j, 1 + 1j], [1 + 1j, 1 - 1j]])
    return [(_H, (e,)), (_ctl(_u1(-math.pi / 2)), (d, e)), (_H, (e,)), (_ctl(_X, 3), (a, b, c, d)), (_H, (d,)),
            (_ctl(_u1(math.pi / 4)), (d, e)), (_H, (d,)), (_ctl(_X, 3), (a, b, c, d)), (_ctl(root, 3), (a, b, c, e))]


def _apply(t, m, axes):
    """The matrix m on the given axes of a tensor of 2s (the first of them the most significant)."""
    k = len(axes)
    m = torch.as_tensor(np.asarray(m, dtype=complex), device=t.device).reshape([2] * (2 * k))
    t = torch.tensordot(m, t, dims=(list(range(k, 2 * k)), list(axes)))
    return torch.movedim(t, list(range(k)), list(axes))


def _psi(n, circuit):
    t = torch.zeros([2] * n, dtype=torch.complex128, device="cuda")
    t[(0,) * n] = 1.0
    for g in circuit:
        for m, qs in _matrices(g):
            t = _apply(t, m, [n - 1 - q for q in qs])
    return t.reshape(-1)


def _kraus(kind, p):
    paulis = [np.eye(2), _X, _Y, np.diag([1.0, -1.0])]
    if kind == "depolarizing":
        return [math.sqrt(1 - 3 * p / 4 if i == 0 else p / 4) * m for i, m in enumerate(paulis)]
    if kind == "depolarizing2":
        return [math.sqrt(1 - 15 * p / 16 if i + j == 0 else p / 16) * np.kron(a, b)
                for i, a in enumerate(paulis) for j, b in enumerate(paulis)]
    return [np.diag([1.0, math.sqrt(1 - p)]), np.array([[0, math.sqrt(p)], [0, 0]])]  # amplitude damping


def _rho(n, circuit):
    """rho[r][c] at [c * 2^n + r]: axes of the bra first."""
    t = torch.zeros([2] * (2 * n), dtype=torch.complex128, device="cuda")
    t[(0,) * (2 * n)] = 1.0
    for g in circuit:
        if isinstance(g[0], str):
            both = sum(np.kron(k.conj(), k) for k in (np.asarray(x, dtype=complex) for x in _kraus(g[0], g[2])))
            t = _apply(t, both, [n - 1 - q for q in g[1]] + [2 * n - 1 - q for q in g[1]])
            continue
        for m, qs in _matrices(g):
            t = _apply(t, m, [2 * n - 1 - q for q in qs])
            t = _apply(t, np.asarray(m).conj(), [n - 1 - q for q in qs])
    return t.reshape(-1)


def exact(case, seed):
    if case["use"] == "sweep":
        diag, zz = [], []
        for n, circ in _sweep(case, seed):
            d = _psi(n, circ).abs().square().cpu().numpy()
            bits = (np.arange(1 << n)[:, None] >> np.arange(n)) & 1
            sign = 1.0 - 2.0 * bits
            diag.append(d)
            zz.append((d[:, None] * sign[:, :-1] * sign[:, 1:]).sum(axis=0))
        return {"diag": np.concatenate(diag), "zz": np.concatenate(zz)}
    circ, n = _circuit(case, seed), case["n"]
    if case["circuit"] == "noisy":
        t = _rho(n, circ)
        re, im = t.real.contiguous(), t.imag.contiguous()
        diag = t.reshape(1 << n, 1 << n).diagonal().real.cpu().numpy()
    else:
        psi = _psi(n, circ)
        pr, pi = psi.real.contiguous(), psi.imag.contiguous()
        re = torch.outer(pr, pr).addr_(pi, pi).reshape(-1)
        im = torch.outer(pr, pi).addr_(pi, pr, alpha=-1).reshape(-1)
        diag = (pr.square() + pi.square()).cpu().numpy()
    if case["use"] == "call":
        return {"shots": None, "re": re.cpu().numpy(), "im": im.cpu().numpy()}
    return {"re": re, "im": im, "diag": diag}

"""Workloads whose time is tracked, through the public API of the `yao_rs`
package: applying circuits to state vectors (one call, or many circuits at
once), density matrices under noise, observables and probabilities, and
energies with their gradients.

listed() gives the fixed cases, draw() further ones of the same ranges.
exact() computes a case's results with torch alone, in 64 bits.
"""
from __future__ import annotations

import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "yao-rs_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

import yao_rs as Y  # noqa: E402

_MODES = {"plain": Y.MODE_PLAIN, "tiled": Y.MODE_TILED, "fused": Y.MODE_FUSED}


def listed():
    return [
        # The smallest call: a dozen qubits or fewer, every kind of gate, run
        # from |0...0> and read back. What a script or the `simulate` command
        # does; launches and latency are all of it.
        {"name": "small_circuit", "task": "simulate", "circuit": "mixed", "n": 9, "depth": 6},
        # The textbook circuit on a given 20-qubit state, gate by gate.
        {"name": "qft_20", "task": "apply", "circuit": "qft", "n": 20, "depth": 1, "mode": "plain", "prec": "c128",
         "k": 0},
        # The default form on a state far larger than the L2 cache.
        {"name": "layered_plain", "task": "apply", "circuit": "layered", "n": 26, "depth": 2, "mode": "plain",
         "prec": "c128", "k": 0},
        # The bit-exact form with several gates a pass, an odd qubit count.
        {"name": "layered_tiled", "task": "apply", "circuit": "layered", "n": 25, "depth": 8, "mode": "tiled",
         "prec": "c128", "k": 0},
        # Deep circuits on large states: the fused form in both precisions.
        {"name": "layered_fused", "task": "apply", "circuit": "layered", "n": 28, "depth": 20, "mode": "fused",
         "prec": "c128", "k": 0},
        {"name": "layered_fused_c64", "task": "apply", "circuit": "layered", "n": 28, "depth": 20, "mode": "fused",
         "prec": "c64", "k": 0},
        # Many circuits of uneven size in one call.
        {"name": "circuit_batch", "task": "batch", "count": 60, "n_min": 10, "n_max": 18, "d_min": 10, "d_max": 40,
         "mode": "fused", "prec": "c128"},
        # An energy and its gradient, the step of a variational optimiser.
        {"name": "vqe_grad", "task": "grad", "n": 22, "depth": 8, "sets": 0},
        # The same for many parameter vectors of one circuit.
        {"name": "vqe_grad_batch", "task": "grad", "n": 13, "depth": 8, "sets": 192},
        # A noisy circuit on a density matrix: the exact Kraus sums (the
        # default) and the fused form.
        {"name": "noisy_plain", "task": "noisy", "n": 11, "depth": 3, "mode": "plain"},
        {"name": "noisy_fused", "task": "noisy", "n": 12, "depth": 8, "mode": "fused"},
        # What is read from a state: a Hamiltonian's expectation value and
        # the marginal probabilities of some qubits.
        {"name": "observables", "task": "observe", "n": 24, "measured": 9, "prec": "c128"},
    ]


def draw(rng):
    task = rng.choice(["simulate", "apply", "apply", "apply", "batch", "grad", "grad", "noisy", "noisy", "observe"])
    if task == "simulate":
        return {"task": task, "circuit": rng.choice(["mixed", "qft", "layered"]), "n": rng.randint(3, 13),
                "depth": rng.randint(1, 8)}
    if task == "apply":
        mode = rng.choice(["plain", "tiled", "fused"])
        n = rng.randint(14, {"plain": 26, "tiled": 26, "fused": 28}[mode])
        circuit = rng.choice(["mixed", "qft", "layered", "layered"])
        depth = rng.randint(1, 4 if mode == "plain" and n > 22 else 8)
        k = rng.choice([0, 0, 3, 4, 5]) if mode == "fused" else 0
        return {"task": task, "circuit": circuit, "n": n, "depth": 1 if circuit == "qft" else depth, "mode": mode,
                "prec": rng.choice(["c128", "c64"]), "k": k}
    if task == "batch":
        lo = rng.randint(5, 12)
        d = rng.randint(2, 16)
        return {"task": task, "count": rng.randint(3, 60), "n_min": lo, "n_max": lo + rng.randint(0, 5), "d_min": d,
                "d_max": d + rng.randint(0, 16), "mode": rng.choice(["tiled", "fused", "fused"]),
                "prec": rng.choice(["c128", "c128", "c64"])}
    if task == "grad":
        if rng.random() < 0.5:
            return {"task": task, "n": rng.randint(6, 22), "depth": rng.randint(1, 8), "sets": 0}
        n = rng.randint(6, 14)
        sets = int(round(math.exp(rng.uniform(math.log(3), math.log(1 << (20 - n))))))
        return {"task": task, "n": n, "depth": rng.randint(1, 8), "sets": sets}
    if task == "noisy":
        mode = rng.choice(["plain", "fused"])
        return {"task": task, "n": rng.randint(3, 11 if mode == "plain" else 12), "depth": rng.randint(1, 3),
                "mode": mode}
    n = rng.randint(10, 24)
    return {"task": task, "n": n, "measured": rng.randint(1, 10), "prec": rng.choice(["c128", "c64"])}


# --------------------------------------------------------------- workloads
# A circuit is a list of (gate, parameters, targets, controls); locations
# count from the most significant qubit. Drawn structures depend on the
# case alone, angles on the seed too, as in a program that runs one ansatz
# with new parameters.

def _structure_rng(case):
    return random.Random(repr(sorted((k, v) for k, v in case.items() if k != "name")))


def _layered(n, depth, angles):
    """Rx, Ry, Rz on every qubit, then a CNOT brickwork."""
    gates = []
    for layer in range(depth):
        for q in range(n):
            for g in ("Rx", "Ry", "Rz"):
                gates.append((g, (angles.uniform(0.0, 2.0 * math.pi),), (q,), ()))
        gates += [("X", (), (q + 1,), (q,)) for q in range(layer % 2, n - 1, 2)]
    return gates


def _qft(n):
    gates = []
    for i in range(n):
        gates.append(("H", (), (i,), ()))
        gates += [("Phase", (2.0 * math.pi / 2 ** (j + 1),), (i,), (i + j,)) for j in range(1, n - i)]
    return gates + [("SWAP", (), (i, n - 1 - i), ()) for i in range(n // 2)]


def _mixed(n, depth, shape, angles):
    """Named gates of every kind on random locations, some controlled."""
    gates = []
    for _ in range(depth * n):
        name = shape.choice(["H", "X", "Y", "Z", "S", "T", "Rx", "Ry", "Rz", "Phase", "SWAP", "FSim", "X", "Phase"])
        nt = 2 if name in ("SWAP", "FSim") else 1
        nc = shape.choice([0, 0, 1, 1, 2]) if name in ("X", "Z", "Ry", "Phase") else 0
        locs = shape.sample(range(n), nt + min(nc, n - nt))
        np_ = {"Rx": 1, "Ry": 1, "Rz": 1, "Phase": 1, "FSim": 2}.get(name, 0)
        gates.append((name, tuple(angles.uniform(-math.pi, math.pi) for _ in range(np_)), tuple(locs[:nt]),
                      tuple(locs[nt:])))
    return gates


def _circuit(case, n, depth, seed, salt=0):
    angles = random.Random(seed * 1000003 + salt)
    kind = case.get("circuit", "layered")
    if kind == "qft":
        return _qft(n)
    if kind == "mixed":
        return _mixed(n, depth, _structure_rng(case), angles)
    return _layered(n, depth, angles)


def _batch_shapes(case):
    rng = _structure_rng(case)
    return [(rng.randint(case["n_min"], case["n_max"]), rng.randint(case["d_min"], case["d_max"]))
            for _ in range(case["count"])]


def _ansatz(n, params):
    """Layers of Ry, Rz on every qubit and a CNOT ring."""
    gates, it = [], iter(params)
    for _ in range(len(params) // (2 * n)):
        for q in range(n):
            gates.append(("Ry", (float(next(it)),), (q,), ()))
            gates.append(("Rz", (float(next(it)),), (q,), ()))
        gates += [("X", (), ((q + 1) % n,), (q,)) for q in range(n)]
    return gates


def _params(case, seed):
    rng = np.random.default_rng([2024, seed])
    return rng.uniform(-math.pi, math.pi, size=(max(1, case["sets"]), 2 * case["n"] * case["depth"]))


def _tfim(n):
    """Transverse-field Ising chain: (coefficient, ((site, op), ...)) terms."""
    return ([(-1.0, ((i, "Z"), ((i + 1) % n, "Z"))) for i in range(n)] + [(-1.0, ((i, "X"),)) for i in range(n)])


def _noisy(case, seed):
    """Ry, Rz and a CZ brickwork, each gate followed by depolarizing noise on
    its qubits, and amplitude damping on every qubit at a layer's end."""
    n, angles, ops = case["n"], random.Random(seed * 7919 + 1), []
    for layer in range(case["depth"]):
        for q in range(n):
            for g in ("Ry", "Rz"):
                ops.append((g, (angles.uniform(0.0, 2.0 * math.pi),), (q,), ()))
                ops.append(("depolarize", (1e-3,), (q,), ()))
        for q in range(layer % 2, n - 1, 2):
            ops.append(("Z", (), (q + 1,), (q,)))
            ops.append(("depolarize", (1e-3,), (q, q + 1), ()))
        ops += [("damp", (1e-3,), (q,), ()) for q in range(n)]
    return ops


def _state(n, seed):
    rng = np.random.default_rng([n, seed])
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return v / np.linalg.norm(v)


def _measured(case):
    return _structure_rng(case).sample(range(case["n"]), min(case["measured"], case["n"]))


# --------------------------------------------------------- the calls timed

def _build(n, gates):
    els = []
    for name, params, targets, controls in gates:
        if name == "depolarize":
            els.append(Y.channel(targets, Y.NoiseChannel.Depolarizing(len(targets), params[0])))
        elif name == "damp":
            els.append(Y.channel(targets, Y.NoiseChannel.AmplitudeDamping(params[0])))
        else:
            gate = getattr(Y.Gate, name)(*params) if params else getattr(Y.Gate, name)
            els.append(Y.control(controls, targets, gate) if controls else Y.put(targets, gate))
    return Y.Circuit.qubits(n, els)


def _operator(terms):
    return Y.OperatorPolynomial([c for c, _ in terms],
                                [Y.OperatorString([(s, getattr(Y.Op, o)) for s, o in ops]) for _, ops in terms])


class _Amplitudes:
    """A register's device memory, for torch (which keeps this alive)."""

    def __init__(self, reg):
        self.reg, p = reg, ctypes.c_void_p()
        Y._abi.check(Y._abi.lib().yao_reg_device_ptr(reg.handle, ctypes.byref(p)))
        self.__cuda_array_interface__ = {
            "shape": (1 << reg.nbits(),), "typestr": "<c16" if reg.precision == Y.C128 else "<c8",
            "data": (p.value, False), "version": 3, "strides": None}


def _amplitudes(reg):
    return torch.as_tensor(_Amplitudes(reg), device="cuda")


def _precision(case):
    return Y.C64 if case.get("prec") == "c64" else Y.C128


def _start_is_zero(case):
    return case["n"] > 22  # larger circuits start from |0...0>, smaller ones from a given state


def prepare(case, seed):
    task, n = case["task"], case.get("n")
    state = {"case": dict(case)}
    if task == "simulate":
        state["circuit"] = _build(n, _circuit(case, n, case["depth"], seed))
    elif task == "apply":
        state["circuit"] = _build(n, _circuit(case, n, case["depth"], seed))
        reg = Y.ArrayReg.zero_state(n) if _start_is_zero(case) else Y.ArrayReg.from_vec(n, _state(n, seed))
        state["reg"] = reg.to_precision(Y.C64) if case["prec"] == "c64" else reg
    elif task == "batch":
        state["shapes"] = _batch_shapes(case)
        state["circuits"] = [_build(m, _circuit(case, m, d, seed, i)) for i, (m, d) in enumerate(state["shapes"])]
    elif task == "grad":
        state["params"] = _params(case, seed)
        state["circuit"] = _build(n, _ansatz(n, state["params"][0]))
        state["hamiltonian"] = _operator(_tfim(n))
        state["reg"] = Y.ArrayReg.zero_state(n)
    elif task == "noisy":
        state["circuit"] = _build(n, _noisy(case, seed))
        state["reg"] = Y.ArrayReg.zero_state(n)
        state["z"] = [_operator([(1.0, ((s, "Z"),))]) for s in range(n)]
    else:
        reg = Y.ArrayReg.from_vec(n, _state(n, seed))
        state["reg"] = reg.to_precision(Y.C64) if case["prec"] == "c64" else reg
        state["hamiltonian"] = _operator(_tfim(n))
        state["locs"] = _measured(case)
    return state


def run(state):
    case = state["case"]
    task = case["task"]
    if task == "simulate":
        reg = Y.ArrayReg.zero_state(case["n"])
        Y.apply_inplace(state["circuit"], reg)
        return reg.state_vec()
    if task == "apply":
        return _amplitudes(Y.apply(state["circuit"], state["reg"], _MODES[case["mode"]], case["k"]))
    if task == "batch":
        regs = [Y.ArrayReg.zero_state(m, _precision(case)) for m, _ in state["shapes"]]
        Y.batch_apply(state["circuits"], regs, _MODES[case["mode"]])
        return [_amplitudes(r) for r in regs]
    if task == "grad":
        if case["sets"]:
            return list(Y.expect_grad_batch(state["hamiltonian"], state["circuit"], state["params"], state["reg"]))
        value, grad = Y.expect_grad(state["hamiltonian"], state["circuit"], state["reg"])
        return [value, np.array(grad)]
    if task == "noisy":
        rho = Y.DensityMatrix.from_reg(state["reg"])
        rho.apply(state["circuit"], _MODES[case["mode"]])
        # the matrix itself is read where it is small; from large ones, as
        # programs do, the outcome probabilities, <Z> of every qubit and the
        # purity (a sum over every entry)
        out = {"probs": Y.probs(rho), "z": np.array([Y.expect_dm(rho, z) for z in state["z"]]),
               "purity": rho.purity()}
        if case["n"] <= 8:
            out["rho"] = rho.state_data()
        return out
    energy = Y.expect_arrayreg(state["reg"], state["hamiltonian"])
    return {"energy": np.array([energy]), "probs": Y.probs(state["reg"], state["locs"])}


# ------------------------------------------------------------------ bounds

def _gate_flops(name, controls):
    """Real operations per amplitude of the whole state."""
    full = {"X": 0.0, "SWAP": 0.0, "Z": 0.5, "S": 3.0, "T": 3.0, "Phase": 3.0, "Y": 1.0, "H": 6.0, "Rx": 6.0,
            "Ry": 6.0, "Rz": 6.0, "FSim": 10.0, "depolarize": 4.0, "damp": 3.0}
    return full[name] / 2 ** len(controls)


def work(case):
    task, n = case["task"], case.get("n")
    size = 8 if case.get("prec") == "c64" else 16
    if task in ("simulate", "apply"):
        gates = _circuit(case, n, case["depth"], 0)
        flops = sum(_gate_flops(g[0], g[3]) for g in gates) * 2.0 ** n
        return {"bytes": (1 if task == "simulate" else 2) * size * 2.0 ** n, "flops": flops}
    if task == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(size * 2.0 ** m for m, _ in shapes), "flops": sum(18.0 * m * d * 2.0 ** m for m, d in shapes)}
    if task == "grad":
        sets = max(1, case["sets"])
        params = 2 * n * case["depth"]
        # forward, then both states backward; the Hamiltonian; the input read once, the results written
        return {"bytes": 16 * 2.0 ** n + 8.0 * sets * (2 * params + 1),
                "flops": sets * 2.0 ** n * (params * (6 + 2 * 6 + 4) + 2 * n * 2)}
    if task == "noisy":
        flops = sum(_gate_flops(g[0], g[3]) * (1 if g[0] in ("depolarize", "damp") else 2) for g in _noisy(case, 0))
        return {"bytes": 16 * 2.0 ** n + 8 * 2.0 ** n, "flops": flops * 4.0 ** n}
    return {"bytes": size * 2.0 ** n + 8 * 2.0 ** len(_measured(case)), "flops": 2.0 ** n * (3 * n + 3)}


# --------------------------------------------------- the same with torch
# Amplitudes as a complex128 tensor of shape (sets, 2^n); a gate's matrix
# may hold one value a set.

def _axes(psi, n, locs):
    """psi with an axis of length 2 for each of the locations, and those axes."""
    shape, at, prev = [psi.shape[0]], {}, 0
    for loc in sorted(locs):
        shape += [1 << (loc - prev), 2]
        at[loc], prev = len(shape) - 1, loc + 1
    return psi.view(shape + [1 << (n - prev)]), at


def _cell(view, at, bits):
    index = [slice(None)] * view.dim()
    for loc, b in bits.items():
        index[at[loc]] = b
    return view[tuple(index)]


def _matrix(name, params, device):
    """Rows of the gate's matrix: numbers, or one value a set."""
    p = [torch.as_tensor(np.atleast_1d(x), dtype=torch.float64, device=device) for x in params]
    half = [x / 2 for x in p]
    r, z = math.sqrt(0.5), 0.0
    if name == "X":
        return [[z, 1.0], [1.0, z]]
    if name == "Y":
        return [[z, -1j], [1j, z]]
    if name == "Z":
        return [[1.0, z], [z, -1.0]]
    if name == "S":
        return [[1.0, z], [z, 1j]]
    if name == "T":
        return [[1.0, z], [z, complex(r, r)]]
    if name == "H":
        return [[r, r], [r, -r]]
    if name == "Phase":
        return [[1.0, z], [z, torch.exp(1j * p[0])]]
    if name == "Rx":
        c, s = torch.cos(half[0]), torch.sin(half[0])
        return [[c + 0j, -1j * s], [-1j * s, c + 0j]]
    if name == "Ry":
        c, s = torch.cos(half[0]) + 0j, torch.sin(half[0]) + 0j
        return [[c, -s], [s, c]]
    if name == "Rz":
        return [[torch.exp(-1j * half[0]), z], [z, torch.exp(1j * half[0])]]
    if name == "SWAP":
        return [[1.0, z, z, z], [z, z, 1.0, z], [z, 1.0, z, z], [z, z, z, 1.0]]
    c, s = torch.cos(p[0]) + 0j, -1j * torch.sin(p[0])  # FSim
    return [[1.0, z, z, z], [z, c, s, z], [z, s, c, z], [z, z, z, torch.exp(-1j * p[1])]]


def _times(m, x):
    if isinstance(m, torch.Tensor):
        return x * (m.reshape([-1] + [1] * (x.dim() - 1)) if m.numel() > 1 else m.item())
    return x * m


def _dagger(m):
    conj = [[x.conj() if isinstance(x, torch.Tensor) else complex(x).conjugate() for x in row] for row in m]
    return [[conj[c][r] for c in range(len(m))] for r in range(len(m))]


def _nonzero(x):
    return isinstance(x, torch.Tensor) or x != 0.0


def _gate(psi, n, m, targets, controls=()):
    """psi with the gate applied, in place (2-qubit matrices: the first target is the low index bit)."""
    view, at = _axes(psi, n, list(targets) + list(controls))
    on = {c: 1 for c in controls}
    cells = [_cell(view, at, {**on, **{t: (i >> q) & 1 for q, t in enumerate(targets)}}) for i in range(len(m))]
    if not any(_nonzero(x) for r, row in enumerate(m) for c, x in enumerate(row) if r != c):  # diagonal
        for cell, x in zip(cells, (m[i][i] for i in range(len(m)))):
            if isinstance(x, torch.Tensor) or x != 1.0:
                cell.copy_(_times(x, cell))
        return psi
    old = [cell.clone() for cell in cells]
    for cell, row in zip(cells, m):
        cell.copy_(sum(_times(x, o) for x, o in zip(row, old) if _nonzero(x)))
    return psi


def _run_gates(psi, n, gates):
    for name, params, targets, controls in gates:
        _gate(psi, n, _matrix(name, params, psi.device), targets, controls)
    return psi


def _pauli(psi, n, ops):
    out = psi.clone()
    for site, op in ops:
        _gate(out, n, _matrix(op, (), psi.device), (site,))
    return out


def _hamiltonian(psi, n, terms):
    out = torch.zeros_like(psi)
    for c, ops in terms:
        out += c * _pauli(psi, n, ops)
    return out


def _zero(n, device, sets=1):
    psi = torch.zeros((sets, 1 << n), dtype=torch.complex128, device=device)
    psi[:, 0] = 1.0
    return psi


def _gradient(case, params, device):
    n, sets = case["n"], params.shape[0]
    gates = []
    for name, p, targets, controls in _ansatz(n, np.arange(params.shape[1])):
        gates.append((name, (params[:, int(p[0])],) if p else (), targets, controls, int(p[0]) if p else -1))
    psi = _run_gates(_zero(n, device, sets), n, [g[:4] for g in gates])
    lam = _hamiltonian(psi, n, _tfim(n))
    value = (psi.conj() * lam).sum(1).real
    grad = torch.zeros((sets, params.shape[1]), dtype=torch.float64, device=device)
    for name, p, targets, controls, at in reversed(gates):
        if at >= 0:  # d/dtheta exp(-i theta P / 2) = -i/2 P
            op = {"Ry": "Y", "Rz": "Z"}[name]
            grad[:, at] = 2.0 * (-0.5j * (lam.conj() * _pauli(psi, n, ((targets[0], op),))).sum(1)).real
        back = _dagger(_matrix(name, p, device))
        _gate(psi, n, back, targets, controls)
        _gate(lam, n, back, targets, controls)
    return value, grad


def _noisy_exact(case, seed, device):
    n = case["n"]
    rho = _zero(2 * n, device)
    for name, params, targets, controls in _noisy(case, seed):
        bra = tuple(t + n for t in targets)
        if name == "depolarize":
            view, at = _axes(rho, 2 * n, targets + bra)
            d, p = 1 << len(targets), params[0]
            at_ = [{t: (i >> q) & 1 for q, t in enumerate(targets)} | {t: (i >> q) & 1 for q, t in enumerate(bra)}
                   for i in range(d)]
            mean = sum(_cell(view, at, b) for b in at_) * (p / d)
            rho *= 1.0 - p
            for b in at_:
                _cell(view, at, b).add_(mean)
        elif name == "damp":
            view, at = _axes(rho, 2 * n, targets + bra)
            g, (t,), (u,) = params[0], targets, bra
            _cell(view, at, {t: 0, u: 0}).add_(g * _cell(view, at, {t: 1, u: 1}))
            _cell(view, at, {t: 1, u: 1}).mul_(1.0 - g)
            _cell(view, at, {t: 0, u: 1}).mul_(math.sqrt(1.0 - g))
            _cell(view, at, {t: 1, u: 0}).mul_(math.sqrt(1.0 - g))
        else:
            m = _matrix(name, params, device)
            _gate(rho, 2 * n, m, targets, controls)
            conj = [[x.conj() if isinstance(x, torch.Tensor) else complex(x).conjugate() for x in row] for row in m]
            _gate(rho, 2 * n, conj, bra, tuple(c + n for c in controls))
    return rho


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    task, n = case["task"], case.get("n")
    if task == "simulate":
        gates = _circuit(case, n, case["depth"], seed)
        return _run_gates(_zero(n, device), n, gates)[0].cpu().numpy()
    if task == "apply":
        gates = _circuit(case, n, case["depth"], seed)
        if len(gates) * 2.0 ** n > 2.0 ** 38:
            return None
        if _start_is_zero(case):
            psi = _zero(n, device)
        else:
            psi = torch.as_tensor(_state(n, seed), device=device)[None].clone()
            if case["prec"] == "c64":
                psi = psi.to(torch.complex64).to(torch.complex128)
        return _run_gates(psi, n, gates)[0]
    if task == "batch":
        return [_run_gates(_zero(m, device), m, _circuit(case, m, d, seed, i))[0]
                if m * d < 400 else None for i, (m, d) in enumerate(_batch_shapes(case))]
    if task == "grad":
        value, grad = _gradient(case, _params(case, seed), device)
        if case["sets"]:
            return [value.cpu().numpy(), grad.cpu().numpy()]
        return [float(value[0]), grad[0].cpu().numpy()]
    if task == "noisy":
        rho = _noisy_exact(case, seed, device)[0]
        probs = rho.view(1 << n, 1 << n).diagonal().real.contiguous()
        index = torch.arange(1 << n, device=device)
        # an observable's site s of a density matrix is bit s of the index
        z = [((1 - 2 * ((index >> s) & 1)) * probs).sum().item() for s in range(n)]
        out = {"probs": probs.cpu().numpy(), "z": np.array(z, dtype=np.complex128),
               "purity": float((rho.real ** 2 + rho.imag ** 2).sum())}
        if n <= 8:
            out["rho"] = rho.cpu().numpy()
        return out
    psi = torch.as_tensor(_state(n, seed), device=device)[None].clone()
    if case["prec"] == "c64":
        psi = psi.to(torch.complex64).to(torch.complex128)
    energy = (psi.conj() * _hamiltonian(psi, n, _tfim(n))).sum()
    locs = _measured(case)
    view, at = _axes((psi.real ** 2 + psi.imag ** 2), n, locs)
    keep = [at[l] for l in locs]
    view = view.sum(dim=[d for d in range(view.dim()) if d not in keep])
    order = sorted(locs)  # the axes left are in ascending location; outcomes have locs[0] as the high bit
    probs = view.permute([order.index(l) for l in locs]).reshape(-1)
    return {"energy": np.array([energy.item()]), "probs": probs.cpu().numpy()}

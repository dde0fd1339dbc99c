"""Register passes (csrc/reg_tiles.cu): TILED and FUSED runs of 1- and
2-qubit gates against the oracle, over register counts around the tile and
thread-layout edges."""
import math

import numpy as np
import pytest

import oracle as O
import yao_rs as Y
from helpers import layered_circuit, random_circuit, random_state, random_unitary
from yao_rs import Gate

pytestmark = pytest.mark.gpu


def mixed_circuit(rng, n, depth):
    """Named gates, controls of either value, 2-qubit matrices (one of them
    not unitary), diagonals of up to three qubits, CNOTs between rotations."""
    els = []
    for _ in range(depth):
        q = [int(x) for x in rng.permutation(n)]
        els.append(Y.put([q[0]], Gate.Ry(float(rng.uniform(-3, 3)))))
        els.append(Y.put([q[1]], Gate.Rx(float(rng.uniform(-3, 3)))))
        els.append(Y.PositionedGate(Gate.X, [q[0]], [q[1]], [bool(rng.integers(2))]))
        els.append(Y.put([q[0]], Gate.Rz(float(rng.uniform(-3, 3)))))
        els.append(Y.put([q[0]], Gate.Rx(float(rng.uniform(-3, 3)))))
        els.append(Y.put(q[:2], Gate.Custom(random_unitary(rng, 4))))
        els.append(Y.PositionedGate(Gate.Ry(0.4), [q[2]], q[:2], [True, False]))
        els.append(Y.put([q[2], q[0]], Gate.SWAP))
        els.append(Y.put(q[:3], Gate.Custom(np.diag(np.exp(1j * rng.uniform(-3, 3, 8))), True)))
        els.append(Y.control([q[1]], [q[2]], Gate.Z))
        els.append(Y.put([q[2]], Gate.H))
        els.append(Y.PositionedGate(Gate.Phase(0.7), [q[1]], [q[0]], [False]))
        els.append(Y.put([q[1]], Gate.T))
    els.append(Y.put([0], Gate.Custom(np.array([[1.0, 0.25], [0.0, 1.0]]))))
    els.append(Y.put([n - 1], Gate.Custom(np.diag([1.0, 0.5j]), True)))
    return Y.Circuit.qubits(n, els)


def circuits(rng, n):
    yield mixed_circuit(rng, n, 6)
    yield layered_circuit(n, 3, seed=n)
    yield random_circuit(rng, n, 60, max_ctrl=min(3, n - 1), custom=False)
    yield Y.Circuit.qubits(n, [Y.put([q], g) for q in range(n) for g in (Gate.X, Gate.Z, Gate.X, Gate.S)])


# n = 4: the smallest; 11/12/13: one tile, two, four; 19..21: 4, 8 or 16
# amplitudes a thread
@pytest.mark.parametrize("n", [4, 5, 7, 8, 10, 11, 12, 13, 16, 19, 20, 21])
def test_register_passes(n):
    rng = np.random.default_rng(n)
    for c in circuits(rng, n):
        psi = random_state(rng, n)
        ref = O.apply_circuit(c, psi)
        norm = float(np.linalg.norm(ref))
        r = Y.ArrayReg.from_vec(n, psi)
        Y.apply_inplace(c, r, Y.MODE_TILED)
        assert np.max(np.abs(r.state_vec() - ref)) == 0.0
        # FP64: a few roundings of 1.1e-16 a gate on amplitudes below 1;
        # FP32: 6e-8 a gate and amplitude, so at most 6e-8 x gates of the norm
        for k in (0, 1, 2):
            r = Y.ArrayReg.from_vec(n, psi)
            Y.apply_inplace(c, r, Y.MODE_FUSED, k)
            assert np.max(np.abs(r.state_vec() - ref)) < 1e-13 * norm, k
            r = Y.ArrayReg.from_vec(n, psi).to_precision(Y.C64)
            Y.apply_inplace(c, r, Y.MODE_FUSED, k)
            assert np.linalg.norm(r.state_vec() - ref) < 6e-8 * len(c.elements) * norm, k


@pytest.mark.parametrize("n", [3, 4, 8, 11, 12, 14, 17, 20])
def test_plain_runs_are_the_same_bits(n):
    """PLAIN shares passes among gates: every bit, signed zeros among them, is
    the oracle's, and every bit and NaN that of one launch a gate (circuits
    of one gate) on states with infinities and NaN, where the launches leave
    amplitudes alone that a diagonal entry of exactly 1 meets.  Gates on
    three qubits are launches of their own in between."""
    rng = np.random.default_rng(50 + n)
    for c in (random_circuit(rng, n, 80, max_ctrl=min(3, n - 1)), layered_circuit(n, 2, seed=n)):
        psi = random_state(rng, n)
        r = Y.ArrayReg.from_vec(n, psi)
        Y.apply_inplace(c, r)
        assert np.array_equal(r.state_vec().view(np.uint64), O.apply_circuit(c, psi).view(np.uint64))
        psi[1], psi[2], psi[5] = np.inf, complex(0.5, np.nan), complex(0.0, -np.inf)
        r, one = Y.ArrayReg.from_vec(n, psi), Y.ArrayReg.from_vec(n, psi)
        Y.apply_inplace(c, r)
        for el in c.elements:
            Y.apply_inplace(Y.Circuit.qubits(n, [el]), one)
        got, ref = r.state_vec().view(np.float64), one.state_vec().view(np.float64)
        finite = ~np.isnan(ref)
        assert np.array_equal(np.isnan(got), ~finite)
        assert np.array_equal(got.view(np.uint64)[finite], ref.view(np.uint64)[finite])


def test_long_program_splits_its_description():
    """More gates on one tile than one pass describes."""
    rng = np.random.default_rng(0)
    c = random_circuit(rng, 11, 900, max_ctrl=2, custom=False)
    psi = random_state(rng, 11)
    ref = O.apply_circuit(c, psi)
    for mode, tol in ((Y.MODE_TILED, 0.0), (Y.MODE_FUSED, 1e-12)):
        r = Y.ArrayReg.from_vec(11, psi)
        Y.apply_inplace(c, r, mode, 1 if mode == Y.MODE_FUSED else 0)
        assert np.max(np.abs(r.state_vec() - ref)) <= tol


def test_plain_copies_instead_of_tma(monkeypatch):
    """YAO_TMA=0: tiles move by plain loads, with the same result."""
    monkeypatch.setenv("YAO_TMA", "0")
    for n in (13, 20):
        rng = np.random.default_rng(n)
        c = mixed_circuit(rng, n, 2)
        psi = random_state(rng, n)
        r = Y.ArrayReg.from_vec(n, psi)
        Y.apply_inplace(c, r, Y.MODE_TILED)
        assert np.max(np.abs(r.state_vec() - O.apply_circuit(c, psi))) == 0.0
        assert math.isfinite(r.norm())


@pytest.mark.parametrize("n", [20, 21])
@pytest.mark.parametrize("gates", [("Ry",), ("Ry", "Rz"), ("Rx", "Ry", "Rz")])
def test_layers_of_rotations(n, gates):
    """Four rotations at a time with one diagonal for their phases and the
    signs of CZs among them (16 amplitudes a thread: 2^20 complex128, 2^21
    complex64), CZs and CNOTs on random pairs and some on three qubits in
    between; without phases (Ry) the signs are an op of their own."""
    rng = np.random.default_rng([n, len(gates)])
    els = []
    for _ in range(4):
        els += [Y.put([q], getattr(Gate, g)(float(rng.uniform(-3, 3)))) for q in range(n) for g in gates]
        for _ in range(n):
            p = [int(x) for x in rng.permutation(n)]
            if rng.random() < 0.1:
                els.append(Y.control(p[:2], [p[2]], Gate.Z))
            else:
                els.append(Y.control([p[0]], [p[1]], Gate.Z if rng.random() < 0.7 else Gate.X))
        els += [Y.put([q], Gate.Ry(float(rng.uniform(-3, 3)))) for q in range(0, n, 3)]
    c, psi = Y.Circuit.qubits(n, els), random_state(rng, n)
    ref = O.apply_circuit(c, psi)
    # a few roundings (1.1e-16, 6e-8) a gate on a state of norm 1
    for prec, eps in ((Y.C128, 5e-16), (Y.C64, 6e-8)):
        r = Y.ArrayReg.from_vec(n, psi).to_precision(prec)
        Y.apply_inplace(c, r, Y.MODE_FUSED, 1)
        assert np.linalg.norm(r.state_vec() - ref) < eps * len(els), prec

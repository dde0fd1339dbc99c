"""Gradients by the register sweep (csrc/sweep.cu), of one and of several
parameter vectors, against the oracle at register counts around its tile
and thread edges."""
import os
import subprocess
import sys
import time
from pathlib import Path

import numpy as np
import pytest

import oracle as O
import yao_rs as Y
from helpers import random_state
from yao_rs import Gate


def ansatz(rng, n, layers, kind):
    """0: Ry, Rz and a CNOT ring; 1: Hadamards, constants and every 1-parameter
    gate in a run; 2: sparse runs.  1 and 2 are entangled by CNOTs with
    controls of either value (one or two), CZ, SWAP and controlled SWAP."""
    def t():
        return float(rng.uniform(-3, 3))
    els = []
    for _ in range(layers):
        for q in range(n):
            run = ([Gate.Ry(t()), Gate.Rz(t())] if kind == 0 else
                   [Gate.H, Gate.Rx(t()), Gate.Phase(t()), Gate.Ry(t()), Gate.T] if kind == 1 else
                   [Gate.Rz(t())] if rng.random() < 0.5 else [Gate.X, Gate.Rx(t()), Gate.Y])
            els += [Y.put([q], g) for g in run]
        for q in range(n):
            p, r = [int(x) for x in rng.permutation(n)], rng.random()
            if kind == 0:
                els.append(Y.control([q], [(q + 1) % n], Gate.X))
            elif r < 0.4:
                els.append(Y.PositionedGate(Gate.X, [p[0]], [p[1]], [bool(rng.integers(2))]))
            elif r < 0.6:
                els.append(Y.control([p[0]], [p[1]], Gate.Z))
            elif r < 0.75:
                els.append(Y.put(p[:2], Gate.SWAP))
            elif r < 0.9:
                els.append(Y.PositionedGate(Gate.X, [p[0]], p[1:3], [True, False]))
            else:
                els.append(Y.PositionedGate(Gate.SWAP, p[:2], [p[2]], [False]))
    return Y.Circuit.qubits(n, els)


def hamiltonian(n):
    cs, ss = [0.3], [Y.OperatorString([(0, Y.Op.Y), (n - 1, Y.Op.X)])]
    for i in range(n):
        cs += [-1.0, 0.7]
        ss += [Y.OperatorString([(i, Y.Op.Z), ((i + 1) % n, Y.Op.Z)]), Y.OperatorString([(i, Y.Op.X)])]
    return Y.OperatorPolynomial(cs, ss)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 4, 7, 8, 10, 11, 12, 13, 14])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_gradients(n, kind):
    rng = np.random.default_rng([n, kind])
    c, h, psi = ansatz(rng, n, 3, kind), hamiltonian(n), random_state(rng, n)
    reg = Y.ArrayReg.from_vec(n, psi)
    # a few hundred gates of 1.1e-16 each on terms of magnitude 1.7 n
    tol = 1e-12
    value, grad = O.expect_grad(h, c, psi)
    v, g = Y.expect_grad(h, c, reg)
    assert abs(v - value) < tol and np.max(np.abs(np.array(g) - np.array(grad))) < tol
    sets = rng.uniform(-3, 3, size=(7, c.num_params()))
    sets[2] = c.parameters()
    vs, gs = Y.expect_grad_batch(h, c, sets, reg)
    assert abs(vs[2] - value) < tol and np.max(np.abs(gs[2] - np.array(grad))) < tol
    c.dispatch(list(sets[6]))
    value, grad = O.expect_grad(h, c, psi)
    assert abs(vs[6] - value) < tol and np.max(np.abs(gs[6] - np.array(grad))) < tol
    assert np.max(np.abs(reg.state_vec() - psi)) == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("n,nsets,extra", [(5, 3, 0), (5, 3, 1), (8, 1, 1), (8, 4, 1), (2, 1, 1)])
def test_sets_of_circuits_that_leave_the_sweep(n, nsets, extra):
    """Odd and even numbers of gradients in all (the complex numbers that lie
    behind them in memory need 16-byte boundaries): a controlled rotation is
    not the register sweep's."""
    rng = np.random.default_rng([n, nsets])
    els = [Y.put([q], Gate.Ry(0.3)) for q in range(n)] + [Y.control([0], [1], Gate.Rx(0.7)), Y.put([1], Gate.Rz(0.2))]
    els += [Y.put([0], Gate.Rx(0.1)) for _ in range(extra + n % 2)]
    c, h, psi = Y.Circuit.qubits(n, els), hamiltonian(n), random_state(rng, n)
    assert c.num_params() % 2 == (1 if extra else 0)
    sets = rng.uniform(-3, 3, size=(nsets, c.num_params()))
    vs, gs = Y.expect_grad_batch(h, c, sets, Y.ArrayReg.from_vec(n, psi))
    for s in range(nsets):
        c.dispatch(list(sets[s]))
        value, grad = O.expect_grad(h, c, psi)
        assert abs(vs[s] - value) < 1e-12 and np.max(np.abs(gs[s] - np.array(grad))) < 1e-12


@pytest.mark.gpu
def test_more_sets_than_a_group():
    """Groups of states that fit the cache, the last one smaller: every set as
    by itself."""
    n, nsets = 14, 131  # 128 sets of 2 x 256 KiB are one group
    rng = np.random.default_rng(0)
    c, h = ansatz(rng, n, 1, 0), hamiltonian(n)
    sets = rng.uniform(-3, 3, size=(nsets, c.num_params()))
    reg = Y.ArrayReg.zero_state(n)
    vs, gs = Y.expect_grad_batch(h, c, sets, reg)
    for s in (0, 127, 128, 130):
        c.dispatch(list(sets[s]))
        v, g = Y.expect_grad(h, c, reg)
        assert abs(v - vs[s]) < 1e-12 and np.max(np.abs(np.array(g) - gs[s])) < 1e-12


@pytest.mark.gpu
def test_long_runs_of_ops_split_passes():
    """More runs on one tile than a pass holds."""
    n = 6
    rng = np.random.default_rng(1)
    c, h, psi = ansatz(rng, n, 30, 0), hamiltonian(n), random_state(rng, n)
    value, grad = O.expect_grad(h, c, psi)
    v, g = Y.expect_grad(h, c, Y.ArrayReg.from_vec(n, psi))
    assert abs(v - value) < 1e-12 and np.max(np.abs(np.array(g) - np.array(grad))) < 1e-12


def projected(n, m):
    """A constant matrix that is not unitary at the end of a run, and before
    and after other runs' ends; parameters on both sides of it."""
    p = Gate.Custom(np.asarray(m, dtype=complex))
    els = [Y.put([q], Gate.Ry(0.3 + 0.1 * q)) for q in range(n)] + [Y.put([1], Gate.Rx(0.4)), Y.put([0], p)]
    els += [Y.control([0], [1], Gate.X), Y.put([1], Gate.Ry(0.5)), Y.put([1], p), Y.put([1], Gate.Rz(0.2))]
    els += [Y.control([1], [2], Gate.X), Y.put([2], p), Y.put([2], Gate.Ry(-0.7)), Y.control([2], [0], Gate.Z)]
    return Y.Circuit.qubits(n, els)


# zero rows and columns; a shear and a damping, which steps on other qubits must not pass
@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 12])
@pytest.mark.parametrize("m", [[[0, 0], [0, 1]], [[1, 0], [0, 0]], [[0, 1], [0, 0]], [[0, 0], [1, 0]], [[0, 0], [0, 0]],
                               [[1, 0.25], [0, 1]], [[1, 0], [0, 0.5j]]])
def test_constants_that_are_not_unitary(n, m):
    rng = np.random.default_rng(n)
    c, h, psi = projected(n, m), hamiltonian(n), random_state(rng, n)
    reg = Y.ArrayReg.from_vec(n, psi)
    value, grad = O.expect_grad(h, c, psi)
    v, g = Y.expect_grad(h, c, reg)
    vs, gs = Y.expect_grad_batch(h, c, np.array([c.parameters()] * 2), reg)
    # some tens of gates of 1.1e-16 each on terms of magnitude 1.7 n
    for got_v, got_g in ((v, g), (vs[0], gs[0]), (vs[1], gs[1])):
        assert abs(got_v - value) < 1e-12 and np.max(np.abs(np.array(got_g) - np.array(grad))) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("n", [21, 22])
def test_several_tiles_a_unit(n, monkeypatch):
    """More tiles than units of work: against one step a gate."""
    rng = np.random.default_rng(n)
    c, h = ansatz(rng, n, 1, 1), hamiltonian(n)
    reg = Y.ArrayReg.zero_state(n)
    v, g = Y.expect_grad(h, c, reg)
    vs, gs = Y.expect_grad_batch(h, c, np.array([c.parameters()] * 2), reg)
    monkeypatch.setenv("YAO_ADJ_TILES", "0")
    value, grad = Y.expect_grad(h, c, reg)
    for got_v, got_g in ((v, g), (vs[0], gs[0]), (vs[1], gs[1])):
        assert abs(got_v - value) < 1e-12 and np.max(np.abs(np.array(got_g) - np.array(grad))) < 1e-12


MEMORY = """
import numpy as np, torch
import yao_rs as Y
from helpers import tfim, vqe_ansatz
n, depth, nsets = 4, 100, 20000
c, h, reg = vqe_ansatz(n, depth, np.zeros(2 * n * depth)), tfim(n), Y.ArrayReg.zero_state(n)
sets = np.random.default_rng(0).uniform(-3, 3, size=(nsets, c.num_params()))
Y.expect_grad_batch(h, c, sets[:4], reg)
before = torch.cuda.mem_get_info(0)[0]
vs, gs = Y.expect_grad_batch(h, c, sets, reg)
print(before - torch.cuda.mem_get_info(0)[0])
for s in (0, 4095, 19999):
    c.dispatch(list(sets[s]))
    v, g = Y.expect_grad(h, c, reg)
    assert abs(v - vs[s]) < 1e-11 and np.max(np.abs(np.array(g) - gs[s])) < 1e-11
"""


@pytest.mark.gpu
def test_memory_of_many_sets_and_runs():
    """800 parameters in 400 runs, 20000 sets: parameters and gradients are
    128 MB each, and what the sweep needs stays below 64 + 256 MB (matrices
    and sums of all sets at once would be 1.3 GB)."""
    pytest.importorskip("torch")
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, PYTHONPATH=f"{root / 'yao-rs_b200'}:{root / 'tests'}")
    r = subprocess.run([sys.executable, "-c", MEMORY], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[0]) < 700e6


@pytest.mark.gpu
def test_two_large_sets_cost_what_two_calls_cost():
    """24 qubits: no part of a batch runs on one SM (the energy alone took
    eight times the gradient)."""
    n = 24
    c, h = ansatz(np.random.default_rng(0), n, 1, 0), hamiltonian(n)
    reg, sets = Y.ArrayReg.zero_state(n), np.array([c.parameters()] * 2)

    def best(f):
        times = []
        for _ in range(4):
            t = time.perf_counter()
            f()
            times.append(time.perf_counter() - t)
        return min(times)
    assert best(lambda: Y.expect_grad_batch(h, c, sets, reg)) < 4.0 * best(lambda: Y.expect_grad(h, c, reg))

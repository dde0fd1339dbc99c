"""FUSED runs of unitary circuits keep the norm: no error that grows with the
number of gates (rotations and CNOTs through csrc/reg_tiles.cu)."""
import numpy as np
import pytest

import yao_rs as Y
from helpers import layered_circuit, random_state


# 160 layers of 18 qubits: 1360 CNOTs, 2880 rotations.  Each rounding of
# 1.1e-16 is as often up as down, so the squared norm strays by about 2e-16
# times the root of the gates of one qubit (480), and of the coefficients'
# roundings, which all amplitudes share, by 2e-16 x sqrt(4240) = 1.3e-14: four
# times that.  A bias of an ulp a CNOT is 3e-13.
@pytest.mark.gpu
@pytest.mark.parametrize("k", [0, 1, 2])
def test_norm_of_a_deep_circuit(k):
    n, layers = 18, 160
    c = layered_circuit(n, layers, seed=5)
    r = Y.ArrayReg.from_vec(n, random_state(np.random.default_rng(1), n))
    before = float(np.sum(np.abs(r.state_vec().astype(np.clongdouble)) ** 2))
    Y.apply_inplace(c, r, Y.MODE_FUSED, k)
    after = float(np.sum(np.abs(r.state_vec().astype(np.clongdouble)) ** 2))
    assert abs(after - before) < 5.2e-14


@pytest.mark.gpu
def test_norm_of_a_batch():
    sizes, layers = (10, 12, 13, 14), 160
    circuits = [layered_circuit(n, layers, seed=n) for n in sizes]
    regs = [Y.ArrayReg.zero_state(n) for n in sizes]
    Y.batch_apply(circuits, regs, Y.MODE_FUSED)
    for r in regs:
        norm = float(np.sum(np.abs(r.state_vec().astype(np.clongdouble)) ** 2))
        assert abs(norm - 1.0) < 5.2e-14  # as above, on fewer qubits


# complex64 with the norm restored (256 gates and more): amplitudes move by
# one FP32 ulp (1.2e-7 at most) where the hash of their index says so, so what
# is left is a sum of 2^23 independent moves: 2.4e-7 / sqrt(2^23) = 8e-11 at
# most, five times that.  (Rounded to nearest, a factor within half an ulp of
# 1 moves no amplitude at all.)
@pytest.mark.gpu
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_norm_of_complex64(seed, batch):
    n = 22
    c = layered_circuit(n, 6, seed=seed)
    r = Y.ArrayReg.zero_state(n, Y.C64)
    if batch:
        Y.batch_apply([c, c], [r, Y.ArrayReg.zero_state(n, Y.C64)], Y.MODE_FUSED)
    else:
        Y.apply_inplace(c, r, Y.MODE_FUSED)
    norm = float(np.sum(np.abs(r.state_vec().astype(np.complex128)) ** 2))
    assert abs(norm - 1.0) < 4e-10

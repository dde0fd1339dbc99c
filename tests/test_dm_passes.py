"""Density-matrix circuits through the register passes (csrc/reg_tiles.cu)
against the oracle: PLAIN bit for bit, FUSED to rounding, at sizes around a
tile (11 of the 2n bits) and the thread's registers, for every channel kind
and for the steps that fall back to a pass of their own."""
import numpy as np
import pytest

import oracle as O
import yao_rs as Y
from helpers import random_state
from yao_rs import Gate, NoiseChannel as N, _abi as A

ONE = [N.AmplitudeDamping(0.1, 0.0), N.AmplitudeDamping(0.1, 0.3), N.PhaseDamping(0.2), N.BitFlip(0.1),
       N.PauliChannel(0.1, 0.05, 0.02), N.Reset(0.1, 0.05), N.PhaseAmplitudeDamping(0.1, 0.1, 0.2),
       N.ThermalRelaxation(100.0, 80.0, 5.0, 0.1), N.Depolarizing(1, 0.03)]


def noisy(rng, n, layers, kind):
    """0: rotations, one-qubit channels, CZ, CNOT and 2-qubit depolarizations;
    1: also SWAP, FSim and controlled gates; 2: also coherent errors, custom
    channels and 3-qubit gates, which register passes do not hold."""
    one = ONE + ([N.Coherent(Gate.Rx(0.3).matrix()), N.Custom([Gate.Ry(0.2).matrix()])] if kind == 2 else [])
    els = []
    for _ in range(layers):
        for q in range(n):
            els += [Y.put([q], Gate.Ry(rng.uniform(-3, 3))), Y.channel([q], N.Depolarizing(1, 0.03)),
                    Y.put([q], Gate.Rz(rng.uniform(-3, 3))), Y.channel([q], one[int(rng.integers(len(one)))])]
            if rng.random() < 0.3:
                els.append(Y.put([q], [Gate.H, Gate.X, Gate.T, Gate.Z, Gate.Y][int(rng.integers(5))]))
        for _ in range(n - 1):
            p, r = [int(x) for x in rng.permutation(n)], rng.random()
            if kind == 0 or r < 0.4:
                els.append(Y.control([p[0]], [p[1]], Gate.Z if r < 0.6 else Gate.X))
            elif r < 0.6:
                els.append(Y.put(p[:2], Gate.SWAP))
            elif r < 0.8:
                els.append(Y.put(p[:2], Gate.FSim(0.3, 0.4)))
            elif n > 2:
                els.append(Y.control(p[:2], [p[2]], Gate.Ry(0.7)))
            els.append(Y.channel(p[:2], N.Depolarizing(2, 0.05)))
            if kind == 2 and n > 2:
                els.append(Y.put(p[:3], Gate.Custom(np.linalg.qr(rng.normal(size=(8, 8)))[0].astype(complex))))
                els.append(Y.channel(p[:2], N.Coherent(np.kron(Gate.H.matrix(), Gate.T.matrix()))))
    return Y.Circuit.qubits(n, els)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 7])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_noisy_circuits(n, kind):
    rng = np.random.default_rng([n, kind])
    c, psi = noisy(rng, n, 3, kind), random_state(rng, n)
    ref = O.dm_apply_circuit(c, O.dm_from_reg(psi, n)).ravel()
    plain, fused = (Y.DensityMatrix.from_reg(Y.ArrayReg.from_vec(n, psi)) for _ in range(2))
    plain.apply(c)
    fused.apply(c, Y.MODE_FUSED)
    assert np.array_equal(plain.state_data(), ref)
    # up to 200 steps of 1e-16 each on entries of magnitude 1 at most
    assert np.abs(fused.state_data() - ref).max() < 1e-13


@pytest.mark.gpu
def test_sixteen_amplitudes_a_thread():
    """512 tiles: PLAIN in one run and step by step are the same bits."""
    rng = np.random.default_rng(3)
    n = 10
    c, psi = noisy(rng, n, 2, 1), random_state(rng, n)
    run, steps, fused = (Y.DensityMatrix.from_reg(Y.ArrayReg.from_vec(n, psi)) for _ in range(3))
    run.apply(c)
    for e in c.elements:
        steps.apply(Y.Circuit.qubits(n, [e]))
    fused.apply(c, Y.MODE_FUSED)
    assert np.array_equal(run.state_data(), steps.state_data())
    assert np.abs(fused.state_data() - run.state_data()).max() < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("ops", [[np.eye(2) * 0.25] * 17, [np.array([[0.5]])]])
def test_channels_that_are_refused(ops):
    """More than 16 Kraus operators, and none of the qubits: refused by PLAIN
    wherever they stand."""
    locs = [1] if ops[0].shape[0] == 2 else []
    c = Y.Circuit.qubits(4, [Y.put([0], Gate.H), Y.channel(locs, N.Custom(ops))] * 2)
    with pytest.raises(Y.YaoError) as e:
        Y.DensityMatrix.from_reg(Y.ArrayReg.zero_state(4)).apply(c)
    assert e.value.status == A.YAO_ERR_UNSUPPORTED


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 6])
def test_channels_that_all_differ(n):
    """As in a calibrated noise model: their coefficients fill several passes."""
    rng = np.random.default_rng(n)
    els = []
    for i in range(60):
        p = [int(x) for x in rng.permutation(n)]
        els += [Y.channel(p[:2] if i % 3 else [0, 1], N.Depolarizing(2, float(rng.uniform(0, 0.1)))),
                Y.channel([p[0]], N.PauliChannel(*rng.uniform(0, 0.1, 3))), Y.put([p[1]], Gate.Ry(rng.uniform(-3, 3)))]
    c, psi = Y.Circuit.qubits(n, els), random_state(rng, n)
    ref = O.dm_apply_circuit(c, O.dm_from_reg(psi, n)).ravel()
    plain, fused = (Y.DensityMatrix.from_reg(Y.ArrayReg.from_vec(n, psi)) for _ in range(2))
    plain.apply(c)
    fused.apply(c, Y.MODE_FUSED)
    assert np.array_equal(plain.state_data(), ref)
    # 180 steps of 1e-16 each on entries of magnitude 1 at most
    assert np.abs(fused.state_data() - ref).max() < 1e-13

"""Expectation values over tiles (csrc/sv_expect.cu): random strings against
the oracle at register counts around the tile edges."""
import numpy as np
import pytest

import oracle as O
import yao_rs as Y
from helpers import random_state

PAULI = [Y.Op.X, Y.Op.Y, Y.Op.Z]
ALL = PAULI + [Y.Op.I, Y.Op.P0, Y.Op.P1, Y.Op.Pu, Y.Op.Pd]


def strings(rng, n, choice, twice):
    """Strings of 0 .. min(n, 14) sites (X masks within a tile and wider),
    complex coefficients; twice: one site carries a second factor, which
    makes some strings anti-Hermitian."""
    cs, ss = [], []
    for _ in range(40):
        sites = [int(q) for q in rng.permutation(n)[:int(rng.integers(0, min(n, 14) + 1))]]
        ops = [(q, choice[int(rng.integers(len(choice)))]) for q in sites]
        if twice and sites:
            ops.append((sites[0], choice[int(rng.integers(len(choice)))]))
        ss.append(Y.OperatorString(ops))
        cs.append(complex(rng.normal(), rng.normal()))
    return Y.OperatorPolynomial(cs, ss)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 11, 12, 13, 14, 18])
def test_expectation_over_tiles(n):
    rng = np.random.default_rng(n)
    psi = random_state(rng, n)
    r = Y.ArrayReg.from_vec(n, psi)
    single = r.to_precision(Y.C64)
    for choice, twice in ((PAULI, False), (PAULI, True), (ALL, True)):
        op = strings(rng, n, choice, twice)
        # FP64 sums of at most 2^18 products below 1, tree-shaped: some 1e-14
        tol = 1e-13 * sum(abs(c) for c in op.coeffs())
        assert abs(Y.expect_arrayreg(r, op) - O.expect_arrayreg(psi, n, op)) < tol
        ref = O.expect_arrayreg(single.state_vec().astype(np.complex128), n, op)
        assert abs(Y.expect_arrayreg(single, op) - ref) < tol


@pytest.mark.gpu
def test_empty_operator():
    r = Y.ArrayReg.zero_state(5)
    assert Y.expect_arrayreg(r, Y.OperatorPolynomial.zero()) == 0


# 20 and 22 qubits: one to four tiles a CTA and more, so that buffers are
# loaded again and the barriers' phases turn; 23: the same for complex64
@pytest.mark.gpu
@pytest.mark.parametrize("tma", ["1", "0"])
@pytest.mark.parametrize("n", [20, 22, 23])
def test_several_tiles_a_cta(n, tma, monkeypatch):
    monkeypatch.setenv("YAO_TMA", tma)
    rng = np.random.default_rng(n)
    psi = random_state(rng, n)
    r = Y.ArrayReg.from_vec(n, psi)
    single = r.to_precision(Y.C64)
    op = strings(rng, n, PAULI, False)
    op = Y.OperatorPolynomial(op.coeffs()[:8], op.opstrings()[:8])
    # FP64 sums of at most 2^23 products whose magnitudes add up to 1 a string
    tol = 1e-13 * sum(abs(c) for c in op.coeffs())
    for reg in (r, single):
        v = reg.state_vec().astype(np.complex128)
        assert abs(Y.expect_arrayreg(reg, op) - O.expect_arrayreg(v, n, op)) < tol

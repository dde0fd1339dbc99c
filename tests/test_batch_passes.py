"""Batches of circuits through shared register passes (csrc/reg_tiles.cu)
against each circuit applied alone and the oracle, with few and many tiles
in all, every precision and mode, and batches that fall back to block passes."""
import numpy as np
import pytest

import oracle as O
import yao_rs as Y
from helpers import layered_circuit, qft_circuit, random_circuit, random_state


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(4, 4, 5), (8, 10, 11, 12), (3, 9), (17, 4, 18, 11, 18, 17), (21, 10)])
@pytest.mark.parametrize("wide", [False, True])
def test_batches(sizes, wide):
    rng = np.random.default_rng([len(sizes), sizes[0], wide])
    circuits = [layered_circuit(n, 3, seed=n) if i % 3 == 0 else qft_circuit(n) if i % 3 == 1 else
                random_circuit(rng, n, 40, max_ctrl=min(2, n - 1), custom=wide) for i, n in enumerate(sizes)]
    states = [random_state(rng, n) for n in sizes]
    refs = [O.apply_circuit(c, v) for c, v in zip(circuits, states)]
    # a few roundings (1.1e-16, 6e-8) a gate on states of norm 1
    for prec, eps in ((Y.C128, 5e-16), (Y.C64, 6e-8)):
        for mode, k in ((Y.MODE_TILED, 0), (Y.MODE_FUSED, 0), (Y.MODE_FUSED, 2), (Y.MODE_FUSED, 4)):
            regs = [Y.ArrayReg.from_vec(n, v).to_precision(prec) for n, v in zip(sizes, states)]
            Y.batch_apply(circuits, regs, mode, k)
            for c, r, ref in zip(circuits, regs, refs):
                if mode == Y.MODE_TILED and prec == Y.C128:
                    assert np.array_equal(r.state_vec(), ref)
                else:
                    assert np.linalg.norm(r.state_vec() - ref) < eps * len(c.elements), (mode, k)

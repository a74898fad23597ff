"""The pivot-block factor of the batched large-N kernels at the edges of its
eight-row blocks: the last 64-pivot block with 1, 4, 5, 8, 9, 60 and 63 real
rows, and the batched family at sizes below one block.

Tolerance: the bound of test_gpu_parity.py for the same seeded systems (5e-8
relative in Y), node counts exact."""
import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import propagate

pytestmark = pytest.mark.gpu
Y_TOL = 5e-8


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


def _check(prop, n, nstep):
    from oracle import oracle as O
    c, seg, ered, y0 = cases.random_case(n, nstep, seed=7700 + n)
    f = O.mdprop if prop == "LDMD" else O.ldprop
    yo, no, st, _ = f(cases.to_oracle(c), seg.rtab, seg.ptab, seg.nstep, seg.dr, ered, y0)
    assert st == 0
    yg, ng = propagate(prop, c, seg, ered, y0)
    assert ng == no
    assert cases.rel_err(yg, yo) < Y_TOL
    assert np.array_equal(yg, yg.T)


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
@pytest.mark.parametrize("n", [255, 257, 260, 261, 264, 265, 316, 449])
def test_last_block(prop, n):
    _check(prop, n, 8)


@pytest.mark.parametrize("n", [1, 4, 9, 63, 65])
def test_below_one_block(n):
    try:
        _lib.set_family_for_n(n, n, _lib.FAMILY_BIG, "LDMD")
        _check("LDMD", n, 40)
    finally:
        _lib.set_family_for_n(-1, -1, -1, "LDMD")

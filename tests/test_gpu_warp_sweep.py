"""The one-warp kernels (N <= 64) at the edges of their tiles: every remainder
of N against 8 and 4 near a tile boundary, the first sizes of each tile count,
and pivots whose reciprocal needs the exact scaling.

Tolerance: the bound of test_gpu_parity.py for the same seeded systems (5e-8
relative in Y: the order in which a pivot block's four rank-one terms are added
differs from the oracle's), node counts exact."""
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


def _check(prop, c, seg, ered, y0):
    from oracle import oracle as O
    f = O.mdprop if prop == "LDMD" else O.ldprop
    yo, no, st, _ = f(cases.to_oracle(c), seg.rtab, seg.ptab, seg.nstep, seg.dr, ered, y0)
    assert st == 0
    yg, ng = propagate(prop, c, seg, ered, y0)
    assert ng == no
    assert cases.rel_err(yg, yo) < Y_TOL
    assert np.array_equal(yg, yg.T)


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
@pytest.mark.parametrize("n", [6, 8, 9, 13, 16, 20, 21, 24, 25, 29, 32, 33, 37, 42, 44, 48, 49, 52, 53, 56, 57, 60, 61, 63])
def test_tile_edges(prop, n):
    _check(prop, *cases.random_case(n, 80, seed=7000 + n))


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
@pytest.mark.parametrize("n", [47, 58])
@pytest.mark.parametrize("kw", [dict(ivlfl=1, nconst=1), dict(nrsq=1, conlen=3.0, inward=True)], ids=["iv-const", "rsq-conf-inward"])
def test_hammat_variants_above_40(prop, n, kw):
    _check(prop, *cases.random_case(n, 60, seed=7100 + n, **kw))


@pytest.mark.parametrize("n", [3, 12, 36, 50])
def test_pivots_beyond_the_plain_reciprocal(n):
    """Hard walls in some channels: H Y0 ~ 1e304 there, so the first pivots lie
    above 2^1000 and take the scaled reciprocal; the rest of the block does not."""
    c, seg, ered, y0 = cases.random_case(n, 40, seed=7200 + n)
    for i in range(0, n, 5):
        y0[i, i] = 1.0e304 / (0.5 * seg.dr)
    _check("LDMD", c, seg, ered, y0)

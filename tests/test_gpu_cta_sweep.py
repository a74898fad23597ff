"""The one-CTA kernels (64 < N <= 200) at the edges of their tiles and of the
buckets, and the CTA shapes of launches with few and with many jobs.

Tolerance: the bound of test_gpu_parity.py for the same seeded systems (5e-8
relative in Y), node counts exact; the two CTA shapes bit for bit (the same
operations on the same tiles)."""
import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import Plan, propagate

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


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
@pytest.mark.parametrize("n", [65, 71, 73, 77, 81, 89, 96, 97, 105, 109, 113, 121, 125, 129, 145, 160, 161, 193])
def test_tile_edges(prop, n):
    from oracle import oracle as O
    c, seg, ered, y0 = cases.random_case(n, 20, seed=7300 + n)
    f = O.mdprop if prop == "LDMD" else O.ldprop
    yo, no, st, _ = f(cases.to_oracle(c), seg.rtab, seg.ptab, seg.nstep, seg.dr, ered, y0)
    assert st == 0
    yg, ng = propagate(prop, c, seg, ered, y0)
    assert ng == no
    assert cases.rel_err(yg, yo) < Y_TOL
    assert np.array_equal(yg, yg.T)


@pytest.mark.parametrize("prop", ["LDMD", "LDJ", "LDMG4"])
@pytest.mark.parametrize("n", [70, 126])
def test_few_and_many_jobs_agree(prop, n):
    kind = "LDMG4" if prop == "LDMG4" else "LD"
    c, seg, ered, y0 = cases.random_case(n, 6, seed=7400 + n, kind=kind)
    nj = 300
    e = ered + np.arange(nj) * 0.01
    plan = Plan(prop, [c], [seg], np.zeros(nj, dtype=np.int32), e)
    ybuf, nodes, status, _ = plan.run_host(plan.pack([y0] * nj))
    assert (status == 0).all()
    for j in (0, 147, 299):
        y1, n1 = propagate(prop, c, seg, e[j], y0)
        assert np.array_equal(plan.unpack(ybuf, j), y1) and nodes[j] == n1
    plan.close()

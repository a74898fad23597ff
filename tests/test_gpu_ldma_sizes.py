"""MAPROP's and AIRY's device sweeps at the edges of their tile counts (1, 8|9,
16|17, .., 100), against the oracle and against the sweep in numpy.

Tolerance: as in test_ldma.py and test_airy.py for random systems (5e-8 of
max|Y|; node counts exact)."""
import numpy as np
import pytest

import cases
from molscat_b200 import airy as AY
from molscat_b200 import ldma as LA
from test_airy import _sweep
from test_ldma import _Pot

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()


@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 17, 24, 25, 32, 40, 41, 48, 49, 65, 80, 81, 100])
def test_ldma_sizes(n):
    from oracle import oracle as O
    nstep = 30
    c, seg, ered, y0 = cases.random_case(n, nstep, seed=7500 + n)
    plan = LA.LDMAPlan(c, seg)
    erg = ered + np.array([0.0, 3.0])
    ys, nodes, status = plan.run_host([y0] * 2, erg)
    assert (status == 0).all()
    for j, e in enumerate(erg):
        yo, no = O.maprop(cases.to_oracle(c), _Pot(seg.pvec), float(seg.rtab[0]), seg.dr, nstep, float(e), y0)
        assert nodes[j] == no
        assert np.abs(ys[j] - yo).max() <= 5e-8 * np.abs(yo).max()
    plan.close()


@pytest.mark.parametrize("n", [1, 8, 17, 41, 100])
@pytest.mark.parametrize("outward", [True, False])
def test_airy_sizes(n, outward):
    rng = np.random.default_rng(7600 + n)
    ns = 6
    q = [np.linalg.qr(np.eye(n) + 0.1 * rng.normal(size=(n, n)))[0] for _ in range(ns + 1)]
    t = AY.AiryTables(n, 1.0, outward, np.full(ns, 0.05), [np.sort(rng.uniform(-20.0, 40.0, n)) for _ in range(ns)],
                      [rng.normal(size=n) for _ in range(ns)], np.stack(q[:ns]), q[ns])
    z0 = np.diag(rng.uniform(1.0, 5.0, n))
    plan = AY.AiryPlan(t)
    erg = [1.0, 2.5]
    zs, nodes, status = plan.run_host([z0] * 2, erg)
    assert (status == 0).all()
    for j, e in enumerate(erg):
        zo, no = _sweep(t, z0, e)
        assert nodes[j] == no
        assert np.abs(zs[j] - zo).max() <= 5e-8 * np.abs(zo).max()
    plan.close()

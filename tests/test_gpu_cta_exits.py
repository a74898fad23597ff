"""Every way out of the one-CTA kernels (64 < N <= 200) but the ordinary one:
cancelled, out of time, a non-finite or zero pivot in the preparation and in the
step loop, and pivots that take the scaled reciprocal; beside good jobs, whose
results must be those of the job alone, bit for bit.  The same for MAPROP's and
AIRY's sweeps, and the scaled reciprocal in the large-N factor.

Tolerance where an oracle is compared: the bound of test_gpu_parity.py for the
same seeded systems (5e-8 relative in Y), node counts exact."""
import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200 import airy as AY
from molscat_b200 import ldma as LA
from molscat_b200.propagators import Coupling, Plan, Segment, propagate

pytestmark = pytest.mark.gpu
Y_TOL = 5e-8
SIZES = [65, 70, 106, 128]  # a bucket each; 70 is launched in two shapes
PROPS = ["LDMD", "LDJ", "LDMG4"]


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


def _case(prop, n, nstep, seed):
    return cases.random_case(n, nstep, seed=seed, kind=prop if prop.startswith("LDMG") else "LD")


def _plan(prop, n, nstep, njobs, seed):
    c, seg, ered, y0 = _case(prop, n, nstep, seed)
    plan = Plan(prop, [c], [seg], np.zeros(njobs, dtype=np.int32), ered + np.linspace(0.0, 3.0, njobs))
    return plan, plan.pack([y0] * njobs)


@pytest.mark.parametrize("prop", PROPS)
@pytest.mark.parametrize("n, njobs", [(70, 3), (70, 300), (106, 3), (128, 3), (128, 150)])
def test_cancel_then_clear(prop, n, njobs):
    plan, y0 = _plan(prop, n, 20, njobs, 8200 + n)
    want, nodes, st, _ = plan.run_host(y0)
    assert (st == 0).all()
    plan.cancel(True)
    _, _, st, kf = plan.run_host(y0)
    assert (st == _lib.MGPU_ERR_CANCELLED).all() and (kf == 1).all()
    plan.cancel(False)
    y, n2, st, _ = plan.run_host(y0)
    assert (st == 0).all() and np.array_equal(n2, nodes) and np.array_equal(y, want)
    plan.close()


@pytest.mark.parametrize("prop", PROPS)
@pytest.mark.parametrize("n", [70, 106])
def test_time_limit_inside_the_run(prop, n):
    """128 steps take 5 ms or more (40 us a step at N = 70), 1200 ten times that."""
    plan, y0 = _plan(prop, n, 1200, 4, 8210 + n)
    plan.set_time_limit(2e-3)
    _, _, st, kf = plan.run_host(y0)
    assert (st == _lib.MGPU_ERR_DEADLINE).all()
    assert ((kf > 1) & ((kf - 1) % 128 == 0)).all(), kf
    plan.set_time_limit(0.0)
    _, _, st, _ = plan.run_host(y0)
    assert (st == 0).all()
    plan.close()


def _among_good_jobs(prop, bad, good, status, step):
    """good, bad, good, bad in one plan; the bad ones at their own energy."""
    sys = [bad, good]
    jsys = np.array([1, 0, 1, 0], dtype=np.int32)
    ered = np.array([sys[s][2] + 0.5 * k * s for k, s in enumerate(jsys)])
    plan = Plan(prop, [s[0] for s in sys], [s[1] for s in sys], jsys, ered)
    y, nodes, st, kf = plan.run_host(plan.pack([sys[s][3] for s in jsys]))
    assert list(st) == [0, status, 0, status]
    assert kf[1] == step and kf[3] == step and nodes[1] == 0 and nodes[3] == 0
    for j in (0, 2):
        ya, na = propagate(prop, good[0], good[1], ered[j], good[3])
        assert np.array_equal(plan.unpack(y, j), ya) and nodes[j] == na
    plan.close()


# (propagator, row of the radial table, step): the preparation's C of step 9,
# the step loop's B of step 8 (met in step 9), LDPROP's two, a stage of sector 5
@pytest.mark.parametrize("prop, row, step", [("LDMD", 17, 9), ("LDMD", 16, 9), ("LDJ", 17, 9), ("LDJ", 16, 9),
                                             ("LDMG4", 18, 5), ("LDMG5", 27, 5)])
@pytest.mark.parametrize("n", SIZES + [150, 200])
def test_nonfinite_potential(prop, row, step, n):
    if prop == "LDJ" and n > 128:
        pytest.skip("the large-N kernels")
    good = _case(prop, n, 12, 8220 + n)
    c, seg, ered, y0 = _case(prop, n, 12, 8230 + n)
    ptab = seg.ptab.copy()
    ptab[row, 1] = np.nan
    bad = (c, Segment(seg.nstep, seg.dr, seg.rtab, ptab, seg.kind), ered, y0)
    _among_good_jobs(prop, bad, good, _lib.MGPU_ERR_NONFINITE, step)


def _free_system(n, ivl=None, v=0.0, row=None, nstep=4):
    """No potential but a coupling v of the pair ivl at one radius; H = 0.5."""
    vl = np.zeros(n * (n + 1) // 2)
    ptab = np.zeros((2 * nstep + 1, 1))
    if ivl:
        lo, hi = ivl
        vl[hi * (hi + 1) // 2 + lo] = v
        ptab[row, 0] = 1.0
    c = Coupling(n=n, nham=1, vl=vl, eint=np.zeros(n), cent=np.zeros(n))
    return c, Segment(nstep, 1.0, 1.0 + 0.5 * np.arange(2 * nstep + 1.0), ptab)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("at", [0, 6, 61, 64])
def test_zero_pivot_in_the_step_loop(n, at):
    """LDPROP's first Z = H Y + I with Y_ii = -2 in one channel: both blocks of
    the first tile, a middle one, the last channels."""
    good = _case("LDJ", n, 12, 8240 + n)
    c, seg = _free_system(n)
    y0 = np.eye(n)
    y0[at, at] = -2.0
    _among_good_jobs("LDJ", (c, seg, 0.0, y0), good, _lib.MGPU_ERR_INVERSION, 1)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("pair", [(1, 2), (2, 6), (5, 63), (62, 64)])
def test_zero_pivot_in_the_preparation(n, pair):
    """MDPROP's U(C_3) with a coupling that makes two channels' rows equal:
    D4 V = 1/8, the diagonal."""
    h = 0.5
    d4 = -(h * h / 3.0) / 16.0
    v = 0.125 / d4
    for _ in range(4):
        if d4 * v == 0.125:
            break
        v = np.nextafter(v, -np.inf if d4 * v < 0.125 else np.inf)
    assert d4 * v == 0.125
    c, seg = _free_system(n, pair, v, row=5)
    good = _case("LDMD", n, 12, 8250 + n)
    _among_good_jobs("LDMD", (c, seg, 0.0, np.eye(n)), good, _lib.MGPU_ERR_INVERSION, 3)


@pytest.mark.parametrize("n", [65, 70, 106, 128, 150, 200, 260, 330])
def test_pivots_beyond_the_plain_reciprocal(n):
    """Hard walls in some channels: H Y0 ~ 1e304 there, so their pivots lie
    above 2^1000 and take the scaled reciprocal; the others do not."""
    from oracle import oracle as O
    c, seg, ered, y0 = cases.random_case(n, 12, seed=8260 + n)
    for i in range(0, n, 5):
        y0[i, i] = 1.0e304 / (0.5 * seg.dr)
    yo, no, st, _ = O.mdprop(cases.to_oracle(c), seg.rtab, seg.ptab, seg.nstep, seg.dr, ered, y0)
    assert st == 0
    yg, ng = propagate("LDMD", c, seg, ered, y0)
    assert ng == no
    assert cases.rel_err(yg, yo) < Y_TOL


@pytest.mark.parametrize("n", [6, 30, 64, 100])
def test_maprop_nonfinite_beside_good_energies(n):
    c, seg, ered, y0 = cases.random_case(n, 20, seed=8270 + n)
    plan = LA.LDMAPlan(c, seg)
    bad = y0.copy()
    bad[n - 1, n - 1] = np.nan
    e = ered + np.array([0.0, 1.0, 2.0])
    ya, na, sa = plan.run_host([y0] * 3, e)
    yb, nb, sb = plan.run_host([y0, bad, y0], e)
    plan.close()
    assert list(sa) == [0, 0, 0] and list(sb) == [0, _lib.MGPU_ERR_NONFINITE, 0]
    assert nb[1] == 0
    for j in (0, 2):
        assert np.array_equal(ya[j], yb[j]) and na[j] == nb[j]


@pytest.mark.parametrize("n", [6, 41, 100])
def test_airy_nonfinite_beside_good_energies(n):
    rng = np.random.default_rng(8280 + n)
    ns = 4
    q = [np.linalg.qr(np.eye(n) + 0.1 * rng.normal(size=(n, n)))[0] for _ in range(ns + 1)]
    t = AY.AiryTables(n, 1.0, True, np.full(ns, 0.05), [np.sort(rng.uniform(-20.0, 40.0, n)) for _ in range(ns)],
                      [rng.normal(size=n) for _ in range(ns)], np.stack(q[:ns]), q[ns])
    z0 = np.diag(rng.uniform(1.0, 5.0, n))
    bad = z0.copy()
    bad[0, 0] = np.inf
    plan = AY.AiryPlan(t)
    za, na, sa = plan.run_host([z0] * 3, [1.0, 1.5, 2.5])
    zb, nb, sb = plan.run_host([z0, bad, z0], [1.0, 1.5, 2.5])
    plan.close()
    assert list(sa) == [0, 0, 0] and list(sb) == [0, _lib.MGPU_ERR_NONFINITE, 0]
    for j in (0, 2):
        assert np.array_equal(za[j], zb[j]) and na[j] == nb[j]

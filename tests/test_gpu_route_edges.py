"""Sizes and uses at the edges of a route: MGPROP on the one-warp kernels by tile
edge, S matrices at the size where a job's matrices no longer fit shared memory,
and two host threads with one plan.

Tolerances: MGPROP as in test_ldmg.py (5e-8 of max|Y|, node counts exact), S as
in test_gpu_smatrix.py (1e-8)."""
import threading

import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import Plan

pytestmark = pytest.mark.gpu
S_TOL = 1e-8


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


class _Pot:
    def __init__(self, f):
        self.pvec = f


@pytest.mark.parametrize("kind", ["LDMG4", "LDMG5"])
@pytest.mark.parametrize("n", [4, 8, 9, 17, 28, 36, 41, 44, 45, 48, 49, 52, 56, 60, 61, 64, 65])
def test_mgprop_tile_edges(kind, n):
    from oracle import oracle as O
    nstep = 40
    c, seg, ered, y0 = cases.random_case(n, nstep, seed=8300 + n, kind=kind)
    plan = Plan(kind, [c], [seg], np.zeros(2, dtype=np.int32), ered + np.array([0.0, 3.0]))
    ybuf, nodes, status, _ = plan.run_host(plan.pack([y0, y0]))
    assert (status == 0).all()
    for j, e in enumerate(ered + np.array([0.0, 3.0])):
        yo, no = O.mgprop(cases.to_oracle(c), _Pot(seg.pvec), float(seg.rtab[0]), seg.dr, nstep, float(e), y0, int(kind[-1]))
        assert nodes[j] == no
        assert np.abs(plan.unpack(ybuf, j) - yo).max() <= 5e-8 * np.abs(yo).max()
    plan.close()


@pytest.mark.parametrize("n, ereds", [(65, (80.0,)), (95, (80.0,)), (96, (80.0,)), (97, (80.0,)), (98, (80.0,)),
                                      (99, (80.0,)), (110, (25.0, 80.0)), (124, (0.5, 80.0))])
def test_smatrices_where_shared_memory_ends(n, ereds):
    """All channels open: 3 N^2 doubles fit up to N = 95 or so; at N = 110 and
    124 the first energy's few open channels fit beside one that does not."""
    from oracle import oracle as O
    c, seg, _, y0 = cases.random_case(n, 20, seed=8400 + n)
    ereds = np.array([max(e, c.eint[0] + 0.1) for e in ereds])
    plan = Plan("LDMD", [c], [seg], np.zeros(len(ereds), dtype=np.int32), ereds)
    sr, si, _, status, _ = plan.run_host_smatrix(plan.pack([y0] * len(ereds)))
    ybuf, _, _, _ = plan.run_host(plan.pack([y0] * len(ereds)))
    assert (status == 0).all()
    oc = cases.to_oracle(c)
    for j, e in enumerate(ereds):
        wvec, nopen = O.gtwvec(e, oc.eint)
        want = O.ktos(O.ytok(O.chnsrt(oc.eint), wvec, n, nopen, plan.unpack(ybuf, j), seg.rtab[-1], oc.cent))
        assert np.abs(plan.unpack_s(sr, j) - want[0]).max() < S_TOL
        assert np.abs(plan.unpack_s(si, j) - want[1]).max() < S_TOL
    plan.close()


@pytest.mark.parametrize("prop", ["LDMD", "LDJ", "LDMG4"])
def test_two_threads_with_one_plan(prop):
    """Their own buffers and streams; MDPROP's preparation beforehand, which
    writes the plan's own tables."""
    import torch
    kind = prop if prop.startswith("LDMG") else "LD"
    items = [cases.random_case(n, 20, seed=8500 + n, kind=kind) for n in (5, 20, 47, 70)]
    jsys = np.repeat(np.arange(len(items), dtype=np.int32), 3)
    ered = np.array([items[s][2] + 4.0 * (k % 3) for k, s in enumerate(jsys)])
    plan = Plan(prop, [i[0] for i in items], [i[1] for i in items], jsys, ered)
    y = plan.pack([items[s][3] for s in jsys])
    want, nodes, status, _ = plan.run_host(y)
    assert (status == 0).all()
    got, errors = {}, []

    def work(t):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                y0 = torch.from_numpy(y).cuda()
                yd = torch.empty_like(y0)
                ints = torch.zeros(3, plan.njobs, dtype=torch.int32, device="cuda")
                res = []
                for _ in range(8):
                    yd.copy_(y0)
                    plan.run_device(yd.data_ptr(), ints[0].data_ptr(), ints[1].data_ptr(), ints[2].data_ptr(),
                                    st.cuda_stream, phases=2)
                    res.append((yd.clone(), ints[0].clone()))
                st.synchronize()
                got[t] = [(a.cpu().numpy(), b.cpu().numpy()) for a, b in res]
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    th = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=120)
    assert not errors and len(got) == 2
    for runs in got.values():
        for yk, nk in runs:
            assert np.array_equal(yk, want) and np.array_equal(nk, nodes)
    plan.close()

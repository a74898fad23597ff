"""Coupling-sum tables of N 41-64 where device memory is short: a plan or a
server that fits without them is not refused for them and its results are the
same bit for bit (the step kernel forms the same sums itself); a refusal for
want of memory does not reach the next call."""
import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import Plan, PropagatorError, propagate
from molscat_b200.serving import Server

pytestmark = pytest.mark.gpu
MB = 1 << 20
TILED = 36 * 64 * 8  # bytes of one tiled N = 64 matrix


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def _fill(keep):
    """All of the device's free memory but `keep` bytes."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(_free() - keep, dtype=torch.uint8, device="cuda")


def _release(filler):
    import torch
    filler.untyped_storage().resize_(0)
    torch.cuda.empty_cache()


def test_a_plan_without_room_for_the_tables():
    nstep = 10000
    q = TILED * nstep
    c, seg, ered, y0 = cases.random_case(64, nstep, seed=8100)
    e = ered + np.array([0.0, 2.0, 5.0])

    def plan():
        f0 = _free()
        p = Plan("LDMD", [c], [seg], np.zeros(3, dtype=np.int32), e)
        return p, f0 - _free()

    p, used = plan()
    assert used > 1.9 * q  # memory is plentiful: the tables are there
    want, nodes, status, _ = p.run_host(p.pack([y0] * 3))
    assert (status == 0).all()
    p.close()
    filler = _fill(q + q // 2)
    try:
        p, used = plan()
        assert used < 1.3 * q
        got, n2, s2, _ = p.run_host(p.pack([y0] * 3))
        p.close()
    finally:
        _release(filler)
    assert (s2 == 0).all() and np.array_equal(n2, nodes)
    assert np.array_equal(got, want)


def test_a_refused_plan_leaves_no_error_behind():
    c, seg, ered, y0 = cases.random_case(12, 20, seed=8101)
    big = cases.random_case(36, 10000, seed=8102)  # 77 MB of 2HQ(C)
    p = Plan("LDMD", [c], [seg], np.zeros(1, dtype=np.int32), np.array([ered]))
    want, nodes, _, _ = p.run_host(p.pack([y0]))
    filler = _fill(48 * MB)
    try:
        with pytest.raises(PropagatorError) as err:
            Plan("LDMD", [big[0]], [big[1]], np.zeros(1, dtype=np.int32), np.array([big[2]]))
        assert err.value.status == _lib.MGPU_ERR_NOMEM
        got, n2, s2, _ = p.run_host(p.pack([y0]))
    finally:
        _release(filler)
    assert s2[0] == 0 and np.array_equal(got, want) and np.array_equal(n2, nodes)
    p.close()


def test_a_server_gives_its_tables_back_for_the_next_system():
    a = cases.random_case(64, 4000, seed=8103)  # 74 MB of 2HQ(C), 76 MB of tables
    b = cases.random_case(64, 6000, seed=8104)  # 110 MB of 2HQ(C)
    ea = a[2] + np.linspace(0.0, 4.0, 24)
    ya, na = zip(*[propagate("LDMD", a[0], a[1], e, a[3]) for e in ea])
    yb, nb = propagate("LDMD", b[0], b[1], b[2], b[3])
    with Server("LDMD", hbm_budget=64 * MB, streams=2, max_batch=8) as srv:
        ia = srv.add_system(a[0], a[1])
        srv.submit(ia, ea[0], a[3]).wait()
        filler = _fill(60 * MB)
        try:
            reqs = [srv.submit(ia, e, a[3]) for e in ea]  # running when the next system arrives
            ib = srv.add_system(b[0], b[1])
            reqs += [srv.submit(ia, e, a[3]) for e in ea] + [srv.submit(ib, b[2], b[3])]
            got = [(r.wait(), r.nodes) for r in reqs]
        finally:
            _release(filler)
    for (y, n), yw, nw in zip(got, list(ya) * 2 + [yb], list(na) * 2 + [nb]):
        assert np.array_equal(y, yw) and n == nw

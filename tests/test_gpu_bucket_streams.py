"""A plan's buckets on streams of their own: ordered after the work queued on
the caller's stream and before what is queued there next, from several streams
in turn, and inside a captured graph (plans without large-N buckets).  Results are those of the same plan's
plain run, bit for bit (the same kernels on the same inputs)."""
import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import Plan

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


def _plan(prop):
    items = [cases.random_case(n, 20, seed=7800 + n) for n in (5, 12, 30, 47, 70, 120)]
    jsys = np.repeat(np.arange(len(items), dtype=np.int32), 3)
    ered = np.array([items[s][2] + 4.0 * (k % 3) for k, s in enumerate(jsys)])
    plan = Plan(prop, [i[0] for i in items], [i[1] for i in items], jsys, ered)
    return plan, plan.pack([items[s][3] for s in jsys])


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
def test_ordered_with_the_callers_stream(prop):
    import torch
    plan, y = _plan(prop)
    want, nodes, status, _ = plan.run_host(y)
    assert (status == 0).all()
    pinned = torch.from_numpy(y).pin_memory()
    ints = torch.zeros(3, plan.njobs, dtype=torch.int32, device="cuda")
    yd = torch.full((y.size,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    got = []
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k in range(4):
        s = streams[k % 2]
        if k:
            s.wait_stream(streams[(k - 1) % 2])
        with torch.cuda.stream(s):
            yd.fill_(float("nan"))
            torch.cuda._sleep(2_000_000)  # the input lands late, on this stream
            yd.copy_(pinned, non_blocking=True)
            plan.run_device(yd.data_ptr(), ints[0].data_ptr(), ints[1].data_ptr(), ints[2].data_ptr(), s.cuda_stream)
            got.append((yd.clone(), ints[0].clone()))
    torch.cuda.synchronize()
    for yk, nk in got:
        assert np.array_equal(yk.cpu().numpy(), want)
        assert np.array_equal(nk.cpu().numpy(), nodes)
    plan.close()


@pytest.mark.parametrize("prop", ["LDMD", "LDJ"])
def test_inside_a_captured_graph(prop):
    import torch
    plan, y = _plan(prop)
    want, nodes, status, _ = plan.run_host(y)
    assert (status == 0).all()
    y0 = torch.from_numpy(y).cuda()
    yd = torch.empty_like(y0)
    ints = torch.zeros(3, plan.njobs, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        yd.copy_(y0)
        plan.run_device(yd.data_ptr(), ints[0].data_ptr(), ints[1].data_ptr(), ints[2].data_ptr(),
                        torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        yd.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(yd.cpu().numpy(), want)
        assert np.array_equal(ints[0].cpu().numpy(), nodes)
    plan.close()

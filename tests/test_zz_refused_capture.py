"""A stream that is capturing a graph is refused by a plan with a large-N bucket
(its own steps replay a graph); the refusal ends with the capture, and the plan
runs afterwards as before."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import numpy as np
import torch
from cuda.bindings import runtime as rt
sys_path = __import__("sys").path
sys_path[:0] = [".", "tests"]
import cases
from molscat_b200.propagators import Plan, PropagatorError

items = [cases.random_case(n, 10, seed=8700 + n) for n in (5, 30, 70, 260)]
jsys = np.repeat(np.arange(4, dtype=np.int32), 2)
ered = np.array([items[s][2] + 2.0 * (k % 2) for k, s in enumerate(jsys)])
for prop in ("LDMD", "LDJ"):
    plan = Plan(prop, [i[0] for i in items], [i[1] for i in items], jsys, ered)
    y = plan.pack([items[s][3] for s in jsys])
    yd = torch.from_numpy(y).cuda()
    ints = torch.zeros(3, plan.njobs, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for warm in (False, True):  # the step graph not captured yet, and captured
        if warm:
            want, nodes, st, _ = plan.run_host(y)
            assert (st == 0).all()
        err, s = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
        assert int(err) == 0
        err, = rt.cudaStreamBeginCapture(s, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
        assert int(err) == 0
        refused = False
        try:
            plan.run_device(yd.data_ptr(), ints[0].data_ptr(), ints[1].data_ptr(), ints[2].data_ptr(), int(s))
        except PropagatorError:
            refused = True
        err, graph = rt.cudaStreamEndCapture(s)
        assert refused, prop
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(s)
        got, n2, st, _ = plan.run_host(y)
        assert (st == 0).all()
        if warm:
            assert np.array_equal(got, want) and np.array_equal(n2, nodes)
    plan.close()
print("refused and usable")
"""


def test_refused_and_usable_afterwards():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    pytest.importorskip("cuda.bindings")
    from molscat_b200.build import build
    build()
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "refused and usable" in r.stdout, r.stdout + r.stderr

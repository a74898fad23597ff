"""The server's last free slot: kept a moment for another size, not longer."""
import time

import numpy as np
import pytest

import cases
from molscat_b200 import _lib
from molscat_b200.propagators import propagate
from molscat_b200.serving import Server

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from molscat_b200.build import build
    build()
    _lib.load()


def test_the_last_slot_is_left_to_another_size():
    """One large propagation runs; a second of its size and a small one arrive
    together: the small one starts at once, the second large one beside the
    first after it."""
    big = cases.random_case(512, 400, seed=8600)  # 100 ms or more
    small = cases.random_case(20, 60, seed=8601)
    with Server("LDMD", streams=2, max_batch=8) as srv:
        b = srv.add_system(big[0], big[1])
        s = srv.add_system(small[0], small[1])
        for sid, c in ((b, big), (s, small)):  # everything loaded
            srv.submit(sid, c[2], c[3]).wait()
        first = srv.submit(b, big[2], big[3])
        t0 = time.time()
        while first.times()[1] == 0.0 and time.time() - t0 < 30:
            time.sleep(0.0002)
        second = srv.submit(b, big[2] + 1.0, big[3])
        other = srv.submit(s, small[2], small[3])
        got = [(r.wait(), r.nodes) for r in (first, second, other)]
        done = first.times()[2]
        assert first.times()[1] > 0.0
        assert other.times()[1] < done and other.times()[2] < done
        assert other.times()[1] < second.times()[1] < done
    for (y, n), (c, e) in zip(got, ((big, big[2]), (big, big[2] + 1.0), (small, small[2]))):
        ya, na = propagate("LDMD", c[0], c[1], e, c[3])
        assert np.array_equal(y, ya) and n == na


def test_one_slot_serves_one_size():
    c, seg, ered, y0 = cases.random_case(16, 60, seed=8602)
    with Server("LDMD", streams=1, max_batch=4) as srv:
        sid = srv.add_system(c, seg)
        reqs = [srv.submit(sid, ered + 0.1 * k, y0) for k in range(12)]
        for k, r in enumerate(reqs):
            ya, na = propagate("LDMD", c, seg, ered + 0.1 * k, y0)
            assert np.array_equal(r.wait(), ya) and r.nodes == na

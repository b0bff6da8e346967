"""Batches whose cases' lists (coarse/fine pairs, domain ghosts, immersed
cells) are uploaded again between the batch's creation, its first run and a
later one: every run equals the cases stepped alone, bit for bit."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
import make_golden  # noqa: E402
from conftest import load_pkg  # noqa: E402
from test_host_lists import upload  # noqa: E402

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads


@pytest.mark.parametrize("precision", [ib.FP64, ib.MIXED])
def test_runs_follow_new_lists(cuda_lib, precision):
    g = make_golden.load("naca_minmod_s4_n64_l3")
    L = wl.naca_lists(g, 0)
    nbc, nib = len(L["bc"]), len(L["ib"])
    single = [wl.naca_solver(g, k, precision) for k in (0, 0)]
    batched = [wl.naca_solver(g, k, precision) for k in (0, 0)]
    b = ib.Batch(batched)
    for step, (pressure, n, m) in enumerate([(0.05, nbc, nib - 7), (0.02, nbc, nib), (0.0, nbc, nib - 1)]):
        for s in (single[1], batched[1]):
            upload(s, L, backpressure=pressure, bc=n, ib=m)
        for s in single:
            s.run(4 * step, 4)
        b.run(4 * step, 4)
        for s, t in zip(single, batched):
            assert t.dt == s.dt and np.array_equal(t.download(), s.download())
    assert not np.array_equal(single[0].download(), single[1].download())
    b.close()
    for s in single + batched:
        s.close()

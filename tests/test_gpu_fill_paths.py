"""The fills' less travelled launches against the usual ones, bit for bit:
bodies of more immersed cells than one CTA takes (two launches, in a batch a
pair per case), batches whose cases' levels write what other levels read, and
batches with kernel timing on (each case's own launches)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
import make_golden  # noqa: E402
from conftest import load_pkg  # noqa: E402
from test_host_lists import chained_mesh, upload  # noqa: E402

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads


def record():
    return make_golden.load("naca_minmod_s4_n64_l3")


def equal(single, batched):
    for s, t in zip(single, batched):
        assert t.dt == s.dt and np.array_equal(t.download(), s.download())


def close(*sols):
    for s in sols:
        s.close()


# the record's cells again and again: every repetition computes the same state
# from the same field, so the flow is that of the short list
@pytest.mark.parametrize("n", [1024, 1025, 2500])
@pytest.mark.parametrize("precision", [ib.FP64, ib.FP64_EXACT])
def test_many_immersed_cells_equal_the_short_list(cuda_lib, precision, n):
    g = record()
    L = wl.naca_lists(g, 0)
    assert len(L["ib"]) < 1024
    short, many = (wl.naca_solver(g, 0, precision) for _ in range(2))
    upload(many, dict(L, ib=np.resize(L["ib"], (n, 18)), ib_f=np.resize(L["ib_f"], (n, 16))), ("ib",))
    for s in (short, many):
        s.run(0, 4)
    equal([short], [many])
    if precision == ib.FP64:
        single = [short, wl.naca_solver(g, 2, precision)]
        batched = [many, wl.naca_solver(g, 2, precision)]
        b = ib.Batch(batched)
        for s in single:
            s.run(4, 4)
        b.run(4, 4)
        equal(single, batched)
        b.close()
        close(*single[1:], *batched[1:])
    close(short, many)


@pytest.mark.parametrize("chained", [(True, False), (True, True), (False, False)])
def test_batched_chained_levels_equal_single_runs(cuda_lib, chained):
    r = np.random.default_rng(11)

    def solver(c, prim):
        P, (lv, x, y), res, pro = chained_mesh(c)
        s = ib.FlowSolver(dict(P, precision=ib.FP64))
        s.upload_topology(lv, x, y, np.full(len(lv), ib.CELL_PRESENT, np.uint8))
        s.upload_interfaces(np.array(res), np.array(pro))
        s.init_flow(prim)
        return s

    single, batched = [], []
    for c in chained:
        P, (lv, _, _), _, _ = chained_mesh(c)
        prim = np.empty((len(lv), 7))
        prim[:, 0], prim[:, 4] = r.uniform(0.5, 1.5, len(lv)), r.uniform(2.0, 3.0, len(lv))
        prim[:, 1], prim[:, 2], prim[:, 3] = r.uniform(-1, 1, len(lv)), r.uniform(-1, 1, len(lv)), 0.0
        prim[:, 5] = prim[:, 4] / (prim[:, 0] * P["Rg"])
        prim[:, 6] = P["Cv"] * prim[:, 5] + 0.5 * (prim[:, 1] ** 2 + prim[:, 2] ** 2)
        single.append(solver(c, prim))
        batched.append(solver(c, prim))
    for s in single:
        s.run(0, 3)
    b = ib.Batch(batched)
    b.run(0, 3)
    equal(single, batched)
    b.close()
    close(*single, *batched)


def test_batch_with_kernel_timing_equals_single_runs(cuda_lib):
    g = record()
    single, batched = ([wl.naca_solver(g, k, ib.FP64) for k in (0, 2)] for _ in range(2))
    b = ib.Batch(batched)
    for k, timed in enumerate((True, False, True)):
        batched[1].set_kernel_timing(timed)  # the per-case launches, the graphs, and back
        for s in single:
            s.run(4 * k, 4)
        b.run(4 * k, 4)
        equal(single, batched)
    b.close()
    close(*single, *batched)

"""Schemes of one stage (the stage is first and final) on grids of many tiles:
its neighbours' input must not change under it, so every step equals the
oracle's bit for bit in the exact build, batches and the allocation-free step
equal single runs, and a batch's tuning leaves the state alone."""
import numpy as np
import pytest

from conftest import load_pkg
from test_gpu_vortex import oracle_levels_for

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads
# per step, as the other parity tests bound them
REL = {ib.FP64: 1e-12, ib.MIXED: 2e-5}
STEPS = 5


def case(n, precision, **kw):
    P, cells, prim = wl.vortex_case(n, nstages=3, precision=precision, cfl=0.2, **kw)
    return dict(P, nstages=1, tp=[1.0]), cells, prim


def solver(c):
    P, cells, prim = c
    s = ib.FlowSolver(P)
    s.upload_topology(**cells)
    s.init_flow(prim)
    return s


def conserved(q):
    return np.stack([q[:, 0], q[:, 0] * q[:, 1], q[:, 0] * q[:, 2], q[:, 0] * q[:, 6]], 1)


@pytest.mark.parametrize("n", [32, 208])
def test_one_stage_steps_match_the_oracle(cuda_lib, oracle, n):
    c = case(n, ib.FP64_EXACT)
    P, cells, prim = c
    d, lv = oracle_levels_for(oracle, cells["ix"], cells["iy"], prim, n, P)
    dt = 1.0
    for ts in range(STEPS):
        rc, dt, _, _ = oracle.step(P, lv, ts, dt)
        assert rc == 0
    ref = lv.state_like_dump(d)[: n * n]
    s = solver(c)
    s.run(0, STEPS)
    assert s.dt == dt and np.array_equal(s.download(), ref)
    s.close()
    for precision, tol in REL.items():
        s = solver(case(n, precision))
        s.run(0, STEPS)
        a, b = conserved(s.download()), conserved(ref)
        assert (np.abs(a - b).max(0) / np.abs(b).max(0)).max() <= STEPS * tol
        assert abs(s.dt - dt) <= STEPS * tol * dt
        s.close()


@pytest.mark.parametrize("precision", [ib.FP64, ib.MIXED])
def test_batched_one_stage_cases_equal_single_runs(cuda_lib, precision):
    cases = [case(n, precision, mach=m) for n, m in [(208, 0.5), (48, 0.3), (160, 0.8)]]
    single, batched = [solver(c) for c in cases], [solver(c) for c in cases]
    for s in single:
        s.run(0, STEPS)
    b = ib.Batch(batched)
    b.run(0, 2)  # tunes first
    assert len(b.info()["tuning"]) > 1
    b.run(2, STEPS - 2)
    for s, t in zip(single, batched):
        assert t.dt == s.dt and np.array_equal(t.download(), s.download())
    b.close()
    for s in single + batched:
        s.close()


@pytest.mark.parametrize("precision", [ib.FP64, ib.MIXED, ib.FP64_EXACT])
def test_allocation_free_one_stage_step_equals_the_regular_one(cuda_lib, precision):
    import torch
    n = 256
    c = case(n, precision)
    rows = torch.from_numpy(c[2]).to("cuda")
    torch.cuda.synchronize()
    s = solver(c)
    dt = 1.0
    for ts in range(STEPS):
        dt, _ = ib.step_periodic_noalloc(c[0], ts, n, n, rows.data_ptr(), rows.data_ptr(), dt)
        s.time_marching(ts)
        assert dt == s.dt
    assert np.array_equal(rows.cpu().numpy(), s.download())
    s.close()

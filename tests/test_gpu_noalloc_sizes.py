"""Allocation-free step over changing grids: its tables and diagnostics live in
one array that keeps the previous call's contents, so grids of one to 256
tiles alternate, with and without a CFL pass, and with a CFL abort in
between; states and dt against the regular entry point bit for bit."""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads


def case(nx, ny, precision, every, seed):
    r = np.random.default_rng(seed)
    g = wl.gas_constants(0.5, 0.0)
    init = wl.freestream(g, 0.7)
    iy, ix = (a.ravel().astype(np.int32) for a in np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij"))
    prim = wl.vortex_state(ix, iy, 10.0 / nx, g, init, 4.0, 5.0 + r.uniform(-1, 1), 5.0 * ny / nx)
    h = 10.0 / nx
    P = dict(g, cfl=0.5, dt_ratio=1.0, dt_var_step=every, nstages=3, tp=wl.TP[3],
             limiter=ib.LIM_VANLEER, viscous=0, precision=precision, initvar=init, nlevels=1,
             dh=[(h, h, 0.1)], march_step=[1], march_left=[0], step_num=[1.0], domain_nx=nx,
             domain_ny=ny, periodic_x=1, periodic_y=1, dt0=1.0)
    flags = np.full(ix.shape, 1 | 2 | 4 | 8 | 32, np.uint8)
    return P, ix, iy, flags, prim


@pytest.mark.parametrize("precision", [ib.FP64, ib.MIXED, ib.FP64_EXACT])
def test_grids_alternate(cuda_lib, precision):
    import torch
    sizes = [(256, 256), (16, 16), (48, 16), (16, 112), (256, 256), (32, 80)]
    for k, (nx, ny) in enumerate(sizes):
        every, ts, dt0 = (1, 0, 1.0) if k % 2 == 0 else (4, 3, 1e-3)  # 4, 3: no CFL pass
        P, ix, iy, flags, prim = case(nx, ny, precision, every, k)
        rows = torch.from_numpy(prim).to("cuda")
        out = torch.empty_like(rows)
        torch.cuda.synchronize()
        if k == 2:
            bad = dict(P, cfl=-0.5)  # a negative time step: abort 424, and the next call is clean
            with pytest.raises(ib.IbgpuError) as e:
                ib.step_periodic_noalloc(bad, 0, nx, ny, rows.data_ptr(), out.data_ptr(), 1.0)
            assert e.value.abort_code == 424
        dt, d = ib.step_periodic_noalloc(P, ts, nx, ny, rows.data_ptr(), out.data_ptr(), dt0)
        s = ib.FlowSolver(P)
        s.upload_topology(np.zeros_like(ix), ix, iy, flags)
        s.init_flow(prim)
        s.dt = dt0
        d2 = s.time_marching(ts)
        assert dt == s.dt and d.cfl_dt == d2.cfl_dt and list(d.res_max) == list(d2.res_max)
        assert np.array_equal(out.cpu().numpy(), s.download())
        s.close()

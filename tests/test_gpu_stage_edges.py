"""Stage kernel of the fast builds at its edges: regions whose outer stencil
cells are missing (one ghost layer only: the reference's one-sided
reconstructions, NS_Solver.H:743-750), ragged regions against the 16 x 16
tiles, single-column and single-row patches, and a periodic grid of one tile
that is its own neighbour.  Held against the exact build (operation for
operation the reference) with the per-step bounds of the other parity tests.
"""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads
REL = {ib.FP64: 1e-12, ib.MIXED: 2e-5}


def patch(nx, ny, x0, y0, layers, seed):
    """Cells of an nx x ny patch at (x0, y0) with `layers` ghost layers on
    each side (no corners) and a smooth random flow."""
    y, x = np.meshgrid(np.arange(-layers, ny + layers), np.arange(-layers, nx + layers),
                       indexing="ij")
    x, y = x.ravel(), y.ravel()
    inx, iny = (x >= 0) & (x < nx), (y >= 0) & (y < ny)
    keep = inx | iny
    x, y, normal = x[keep], y[keep], (inx & iny)[keep]
    flags = np.where(normal, ib.CELL_PRESENT | ib.CELL_NORMAL | ib.CELL_UPDATE | ib.CELL_PRIM |
                     ib.CELL_RESNORM, ib.CELL_PRESENT).astype(np.uint8)
    r = np.random.default_rng(seed)

    def wave(mean, amp):
        k = r.uniform(0.2, 1.1, (3, 2))
        p = r.uniform(0, 6.28, 3)
        return mean + amp * sum(np.sin(k[i, 0] * x + k[i, 1] * y + p[i]) for i in range(3)) / 3

    g = wl.gas_constants(0.5, 0.0)
    init = wl.freestream(g, 0.3)
    rho, u, v, p = wave(1.0, 0.2), wave(0.6, 0.5), wave(-0.2, 0.5), wave(init[4], 0.4)
    T = p / (rho * g["Rg"])
    prim = np.stack([rho, u, v, 0 * u, p, T, g["Cv"] * T + 0.5 * (u * u + v * v)], 1)
    return g, init, x + x0, y + y0, flags, prim


def one_step(g, init, x, y, flags, prim, precision, limiter, stages, periodic, n):
    P = dict(g, cfl=0.4, dt_ratio=1.0, dt_var_step=1, nstages=stages, tp=wl.TP[stages],
             limiter=limiter, viscous=0, precision=precision, initvar=init, nlevels=1,
             dh=[(0.1, 0.1, 0.1)], march_step=[1], march_left=[0], step_num=[1.0],
             domain_nx=n, domain_ny=n, periodic_x=periodic, periodic_y=periodic, dt0=1.0)
    s = ib.FlowSolver(P)
    s.upload_topology(np.zeros_like(x), x, y, flags)
    s.init_flow(prim)
    d = s.run(0, 2)
    out, dt, res = s.download(), s.dt, np.array(list(d.res_max))
    s.close()
    return out, dt, res


def conserved(q):
    return np.stack([q[:, 0], q[:, 0] * q[:, 1], q[:, 0] * q[:, 2], q[:, 0] * q[:, 6]], 1)


@pytest.mark.parametrize("limiter", [ib.LIM_VANLEER, ib.LIM_MINMOD])
@pytest.mark.parametrize("nx,ny,x0,y0,layers", [(1, 1, 20, 20, 1), (1, 40, 15, 9, 1),
                                                (37, 2, 30, 31, 1), (16, 16, 32, 16, 1),
                                                (47, 33, 17, 30, 1), (31, 18, 16, 15, 2)])
def test_patches_match_the_exact_build(cuda_lib, limiter, nx, ny, x0, y0, layers):
    args = patch(nx, ny, x0, y0, layers, 7 * nx + ny)
    normal = (args[4] & ib.CELL_NORMAL) != 0
    ref, dt, res = one_step(*args, ib.FP64_EXACT, limiter, 4, 0, 256)
    assert np.all(np.isfinite(ref)) and np.any(ref[normal] != args[5][normal])
    for precision, tol in REL.items():
        got, dt2, res2 = one_step(*args, precision, limiter, 4, 0, 256)
        a, b = conserved(got)[normal], conserved(ref)[normal]
        # two steps of the per-step bound
        assert (np.abs(a - b).max(0) / np.abs(b).max(0)).max() <= 2 * tol
        assert np.array_equal(got[~normal], ref[~normal])
        assert abs(dt2 - dt) <= 2 * tol * dt
        assert np.all(np.abs(res2 - res) <= 2 * tol / 1e-12 * 1e-9 * np.maximum(res.max(), 1e-12))


@pytest.mark.parametrize("n", [16, 32])
def test_smallest_periodic_grids_match_the_exact_build(cuda_lib, n):
    p, c, prim = wl.vortex_case(n, precision=ib.FP64_EXACT)
    args = (wl.gas_constants(0.5, 0.0), p["initvar"], c["ix"], c["iy"], c["flags"], prim)
    ref, dt, _ = one_step(*args, ib.FP64_EXACT, ib.LIM_VANLEER, 3, 1, n)
    for precision, tol in REL.items():
        got, dt2, _ = one_step(*args, precision, ib.LIM_VANLEER, 3, 1, n)
        assert (np.abs(conserved(got) - conserved(ref)).max(0) / np.abs(conserved(ref)).max(0)).max() <= 2 * tol
        assert abs(dt2 - dt) <= 2 * tol * dt

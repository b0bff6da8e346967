"""Viscous pass of the fast builds at its edges: patches ragged against the
16 x 16 tiles (partly filled tiles, corners in a diagonal neighbour tile,
absent neighbour tiles), all moving and one cell wide, held against the exact
build (operation for operation the reference) after two viscous steps with
the per-step bounds of the other parity tests."""
import numpy as np
import pytest

from conftest import load_pkg
from test_gpu_stage_edges import REL, conserved, patch

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads


@pytest.mark.parametrize("nx,ny,x0,y0", [(1, 1, 31, 32), (2, 35, 15, 15), (16, 16, 16, 32),
                                         (33, 17, 31, 15), (48, 31, 9, 30)])
def test_viscous_patches_match_the_exact_build(cuda_lib, nx, ny, x0, y0):
    # ghosts with corners: the tangential differences read them
    g, init, x, y, flags, prim = patch(nx, ny, x0, y0, 2, 3 * nx + ny)
    cx, cy = np.meshgrid([x0 - 2, x0 - 1, x0 + nx, x0 + nx + 1],
                         [y0 - 2, y0 - 1, y0 + ny, y0 + ny + 1])
    x, y = np.append(x, cx.ravel()), np.append(y, cy.ravel())
    flags = np.append(flags, np.full(16, ib.CELL_PRESENT, np.uint8))
    prim = np.vstack([prim, prim[np.arange(16) % len(prim)]])
    v = wl.gas_constants(0.5, 1e-2)
    out = {}
    for precision in (ib.FP64_EXACT, *REL):
        P = dict(v, cfl=0.3, dt_ratio=1.0, dt_var_step=1, nstages=3, tp=wl.TP[3],
                 limiter=ib.LIM_MINMOD, viscous=1, precision=precision, initvar=init, nlevels=1,
                 dh=[(0.1, 0.07, 0.1)], march_step=[1], march_left=[0], step_num=[1.0],
                 domain_nx=256, domain_ny=256, dt0=1.0)
        s = ib.FlowSolver(P)
        s.upload_topology(np.zeros_like(x), x, y, flags)
        s.init_flow(prim)
        s.run(0, 2)
        out[precision] = s.download()
        s.close()
    normal = (flags & ib.CELL_NORMAL) != 0
    ref = out[ib.FP64_EXACT]
    assert np.all(np.isfinite(ref)) and np.any(ref[normal] != prim[normal])
    for precision, tol in REL.items():
        a, b = conserved(out[precision])[normal], conserved(ref)[normal]
        assert (np.abs(a - b).max(0) / np.abs(b).max(0)).max() <= 2 * tol
        assert np.array_equal(out[precision][~normal], ref[~normal])

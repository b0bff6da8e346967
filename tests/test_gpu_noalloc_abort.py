"""Diagnostics of an allocation-free step that aborts on a negative time step
(424), on grids of one tile to the largest (256 tiles, one per thread of the
CTA that reduces them): those of the regular entry point."""
import numpy as np
import pytest

from conftest import load_pkg
from test_gpu_noalloc_sizes import case

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib = pkg.ibgpu


@pytest.mark.parametrize("nx,ny", [(16, 16), (48, 32), (256, 240), (256, 256)])
def test_negative_time_step_reports_as_the_regular_step(cuda_lib, nx, ny):
    import torch
    P, ix, iy, flags, prim = case(nx, ny, ib.FP64, 1, 3)
    P["cfl"] = -0.5
    rows = torch.from_numpy(prim).to("cuda")
    torch.cuda.synchronize()
    with pytest.raises(ib.IbgpuError) as e:
        ib.step_periodic_noalloc(P, 0, nx, ny, rows.data_ptr(), rows.data_ptr(), 1.0)
    s = ib.FlowSolver(P)
    s.upload_topology(np.zeros_like(ix), ix, iy, flags)
    s.init_flow(prim)
    with pytest.raises(ib.IbgpuError) as r:
        s.time_marching(0)
    s.close()
    got, ref = e.value.diag, r.value.diag
    assert got.abort_code == ref.abort_code == 424
    assert got.cfl_dt == ref.cfl_dt == 10000.0
    assert got.dt == ref.dt

"""Indicator kernels at the edges of their 128-row tiles, with more tiles than
resident CTAs, and with parameter arrays that are not 16-byte aligned (weights
loaded one by one), against the CPU oracle with the tolerances of the other
indicator tests."""
import os
import sys

import numpy as np
import pytest

from conftest import ORACLE_DIR, load_pkg

sys.path.insert(0, ORACLE_DIR)
import indicator_oracle as io  # noqa: E402
from test_gpu_indicator import GRAD_REL_TOL, LOGIT_TOL, random_problem  # noqa: E402

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads


@pytest.fixture(scope="module")
def solver(cuda_lib):
    p, c, prim = wl.vortex_case(16)
    s = ib.FlowSolver(p)
    s.upload_topology(**c)
    yield s
    s.close()


def shifted(a, off):
    """a on the device, off elements past an aligned address."""
    import torch
    t = torch.zeros(a.size + off, dtype=torch.from_numpy(a).dtype, device="cuda")
    t[off:] = torch.from_numpy(a).to("cuda").reshape(-1)
    return t, t.data_ptr() + off * a.itemsize


@pytest.mark.parametrize("n,off", [(1, 1), (127, 0), (129, 3), (256, 0)])
def test_forward_tiles(solver, n, off):
    import torch
    P, X, _ = random_problem(n, 17 + n)
    keep, pptr = shifted(P, off)
    feat = torch.from_numpy(X.view(np.int16)).to("cuda")
    cls = torch.full((n + 1,), 9, dtype=torch.uint8, device="cuda")
    logits = torch.full((n + 1, 3), -7.0, device="cuda")
    solver.mlp_forward(pptr, n, feat.data_ptr(), cls.data_ptr(), logits.data_ptr())
    ref, _ = io.mlp_forward(P, X_bits=X)
    got = logits.cpu().numpy()
    assert np.abs(got[:n] - ref).max() <= LOGIT_TOL * max(1.0, np.abs(ref).max())
    assert np.array_equal(cls.cpu().numpy()[:n], np.argmax(got[:n], axis=1))
    assert cls[n] == 9 and torch.all(logits[n] == -7.0)  # nothing past the rows
    del keep


def test_forward_rows_do_not_depend_on_their_call(solver):
    """More tiles than resident CTAs: the rows of one call give bit for bit
    what they give in a call of their own."""
    import torch
    n, cut = 592 * 128 + 5, 592 * 128 - 128
    P, X, _ = random_problem(n, 41)
    Pd = torch.from_numpy(P).to("cuda")
    out = []
    for lo in (0, cut):
        feat = torch.from_numpy(X[lo:].view(np.int16).copy()).to("cuda")
        cls = torch.zeros(n - lo, dtype=torch.uint8, device="cuda")
        logits = torch.zeros((n - lo, 3), device="cuda")
        torch.cuda.synchronize()
        solver.mlp_forward(Pd.data_ptr(), n - lo, feat.data_ptr(), cls.data_ptr(), logits.data_ptr())
        out.append((cls.cpu().numpy()[cut - lo:], logits.cpu().numpy()[cut - lo:]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n,off", [(100, 0), (129, 1), (148 * 128 + 77, 0)])
def test_gradient_tiles(solver, n, off):
    import torch
    P, X, y = random_problem(n, 23 + n)
    keep, pptr = shifted(P, off)
    feat = torch.from_numpy(X.view(np.int16)).to("cuda")
    lab = torch.from_numpy(y).to("cuda")
    g = torch.zeros(P.size, device="cuda")
    st = torch.zeros(2, device="cuda")
    torch.cuda.synchronize()
    cw = np.array([1.0, 2.0, 0.5], np.float32)
    solver.mlp_grad(pptr, n, feat.data_ptr(), lab.data_ptr(), cw, g.data_ptr(), st.data_ptr())
    _, ref, _ = io.mlp_loss_grad(P, y, cw.astype(np.float64), X_bits=X)
    got = g.cpu().numpy()
    for a, b in ((0, io.P_B1), (io.P_B1, io.P_W2), (io.P_W2, io.P_B2), (io.P_B2, io.P_W3),
                 (io.P_W3, io.P_COUNT)):
        assert np.linalg.norm(got[a:b] - ref[a:b]) <= GRAD_REL_TOL * np.linalg.norm(ref[a:b])
    del keep

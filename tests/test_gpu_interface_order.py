"""Coarse/fine fills of several levels in one launch: where a level's pairs
read what another level's pairs write, the reference's order (restriction of
ascending coarse levels, then prolongation of ascending coarse levels,
AMRInterface.cpp:3-35) has to hold; where they do not, the launch is shared.
Held against the formulas applied pair by pair in that order.
"""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu

pkg = load_pkg()
ib, wl = pkg.ibgpu, pkg.workloads
SONS = [(0, 0), (0, 1), (1, 0), (1, 1)]


def pair(l, cx, cy, fx, fy):
    row = [l, cx, cy]
    for dx, dy in SONS:
        row += [fx + dx, fy + dy]
    return row


def recover(g, rho, u, v, e):
    p = (e - 0.5 * (u * u + v * v)) * (g["gama"] - 1.0) * rho
    return [rho, u, v, 0.0, p, p / (rho * g["Rg"]), e]


def fill(g, cells, res, pro):
    for r in sorted(res, key=lambda r: r[0]):
        s = [cells[r[0] + 1, r[3 + 2 * k], r[4 + 2 * k]] for k in range(4)]
        rho = sum(c[0] for c in s)
        u, v, e = (sum(c[k] * c[0] for c in s) / rho for k in (1, 2, 6))
        cells[r[0], r[1], r[2]] = recover(g, 0.25 * rho, u, v, e)
    for r in sorted(pro, key=lambda r: r[0]):
        l, x, y = r[:3]
        U = [np.array([c[0], c[0] * c[1], c[0] * c[2], c[0] * c[6]]) for c in
             (cells[l, x, y], cells[l, x - 1, y], cells[l, x + 1, y], cells[l, x, y - 1],
              cells[l, x, y + 1])]
        for k, (dx, dy) in enumerate(SONS):
            f = U[0] + (dx - 0.5) * 0.5 * 0.5 * (U[2] - U[1]) + (dy - 0.5) * 0.5 * 0.5 * (U[4] - U[3])
            cells[l + 1, r[3 + 2 * k], r[4 + 2 * k]] = recover(g, f[0], f[1] / f[0], f[2] / f[0], f[3] / f[0])


# the level-1 pairs read the level-0 pairs' sons (chained) or cells apart
@pytest.mark.parametrize("chained", [True, False])
@pytest.mark.parametrize("precision", [ib.FP64, ib.FP64_EXACT])
def test_fills_keep_the_order_between_levels(cuda_lib, chained, precision):
    g = wl.gas_constants(0.5, 0.0)
    init = wl.freestream(g, 0.2)
    r = np.random.default_rng(5)
    keys = [(l, x, y) for l in range(3) for y in range(40) for x in range(40)]
    lv, x, y = np.array(keys, np.int32).T
    prim = np.empty((len(keys), 7))
    prim[:, 0], prim[:, 4] = r.uniform(0.5, 1.5, len(keys)), r.uniform(2.0, 3.0, len(keys))
    prim[:, 1], prim[:, 2], prim[:, 3] = r.uniform(-1, 1, len(keys)), r.uniform(-1, 1, len(keys)), 0.0
    prim[:, 5] = prim[:, 4] / (prim[:, 0] * g["Rg"])
    prim[:, 6] = g["Cv"] * prim[:, 5] + 0.5 * (prim[:, 1] ** 2 + prim[:, 2] ** 2)
    cx = 6 if chained else 30  # level-1 coarse cells: inside the sons below, or not
    res = [pair(1, cx, 6, 20, 20), pair(0, 9, 9, 6, 6), pair(0, 4, 9, 30, 10)]
    pro = [pair(1, cx + 1, 11, 2, 2), pair(0, 17, 3, 6, 10), pair(0, 20, 3, 8, 10),
           pair(1, 34, 30, 12, 2)]
    params = dict(g, cfl=0.5, dt_ratio=1.0, dt_var_step=4, nstages=3, tp=wl.TP[3], limiter=0,
                  viscous=0, precision=precision, initvar=init, nlevels=3,
                  dh=[(0.4 / 2 ** l, 0.4 / 2 ** l, 0.1) for l in range(3)], march_step=[4, 2, 1],
                  march_left=[0, 0, 0], step_num=[4.0, 2.0, 1.0], average_step=[1, 1, 1],
                  average_left=[0, 0, 0], prolong_step=[1, 1, 1], prolong_left=[0, 0, 0],
                  domain_nx=64, domain_ny=64, dt0=1.0)
    s = ib.FlowSolver(params)
    s.upload_topology(lv, x, y, np.full(len(keys), ib.CELL_PRESENT, np.uint8))
    s.upload_interfaces(np.array(res), np.array(pro))
    s.init_flow(prim)
    s.run(0, 1)
    got = s.download()
    s.close()
    cells = {k: list(row) for k, row in zip(keys, prim)}
    fill(g, cells, res, pro)
    ref = np.array([cells[k] for k in keys])
    assert np.abs(ref - prim).max() > 0.1  # the fills did something
    # a few dozen roundings of values of order one
    assert np.abs(got - ref).max() <= 1e-13

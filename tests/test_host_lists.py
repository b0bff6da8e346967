"""The lists of a context (coarse/fine pairs, domain ghosts, immersed cells)
on their way into the fills' launches: what a step launches is what was
uploaded last, and arrays that were freed are never passed on."""
import os
import struct
import sys

import numpy as np
import pytest

from conftest import GOLDEN_DIR, load_pkg
from host_api import HostApi, words

sys.path.insert(0, GOLDEN_DIR)
import make_golden  # noqa: E402

wl = load_pkg().workloads


@pytest.fixture(scope="module")
def api(tmp_path_factory):
    return HostApi(str(tmp_path_factory.mktemp("host")))


@pytest.fixture(scope="module")
def record():
    return make_golden.load("naca_minmod_s4_n64_l3")


def upload(s, L, which=("cf", "bc", "ib"), backpressure=None, bc=None, ib=None):
    if "cf" in which:
        s.upload_interfaces(L["res"], L["pro"])
    if "bc" in which:
        n = len(L["bc"]) if bc is None else bc
        s.upload_boundaries(L["bc"][:n], L["bc_nmv"][:n], L["facevar"],
                            L["bc_scalars"][0] if backpressure is None else backpressure,
                            L["bc_scalars"][1])
    if "ib" in which:
        n = len(L["ib"]) if ib is None else ib
        s.upload_ib(L["ib"][:n], L["ib_f"][:n], L["patch"], L["patch_f"], L["body_center"])


def solver(api, record, precision="FP64"):
    L = wl.naca_lists(record, 0)
    s = api.ib.FlowSolver(wl.naca_params(record, 0, getattr(api.ib, precision)))
    s.upload_topology(L["level"], L["ix"], L["iy"], L["flags"])
    upload(s, L)
    s.init_flow(L["prim"])
    return s, L


def low32(word):
    return struct.unpack("<i", struct.pack("<q", word)[:4])[0]


def as_double(word):
    return struct.unpack("<d", struct.pack("<q", word))[0]


# the first segment of a batched launch is the first case's
def first_bc(api):
    """(ghost pointer, backpressure) of BatchBc[0]"""
    w = words(api.launches("bc_kernel_batch")[-1][2][0], 8)
    return w[0], as_double(w[7])


def first_ib(api):
    """(cell pointer, cells) of BatchIb[0]"""
    w = words(api.launches("ib_kernel_batch")[-1][2][0], 5)
    return w[0], low32(w[4])


def test_batch_takes_up_lists_uploaded_after_its_creation(api, record):
    (a, L), (b, _) = solver(api, record), solver(api, record)
    batch = api.ib.Batch([a, b])
    for k, (pressure, nbc, nib) in enumerate([(0.25, 40, 30), (0.5, len(L["bc"]), len(L["ib"]))]):
        upload(a, L, backpressure=pressure, bc=nbc, ib=nib)  # before the first run, and after it
        api.clear()
        batch.run(0, 4)
        ghost, got = first_bc(api)
        assert got == pressure and api.live(ghost)
        cell, n = first_ib(api)
        assert n == nib and api.live(cell)
        for part in ("restrict_kernel_batch", "prolong_kernel_batch"):
            seg = words(api.launches(part)[-1][2][0], 2)
            assert api.live(seg[0]) and api.live(seg[1])
        # unchanged lists: the captured steps serve
        api.clear()
        batch.run(4, 4)
        assert not api.launches("bc_kernel_batch")
    batch.close()
    a.close()
    b.close()


def run_and_check_pointers(api, s, part, n):
    """Four steps; every launch whose kernel's name contains `part` gets live
    arrays in its first n arguments.  Returns the number of these launches."""
    api.clear()
    s.run(0, 4)
    launches = api.launches(part)
    assert api.launches("stage_kernel")
    for name, _, w in launches:
        assert all(api.live(p) for p in w[:n]), name
    return len(launches)


# five arrays: coarse, sons (and neighbours) of both lists
@pytest.mark.parametrize("nth", range(1, 6))
def test_failed_interface_upload_leaves_no_pairs(api, record, nth):
    s, L = solver(api, record)
    assert run_and_check_pointers(api, s, "restrict_kernel", 2)
    assert run_and_check_pointers(api, s, "prolong_kernel", 3)
    api.fail_malloc(nth)
    with pytest.raises(api.ib.IbgpuError) as e:
        upload(s, L, ("cf",))
    api.fail_malloc(0)
    assert e.value.code == api.ib.E_NOMEM
    assert run_and_check_pointers(api, s, "restrict_kernel", 2) == 0
    assert run_and_check_pointers(api, s, "prolong_kernel", 3) == 0
    upload(s, L, ("cf",))
    assert run_and_check_pointers(api, s, "restrict_kernel", 2)
    s.close()


# refused (an unknown type), or one of its six allocations fails
@pytest.mark.parametrize("nth", range(7))
def test_failed_boundary_upload_leaves_no_ghosts(api, record, nth):
    s, L = solver(api, record)
    assert run_and_check_pointers(api, s, "bc_kernel", 6)
    if nth == 0:
        bad = dict(L, bc=L["bc"].copy())
        bad["bc"][-1, 6] = -3
    else:
        bad = L
        api.fail_malloc(nth)
    with pytest.raises(api.ib.IbgpuError) as e:
        upload(s, bad, ("bc",))
    api.fail_malloc(0)
    assert e.value.code == (api.ib.E_NOMEM if nth else api.ib.E_ARG)
    assert run_and_check_pointers(api, s, "bc_kernel", 6) == 0
    upload(s, L, ("bc",))
    assert run_and_check_pointers(api, s, "bc_kernel", 6)
    s.close()


# eleven buffers, which longer lists make grow (all but the body's own three)
@pytest.mark.parametrize("nth", range(1, 9))
def test_failed_body_upload_leaves_no_cells(api, record, nth):
    s, L = solver(api, record)
    assert run_and_check_pointers(api, s, "ib_kernel", 4)
    longer = dict(L, **{k: np.repeat(L[k], 2, 0) for k in ("ib", "ib_f", "patch", "patch_f")})
    api.fail_malloc(nth)
    with pytest.raises(api.ib.IbgpuError) as e:
        upload(s, longer, ("ib",))
    api.fail_malloc(0)
    assert e.value.code == api.ib.E_NOMEM
    assert run_and_check_pointers(api, s, "ib_", 4) == 0
    api.clear()
    s.wall_forces()
    assert not api.launches("force")
    upload(s, longer, ("ib",))
    assert run_and_check_pointers(api, s, "ib_kernel", 4)
    s.close()


def chained_mesh(chained):
    """Three levels of 40 x 40 cells whose level-1 pairs touch the cells that
    the level-0 pairs read (restriction) and write (prolongation), or not."""
    from test_gpu_interface_order import pair
    cx = 6 if chained else 30
    keys = np.array([(l, x, y) for l in range(3) for y in range(40) for x in range(40)], np.int32)
    g = wl.gas_constants(0.5, 0.0)
    P = dict(g, cfl=0.5, dt_ratio=1.0, dt_var_step=4, nstages=3, tp=wl.TP[3],
             initvar=wl.freestream(g, 0.2), nlevels=3,
             dh=[(0.4 / 2 ** l, 0.4 / 2 ** l, 0.1) for l in range(3)], march_step=[4, 2, 1],
             march_left=[0, 0, 0], step_num=[4.0, 2.0, 1.0], average_step=[1, 1, 1],
             average_left=[0, 0, 0], prolong_step=[1, 1, 1], prolong_left=[0, 0, 0],
             domain_nx=64, domain_ny=64, dt0=1.0)
    res = [pair(1, cx, 6, 20, 20), pair(0, 9, 9, 6, 6)]
    pro = [pair(1, cx + 1, 11, 2, 2), pair(0, 17, 3, 6, 10)]
    return P, keys.T, res, pro


@pytest.mark.parametrize("chained", [True, False])
def test_levels_share_a_fill_launch_only_when_independent(api, chained):
    P, (lv, x, y), res, pro = chained_mesh(chained)
    sols = []
    for _ in range(2):
        s = api.ib.FlowSolver(P)
        s.upload_topology(lv, x, y, np.full(len(lv), api.ib.CELL_PRESENT, np.uint8))
        s.upload_interfaces(np.array(res), np.array(pro))
        s.init_flow(np.ones((len(lv), 7)))
        sols.append(s)
    pairs = [1, 1] if chained else [2]
    api.clear()
    sols[0].run(0, 1)
    for part in ("restrict_kernel", "prolong_kernel"):
        assert [low32(w[3]) for _, _, w in api.launches(part)] == pairs
    # the k-th launch of every case in one: a block each
    b = api.ib.Batch(sols)
    api.clear()
    b.run(0, 1)
    for part in ("restrict_kernel_batch", "prolong_kernel_batch"):
        grids = [g for _, g, _ in api.launches(part)]
        assert grids[:len(pairs)] == [2] * len(pairs)
    b.close()
    for s in sols:
        s.close()


# one CTA takes 1024 immersed cells; more, two launches with the states between
@pytest.mark.parametrize("n,kernels", [(1024, ["ib_kernel"]), (1025, ["ib_compute", "ib_store"])])
def test_immersed_cells_choose_their_launches(api, record, n, kernels):
    (a, L), (b, _) = solver(api, record), solver(api, record)
    many = dict(L, ib=np.resize(L["ib"], (n, 18)), ib_f=np.resize(L["ib_f"], (n, 16)))
    upload(a, many, ("ib",))
    api.clear()
    a.run(0, 1)
    names = [name for name, _, _ in api.launches("ib_")]
    assert len(names) == len(kernels) and all(k in m for k, m in zip(kernels, names))
    batch = api.ib.Batch([a, b])
    api.clear()
    batch.run(0, 1)
    assert bool(api.launches("ib_kernel_batch")) == (n <= 1024)
    assert bool(api.launches("ib_compute")) == (n > 1024)
    batch.close()
    a.close()
    b.close()

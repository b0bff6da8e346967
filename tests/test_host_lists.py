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

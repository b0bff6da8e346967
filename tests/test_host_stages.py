"""What the stages of a step read and write, from their recorded launches: no
stage may read the step state's rho, u, v, p as its input and write them back
in the same launch (neighbouring CTAs read what it overwrites)."""
import re

import pytest

from conftest import load_pkg
from host_api import HostApi, words

wl = load_pkg().workloads

# StageArgs (csrc/layout.h) in 64-bit words: the six state fields from 4,
# then vsd, nslots, diag, two words of integers, the input's four fields
S0, SIN, SIZE = 4, 15, 200
# FINAL among the template arguments (type, limiter, viscous, final)
FINAL = re.compile(r"I[df]Li[01]ELb[01]ELb([01])E")


@pytest.fixture(scope="module")
def api(tmp_path_factory):
    return HostApi(str(tmp_path_factory.mktemp("host")))


def case(n, precision, nstages):
    tp = {1: [1.0], **wl.TP}[nstages]
    P, cells, prim = wl.vortex_case(n, nstages=max(nstages, 3), precision=precision)
    return dict(P, nstages=nstages, tp=tp), cells, prim


def solver(api, n, precision, nstages):
    P, cells, prim = case(n, precision, nstages)
    s = api.ib.FlowSolver(P)
    s.upload_topology(**cells)
    s.init_flow(prim)
    return s


def races(w):
    return sorted(set(w[S0:S0 + 6]) & set(w[SIN:SIN + 4]))


def step(f):
    """A step; nothing computed here, so a zero dt or residual is no matter."""
    try:
        f()
    except Exception as e:  # noqa: BLE001
        assert getattr(e, "code", None) is not None, e


@pytest.mark.parametrize("nstages", [1, 3])
@pytest.mark.parametrize("precision", ["FP64", "MIXED", "FP64_EXACT"])
def test_final_stage_reads_no_field_it_writes(api, precision, nstages):
    s = solver(api, 48, getattr(api.ib, precision), nstages)
    api.clear()
    step(lambda: s.run(0, 2))
    stages = api.launches("stage_kernel")
    assert len(stages) == 2 * nstages
    for k, (_, _, w) in enumerate(stages):
        assert all(api.live(p) for p in w[S0:S0 + 6] + w[SIN:SIN + 4])
        if k % nstages == nstages - 1:
            assert not races(w)
    s.close()


@pytest.mark.parametrize("nstages", [1, 3])
@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_batched_final_stage_reads_no_field_it_writes(api, precision, nstages):
    sols = [solver(api, n, getattr(api.ib, precision), nstages) for n in (48, 32)]
    b = api.ib.Batch(sols)
    api.clear()
    step(lambda: b.run(0, 2))
    launches = api.launches("stage_kernel_batch")
    args = launches[0][2][0]
    for c in range(2):
        assert not races(words(args, 20, SIZE * (c * nstages + nstages - 1)))
    # tuning comes first and advances nothing, then the captured steps (the
    # CFL pass's and, for these cases, the one with the folded bound)
    final = [FINAL.search(n).group(1) == "1" for n, _, _ in launches]
    captured = 2 * nstages
    assert len(final) > captured and not any(final[:-captured])
    assert final[-captured:] == 2 * ([False] * (nstages - 1) + [True])
    b.close()
    for s in sols:
        s.close()


@pytest.mark.parametrize("nstages", [1, 3])
@pytest.mark.parametrize("precision", ["FP64", "MIXED", "FP64_EXACT"])
def test_allocation_free_final_stage_reads_no_field_it_writes(api, precision, nstages):
    import numpy as np
    P, cells, prim = case(48, getattr(api.ib, precision), nstages)
    rows = np.ascontiguousarray(prim)
    api.clear()
    step(lambda: api.ib.step_periodic_noalloc(P, 0, 48, 48, rows.ctypes.data, rows.ctypes.data, 1.0))
    stages = api.launches("stage_kernel")
    assert len(stages) == nstages and not races(stages[-1][2])


@pytest.mark.parametrize("precision,resident", [("FP64", {256: 4, 288: 4}), ("MIXED", {256: 5, 288: 4})])
def test_tuning_times_resident_grids_only(api, precision, resident):
    s = solver(api, 512, getattr(api.ib, precision), 3)  # 1024 tiles
    b = api.ib.Batch([s])
    b.run(0, 1)
    tuned = {}
    for grid, threads, _ in b.info()["tuning"]:
        tuned.setdefault(threads, []).append(grid)
    # one CTA per item, then persistent ones on 148 multiprocessors
    assert tuned == {t: [148 * m for m in range(n + 1)] for t, n in resident.items()}
    b.close()
    s.close()

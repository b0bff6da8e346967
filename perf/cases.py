"""The work that users of this framework run, as measurable cases.

Each case goes through the public Python entry points (``FlowSolver``,
``Batch``, ``step_periodic_noalloc``).  What a user's program keeps between
calls (the uploaded mesh, the batch, network parameters, pinned buffers) is
made in ``prepare``; ``run`` is one pass.  ``exact`` computes the same
outputs in 64 bits with plain torch on the list form of the mesh.

Kinds of case:
  step     one step of a small periodic grid whose rows the caller keeps on
           the device (coupling loops with foreign device memory)
  coupled  one step with the state handed over from and to pinned host
           memory (a host code that keeps the authoritative copy)
  run      the steps between two regrids: state in, ``steps`` steps with one
           synchronisation, state out.  mesh "vortex" is one periodic level,
           "nested" a periodic viscous flow on nested AMR levels, "airfoil"
           the static NACA0012 meshes of tests/golden (immersed body, far
           field, wall forces at the end)
  batch    the same for several airfoil cases advanced together
  train    one optimiser step of the refinement indicator on a minibatch
  forward  its classification of feature rows
  tag      its tags for every cell of a mesh (once per regrid)
"""
from __future__ import annotations

import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

VANLEER, MINMOD = "vanleer", "minmod"


def _pkg():
    name = "immsered_boundary_b200"
    if name not in sys.modules:
        d = os.path.abspath("immsered-boundary_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# --------------------------------------------------------------------------
# the cases

def listed():
    return [
        # smallest call: one step of a small coupled patch, all latency
        dict(name="step_small", kind="step", nx=64, ny=48, precision="fp64", limiter=VANLEER,
             stages=4),
        # a host code exchanging the state every step
        dict(name="coupled_352", kind="coupled", n=352, precision="fp64", limiter=VANLEER,
             stages=4),
        # single-level flow at ordinary size, three-stage minmod
        dict(name="vortex_464_minmod", kind="run", mesh="vortex", n=464, precision="fp64",
             limiter=MINMOD, stages=3, steps=20),
        # the bandwidth workload, both arithmetics, 20 steps between hand-overs
        dict(name="vortex_2048_fp64", kind="run", mesh="vortex", n=2048, precision="fp64",
             limiter=VANLEER, stages=4, steps=20),
        dict(name="vortex_2048_mixed", kind="run", mesh="vortex", n=2048, precision="mixed",
             limiter=VANLEER, stages=4, steps=20),
        # the stated plain airfoil: 45,448 leaf cells, 4 levels, between regrids
        dict(name="airfoil_128", kind="run", mesh="airfoil", base=128, precision="fp64",
             limiter=MINMOD, stages=4, steps=24),
        # a large viscous AMR mesh (900 k cell rows on 4 levels)
        dict(name="nested_914k", kind="run", mesh="nested", n=448, levels=4, frac=0.62,
             precision="fp64", limiter=MINMOD, stages=4, steps=16),
        # a parameter sweep of airfoils in one batch, mixed precision
        dict(name="batch_airfoils", kind="batch", cases=6, precision="mixed", limiter=MINMOD,
             stages=4, steps=16),
        # the indicator's default minibatch, and a full-record gradient step
        dict(name="train_8192", kind="train", rows=8192),
        dict(name="train_262144", kind="train", rows=262144),
        # classification of every box of a regrid
        dict(name="forward_200003", kind="forward", rows=200003),
        # learned tags of a whole mesh
        dict(name="tag_1024", kind="tag", n=1024),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "coupled", "run", "run", "run", "run", "batch", "train", "forward",
                       "tag"])
    flow = dict(precision=rng.choice(["fp64", "fp64", "mixed"]),
                limiter=rng.choice([VANLEER, MINMOD]), stages=rng.choice([3, 4]))
    if kind == "step":
        nx = 16 * int(_log(rng, 1, 16.9))
        return dict(kind=kind, nx=nx, ny=16 * rng.randint(1, min(16, 65536 // (16 * nx))), **flow)
    if kind == "coupled":
        return dict(kind=kind, n=16 * int(_log(rng, 2, 64)), **flow)
    if kind == "run":
        mesh = rng.choice(["vortex", "nested", "nested", "airfoil"])
        if mesh == "vortex":
            return dict(kind=kind, mesh=mesh, n=16 * int(_log(rng, 3, 112)),
                        steps=rng.randint(1, 20), **flow)
        if mesh == "nested":
            return dict(kind=kind, mesh=mesh, n=16 * int(_log(rng, 4, 26)),
                        levels=rng.randint(2, 5), frac=round(rng.uniform(0.4, 0.62), 3),
                        steps=rng.randint(8, 24), **flow)
        return dict(kind=kind, mesh=mesh, base=rng.choice([64, 128]), steps=rng.randint(4, 40),
                    **flow)
    if kind == "batch":
        return dict(kind=kind, cases=rng.randint(2, 8), steps=rng.randint(8, 24), **flow)
    if kind == "tag":
        return dict(kind=kind, n=16 * int(_log(rng, 6, 72)))
    return dict(kind=kind, rows=int(_log(rng, 300, 260000)))


# --------------------------------------------------------------------------
# meshes: canonical lists (the arguments of the upload calls) and parameters

def _rng(case, seed):
    text = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, sum(map(ord, text))])


def _gas(mach, re):
    wl = _pkg().workloads
    g = wl.gas_constants(mach, 0.0 if re is None else 1.0 / re)
    return g


def _flow_params(case, g, init, levels, h, n, viscous):
    """Parameters of a periodic n x n base grid with ``levels`` levels."""
    ib, wl = _pkg().ibgpu, _pkg().workloads
    prec = dict(fp64=ib.FP64, mixed=ib.MIXED)[case["precision"]]
    march = [2 ** (levels - 1 - l) for l in range(levels)]
    nx, ny = n
    return dict(g, cfl=0.5, dt_ratio=1.0, dt_var_step=march[0], nstages=case["stages"],
                tp=wl.TP[case["stages"]], limiter=dict(vanleer=ib.LIM_VANLEER, minmod=ib.LIM_MINMOD)[case["limiter"]],
                viscous=int(viscous), precision=prec, initvar=init, nlevels=levels,
                dh=[(h / 2 ** l, h / 2 ** l, 0.1) for l in range(levels)], march_step=march,
                march_left=[0] * levels, step_num=[float(m) for m in march],
                average_step=[2 * m for m in march], average_left=march,
                prolong_step=[2 * m for m in march], prolong_left=march,
                domain_nx=nx, domain_ny=ny, periodic_x=1, periodic_y=1, dt0=1.0)


LEAF = 1 | 2 | 4 | 8 | 32  # present, normal, update, recovers primitives, in the residual norm


def _vortex(case, seed, nx, ny):
    """One periodic level holding an advected isentropic vortex."""
    wl = _pkg().workloads
    r = _rng(case, seed)
    g = _gas(float(r.uniform(0.2, 0.7)), None)
    init = wl.freestream(g, float(r.uniform(0.0, 1.5)))
    h = 10.0 / max(nx, ny)
    iy, ix = np.meshgrid(np.arange(ny, dtype=np.int32), np.arange(nx, dtype=np.int32), indexing="ij")
    ix, iy = ix.ravel(), iy.ravel()
    c = r.uniform(0.4, 0.6, 2) * (nx * h, ny * h)
    prim = wl.vortex_state(ix, iy, h, g, init, float(r.uniform(3.0, 5.0)), c[0], c[1])
    return dict(params=_flow_params(case, g, init, 1, h, (nx, ny), False),
                level=np.zeros_like(ix), ix=ix, iy=iy, flags=np.full(ix.shape, LEAF, np.uint8),
                prim=prim)


def _any8(m):
    """Positions with a set position among their 8 neighbours."""
    p = np.pad(m, 1)
    row = p[:-2] | p[1:-1] | p[2:]
    out = row[:, :-2] | row[:, 2:]
    return out | p[:-2, 1:-1] | p[2:, 1:-1]


@functools.lru_cache(maxsize=4)
def _nested_mesh(n, levels, frac):
    """Leaf, interface-ghost and pair lists of nested refined rectangles
    (wake-shaped: longer than high, off centre, edges off the tile grid)."""
    refined, leaf = [], []
    cover = np.ones((n, n), bool)
    x0, y0, w, hgt = 0.0, 0.0, 1.0, 1.0
    for l in range(levels):
        m = n << l
        ref = np.zeros((m, m), bool)
        if l + 1 < levels:
            x0, y0 = x0 + w * (1 - frac) * 0.4, y0 + hgt * (1 - frac * 0.8) * 0.55
            w, hgt = w * frac, hgt * frac * 0.8
            ref[int(y0 * m):int((y0 + hgt) * m), int(x0 * m):int((x0 + w) * m)] = True
        refined.append(ref)
        leaf.append(cover & ~ref)
        cover = np.repeat(np.repeat(ref, 2, 0), 2, 1)
    sons = [(0, 0), (0, 1), (1, 0), (1, 1)]

    def rows(l, mask):
        y, x = np.nonzero(mask)
        cols = [np.full(len(x), l), x, y]
        for dx, dy in sons:
            cols += [2 * x + dx, 2 * y + dy]
        return np.stack(cols, 1).astype(np.int32)

    res, pro, ghost = [], [], [np.zeros_like(r) for r in refined]
    for l in range(levels - 1):
        four = refined[l] & ~np.any(
            [refined[l + 1][dy::2, dx::2] for dx, dy in sons], axis=0)
        two = np.zeros_like(leaf[l])
        for ax in (0, 1):
            for s in (-2, 2):
                two |= np.roll(leaf[l], s, ax)
        layer0 = four & _any8(leaf[l])
        r = layer0 | (four & two)
        p = leaf[l] & _any8(refined[l])
        ghost[l] |= r
        for dx, dy in sons:
            ghost[l + 1][dy::2, dx::2] |= p
        res.append(rows(l, r))
        pro.append(rows(l, p))
    lv, xs, ys, fl = [], [], [], []
    for l in range(levels):
        for mask, f in ((leaf[l], LEAF), (ghost[l], 1)):
            y, x = np.nonzero(mask)
            lv.append(np.full(len(x), l, np.int32))
            xs.append(x.astype(np.int32))
            ys.append(y.astype(np.int32))
            fl.append(np.full(len(x), f, np.uint8))
    empty = [np.zeros((0, 11), np.int32)]
    return (np.concatenate(lv), np.concatenate(xs), np.concatenate(ys), np.concatenate(fl),
            np.concatenate(res + empty), np.concatenate(pro + empty))


def _nested(case, seed):
    wl = _pkg().workloads
    n, levels = case["n"], case["levels"]
    lv, ix, iy, fl, res, pro = _nested_mesh(n, levels, case["frac"])
    r = _rng(case, seed)
    g = _gas(float(r.uniform(0.2, 0.7)), 10 ** float(r.uniform(3.3, 4.3)))
    init = wl.freestream(g, float(r.uniform(-0.1, 0.2)))
    h = 10.0 / n
    xy = r.uniform(4.5, 5.5, 2)
    beta = float(r.uniform(3.0, 5.0))
    prim = np.empty((len(lv), 7))
    for l in range(levels):
        m = lv == l
        prim[m] = wl.vortex_state(ix[m], iy[m], h / 2 ** l, g, init, beta, xy[0], xy[1])
    return dict(params=_flow_params(case, g, init, levels, h, (n, n), True), level=lv, ix=ix,
                iy=iy, flags=fl, res=res, pro=pro, prim=prim)


RECORD = {64: "naca_minmod_s4_n64_l3", 128: "naca_minmod_s4_n128_l4"}


@functools.lru_cache(maxsize=2)
def _record(base):
    with np.load(os.path.join("tests", "golden", RECORD[base] + ".npz")) as z:
        return {k: z[k] for k in z.files if k != "tags"}


def _airfoil(case, seed, base, salt=0):
    """A recorded NACA0012 mesh with its flow, disturbed a little."""
    ib, wl = _pkg().ibgpu, _pkg().workloads
    g = _record(base)
    k = len(g["prim"]) - 1
    P = wl.naca_params(g, k, dict(fp64=ib.FP64, mixed=ib.MIXED)[case["precision"]])
    L = wl.naca_lists(g, k)
    P.update(dt0=1.0, nstages=case["stages"], tp=wl.TP[case["stages"]],
             limiter=dict(vanleer=ib.LIM_VANLEER, minmod=ib.LIM_MINMOD)[case["limiter"]])
    r = np.random.default_rng([int(seed) & 0x7FFFFFFF, salt, base])
    h = np.array([d[0] for d in P["dh"]])[L["level"]]
    x, y = (L["ix"] + 0.5) * h, (L["iy"] + 0.5) * h
    a, kx, ky, ph = r.uniform(0.005, 0.02), *r.uniform(1.0, 3.0, 2), r.uniform(0, 6.28)
    prim = L["prim"].copy()
    prim[:, 1] *= 1 + a * np.sin(kx * x + ph) * np.cos(ky * y)
    prim[:, 2] += 0.5 * a * np.cos(kx * x) * np.sin(ky * y + ph)
    prim[:, 6] = P["Cv"] * prim[:, 5] + 0.5 * (prim[:, 1] ** 2 + prim[:, 2] ** 2)
    return dict(L, params=P, prim=prim)


def _meshes(case, seed):
    if case["kind"] == "coupled":
        return [_vortex(case, seed, case["n"], case["n"])]
    if case["kind"] == "batch":
        return [_airfoil(case, seed, (128, 64)[i % 2], i) for i in range(case["cases"])]
    if case["mesh"] == "vortex":
        return [_vortex(case, seed, case["n"], case["n"])]
    if case["mesh"] == "nested":
        return [_nested(case, seed)]
    return [_airfoil(case, seed, case["base"])]


# --------------------------------------------------------------------------
# states

def _solver(M):
    s = _pkg().ibgpu.FlowSolver(M["params"])
    s.upload_topology(M["level"], M["ix"], M["iy"], M["flags"])
    if "res" in M:
        s.upload_interfaces(M["res"], M["pro"])
    if "bc" in M:
        s.upload_boundaries(M["bc"], M["bc_nmv"], M["facevar"], *M["bc_scalars"])
        s.upload_ib(M["ib"], M["ib_f"], M["patch"], M["patch_f"], M["body_center"])
    return s


def _flow_state(M, compact):
    s = _solver(M)
    rows = M["prim"][:, [0, 1, 2, 4]] if compact else M["prim"]
    if compact:
        s.set_state_rows(_pkg().ibgpu.ROWS_COMPACT)
    host = torch.from_numpy(np.ascontiguousarray(rows)).pin_memory()
    return dict(solver=s, rows=host, out=torch.empty_like(host).pin_memory())


def _network(case, seed):
    """Parameters of a half-trained indicator, feature rows and labels like
    the ones a record gives: small flow deviations, clipped distances, a
    one-hot level; labels mostly "keep"."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    n = case.get("rows", 0)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, dtype=torch.float32)

    P = torch.cat([normal(64 * 112) * math.sqrt(2 / 112), normal(64) * 0.1,
                   normal(64 * 64) * math.sqrt(2 / 64), normal(64) * 0.1,
                   normal(3 * 64) * math.sqrt(1 / 64), normal(3) * 0.1])
    if not n:
        return P, None, None, None, None
    X = torch.zeros(n, 112)
    X[:, :100] = normal(n, 100) * 0.15 + normal(n, 1) * 0.3
    X[:, 100:105] = normal(n, 5).clamp(-1, 1)
    lev = torch.randint(0, 5, (n,), generator=gen)
    X[torch.arange(n), 105 + lev] = 1.0
    y = torch.randint(0, 10, (n,), generator=gen).clamp(max=2).to(torch.uint8)
    m = normal(P.numel()) * 1e-3
    v = (normal(P.numel()) * 1e-2) ** 2 + 1e-5
    return P, X.to(torch.bfloat16), y, m, v


def _wake_distance(M):
    h = np.array([d[0] for d in M["params"]["dh"]])[M["level"]]
    x, y = (M["ix"] + 0.5) * h, (M["iy"] + 0.5) * h
    return np.hypot(x - np.clip(x, 4.5, 5.5), y - 5.0) - 0.06


def _indicator_solver():
    """The solver an indicator belongs to (its stream and device)."""
    return _solver(_vortex(dict(kind="net", precision="fp64", limiter=VANLEER, stages=4), 0, 32, 32))


def prepare(case, seed):
    kind = case["kind"]
    torch.cuda.init()
    if kind == "step":
        M = _vortex(case, seed, case["nx"], case["ny"])
        rows = torch.from_numpy(M["prim"]).cuda()
        return dict(case=case, params=M["params"], rows=rows, out=torch.empty_like(rows))
    if kind in ("coupled", "run"):
        M = _meshes(case, seed)[0]
        compact = kind == "coupled" or case["mesh"] == "vortex"
        return dict(case=case, body="bc" in M, **_flow_state(M, compact))
    if kind == "batch":
        each = [_flow_state(M, False) for M in _meshes(case, seed)]
        for s in each:
            s["solver"].init_flow(s["rows"].data_ptr())
        batch = _pkg().ibgpu.Batch([s["solver"] for s in each])
        return dict(case=case, each=each, batch=batch)
    if kind == "tag":
        M = _vortex(dict(case, precision="fp64", limiter=VANLEER, stages=4), seed, case["n"], case["n"])
        s = _solver(M)
        s.init_flow(M["prim"])
        s.upload_signdis(_wake_distance(M))
        rule = _pkg().workloads.naca_tag_rule(3, [d[0] for d in M["params"]["dh"] * 3], 4.5, 5.0)
        return dict(case=case, solver=s, rule=rule, params=_network(case, seed)[0].cuda())
    P, X, y, m, v = (t.cuda() for t in _network(case, seed))
    stream = torch.cuda.Stream()
    s = _indicator_solver()
    s.set_stream(stream.cuda_stream)
    n = case["rows"]
    st = dict(case=case, solver=s, stream=stream, params=P, feat=X.view(torch.int16))
    if kind == "forward":
        st.update(cls=torch.empty(n, dtype=torch.uint8, device="cuda"),
                  logits=torch.empty((n, 3), device="cuda"))
    else:
        st.update(m=m, v=v, label=y, grad=torch.zeros_like(P), stats=torch.zeros(2, device="cuda"),
                  step=60)
    return st


WEIGHTS = (1.2, 1.1, 0.6)  # class weights of a record with mostly "keep" boxes


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "step":
        dt, d = _pkg().ibgpu.step_periodic_noalloc(
            state["params"], 0, c["nx"], c["ny"], state["rows"].data_ptr(),
            state["out"].data_ptr(), 1.0)
        return dict(rows=state["out"], dt=dt, res=np.array(list(d.res_max)))
    if kind == "coupled":
        s = state["solver"]
        s.dt = 1.0
        s.upload_async(state["rows"].data_ptr())
        s.step_async(0)
        s.download_async(state["out"].data_ptr())
        d = s.step_result()
        s.synchronize()
        return dict(rows=state["out"], dt=s.dt, res=np.array(list(d.res_max)))
    if kind == "run":
        s = state["solver"]
        s.dt = 1.0
        s.init_flow(state["rows"].data_ptr())
        d = s.run(0, c["steps"])
        s.download(state["out"].data_ptr())
        got = dict(rows=state["out"], dt=s.dt, res=np.array(list(d.res_max)))
        if state["body"]:
            got["forces"] = s.wall_forces()
        return got
    if kind == "batch":
        for e in state["each"]:
            e["solver"].dt = 1.0
            e["solver"].init_flow(e["rows"].data_ptr())
        state["batch"].run(0, c["steps"])
        for e in state["each"]:
            e["solver"].download(e["out"].data_ptr())
        return dict(rows=[e["out"] for e in state["each"]],
                    forces=[e["solver"].wall_forces() for e in state["each"]],
                    dt=[e["solver"].dt for e in state["each"]])
    s = state["solver"]
    if kind == "tag":
        return dict(tags=s.tag_mesh(state["rule"], state["params"].data_ptr()))
    if kind == "forward":
        s.mlp_forward(state["params"].data_ptr(), c["rows"], state["feat"].data_ptr(),
                      state["cls"].data_ptr(), state["logits"].data_ptr())
        return dict(cls=state["cls"], logits=state["logits"])
    state["step"] += 1
    with torch.cuda.stream(state["stream"]):
        state["stats"].zero_()
    s.mlp_train_step(state["params"].data_ptr(), state["m"].data_ptr(), state["v"].data_ptr(),
                     state["grad"].data_ptr(), state["step"], 3e-3, c["rows"],
                     state["feat"].data_ptr(), state["label"].data_ptr(), WEIGHTS,
                     state["stats"].data_ptr())
    return dict(grad=state["grad"], params=state["params"], m=state["m"], v=state["v"],
                stats=state["stats"])


# --------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind in ("train", "forward"):
        n = case["rows"]
        products = 112 * 64 + 64 * 64 + 64 * 3
        if kind == "forward":
            return dict(bytes=n * (224 + 1 + 12) + 46348, flops=2 * n * products)
        return dict(bytes=n * 225 + 7 * 46348, flops=2 * n * (3 * products - 112 * 64))
    if kind == "tag":
        cells = case["n"] ** 2
        return dict(bytes=cells * (4 * 8 + 8 + 1 + 1),
                    flops=2 * cells * (112 * 64 + 64 * 64 + 64 * 3))
    per_stage = 400  # two faces, eight limited slopes, update and recovery
    if kind == "step":
        cells = case["nx"] * case["ny"]
        return dict(bytes=2 * 56 * cells, flops=per_stage * case["stages"] * cells)
    if kind == "coupled":
        return dict(bytes=2 * 32 * case["n"] ** 2,
                    flops=per_stage * case["stages"] * case["n"] ** 2)
    # several steps: the state goes through memory once per step, and over
    # the bus at both ends
    total = rows = 0
    for leaves, steps, present in _leaf_counts(case):
        total += sum(c for ts in range(steps) for l, c in enumerate(leaves)
                     if ts % 2 ** (len(leaves) - 1 - l) == 0)
        rows += present
    width = 32 if case.get("mesh") == "vortex" else 56
    viscous = 0 if case.get("mesh") == "vortex" else 120
    return dict(bytes=64 * total + 2 * width * rows,
                flops=total * (per_stage * case["stages"] + viscous))


def _leaf_counts(case):
    """(leaf cells per level, steps, rows) of each mesh of a case."""
    if case.get("mesh") == "vortex":
        return [([case["n"] ** 2], case["steps"], case["n"] ** 2)]
    if case.get("mesh") == "nested":
        lv, _, _, fl, _, _ = _nested_mesh(case["n"], case["levels"], case["frac"])
        return [(np.bincount(lv[(fl & 2) != 0]).tolist(), case["steps"], len(lv))]
    bases = [case["base"]] if case["kind"] == "run" else [(128, 64)[i % 2] for i in range(case["cases"])]
    out = []
    for b in bases:
        g = _record(b)
        out.append((np.bincount(g["level"][g["kind"] == 0]).tolist(), case["steps"], len(g["level"])))
    return out


# --------------------------------------------------------------------------
# the same in 64 bits

class _Level:
    """Neighbour lookup of one level over the rows of the cell list."""

    def __init__(self, M, l, dev):
        P = M["params"]
        rows = np.nonzero(M["level"] == l)[0]
        x, y = M["ix"][rows].astype(np.int64), M["iy"][rows].astype(np.int64)
        dummy = len(M["level"])
        self.wrap = (P["domain_nx"] << l if P["periodic_x"] else 0,
                     P["domain_ny"] << l if P["periodic_y"] else 0)
        self.x0, self.y0 = (x.min() - 3, y.min() - 3) if len(x) else (0, 0)
        w, h = (x.max() + 4 - self.x0, y.max() + 4 - self.y0) if len(x) else (1, 1)
        if self.wrap[0]:
            self.x0, w = 0, self.wrap[0]
        if self.wrap[1]:
            self.y0, h = 0, self.wrap[1]
        ids = torch.full((h, w), dummy, dtype=torch.int64, device=dev)
        self.x, self.y = (torch.from_numpy(a).to(dev) for a in (x, y))
        self.rows = torch.from_numpy(rows).to(dev)
        # periodic copies outside the domain hold no state of their own
        inside = torch.ones_like(self.rows, dtype=torch.bool)
        if self.wrap[0]:
            inside &= (self.x >= 0) & (self.x < w)
        if self.wrap[1]:
            inside &= (self.y >= 0) & (self.y < h)
        ids[(self.y - self.y0)[inside], (self.x - self.x0)[inside]] = self.rows[inside]
        self.ids, self.w, self.h = ids, w, h

    def at(self, x, y):
        x, y = x - self.x0, y - self.y0
        x = x % self.w if self.wrap[0] else x.clamp(0, self.w - 1)
        y = y % self.h if self.wrap[1] else y.clamp(0, self.h - 1)
        return self.ids[y, x]


def _limited(lim, a, b):
    """phi(b / a) a / 2: the limited half difference of both reconstructions."""
    ab = a * b
    if lim == MINMOD:
        s = 0.5 * torch.where(b.abs() < a.abs(), b, a)
    else:
        s = ab / torch.where(ab > 0, a + b, torch.ones_like(ab))
    return torch.where(ab > 0, s, torch.zeros_like(ab))


def _roe(P, area, L, R):
    """All-speed Roe flux of reconstructed states (rho, u_n, u_t, p)."""
    g, Rg, Cv, Mref = P["gama"], P["Rg"], P["Cv"], P["Ma"]
    rl, ul, tl, pl = L
    rr, ur, tr, pr = R
    Tl, Tr = pl / (rl * Rg), pr / (rr * Rg)
    el, er = Cv * Tl + 0.5 * (ul * ul + tl * tl), Cv * Tr + 0.5 * (ur * ur + tr * tr)
    hl, hr = el + pl / rl, er + pr / rr
    q = torch.sqrt(rr / rl)
    ra = torch.sqrt(rl * rr)
    ua, ta, ha = ((a + b * q) / (1 + q) for a, b in ((ul, ur), (tl, tr), (hl, hr)))
    kin = ha - 0.5 * (ua * ua + ta * ta)
    c2 = (g - 1) * kin
    c = torch.sqrt(c2)
    dp, du, dr = pr - pl, ur - ul, rr - rl
    f = (0.5 * (ul + ur)).abs() / torch.sqrt(g * Rg * 0.5 * (Tl + Tr))
    f = f.clamp(min=Mref, max=1.0)
    root = torch.sqrt(4 * c2 * f + (1 - f) ** 2 * ua * ua)
    l1, l2 = (0.5 * ((1 + f) * ua + root)).abs(), (0.5 * ((1 + f) * ua - root)).abs()
    a0 = area * ua.abs() * (dr - dp / c2)
    a1 = area / (2 * c2) * l1 * (dp + ra * c * du)
    a2 = area / (2 * c2) * l2 * (dp - ra * c * du)
    a3, a4, at = a0 + a1 + a2, c * (a1 - a2), area * ua.abs() * ra * (tr - tl)
    h = 0.5 * area
    return (h * (rl * ul + rr * ur) - a3,
            h * (rl * ul * ul + pl + rr * ur * ur + pr) - (ua * a3 + a4),
            h * (rl * ul * tl + rr * ur * tr) - (ta * a3 + at),
            h * ((pl + el * rl) * ul + (pr + er * rr) * ur)
            - (ha * a3 + ua * a4 + ta * at - kin * a0))


class _Reference:
    """The explicit step on the list form of a mesh, in 64 bits."""

    def __init__(self, M):
        self.M, self.P = M, M["params"]
        dev = self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        P = self.P
        self.lim = MINMOD if P["limiter"] == _pkg().ibgpu.LIM_MINMOD else VANLEER
        self.N = len(M["level"])
        fl = torch.from_numpy(np.append(M["flags"], 0).astype(np.int64)).to(dev)
        prim = torch.from_numpy(M["prim"]).to(dev)
        z = torch.zeros(1, 7, dtype=torch.float64, device=dev)
        prim = torch.cat([prim, z])
        # rho u v p e T per row, one absent row at the end
        self.Q = [prim[:, k].clone() for k in (0, 1, 2, 4, 6, 5)]
        self.levels = [_Level(M, l, dev) for l in range(P["nlevels"])]
        self.fl = fl
        self.lists = [self._faces(l) for l in range(P["nlevels"])]
        self.waves = self._waves() if "bc" in M else None
        self.pairs = {}
        for name in ("res", "pro"):
            t = torch.from_numpy(np.asarray(M.get(name, np.zeros((0, 11))), np.int64)).to(dev)
            for l in range(P["nlevels"] - 1):
                p = t[t[:, 0] == l]
                C, F = self.levels[l], self.levels[l + 1]
                nb = [C.at(p[:, 1] + dx, p[:, 2] + dy)
                      for dx, dy in ((0, 0), (-1, 0), (1, 0), (0, -1), (0, 1))]
                self.pairs[name, l] = nb, [F.at(p[:, 3 + 2 * k], p[:, 4 + 2 * k]) for k in range(4)]
        if "ib" in M and len(M["ib"]):
            B = self.levels[-1]
            t = torch.from_numpy(np.asarray(M["ib"], np.int64)).to(dev)
            self.ib = (B.at(t[:, 0], t[:, 1]),
                       [B.at(t[:, 2 + 2 * k], t[:, 3 + 2 * k]) for k in range(8)],
                       torch.from_numpy(np.asarray(M["ib_f"], np.float64)).to(dev))
        else:
            self.ib = None

    def _faces(self, l):
        L, fl = self.levels[l], self.fl
        normal = L.rows[(fl[L.rows] & 2) != 0]
        sides = []
        for dx, dy in ((1, 0), (0, 1)):
            at = [L.at(L.x + k * dx, L.y + k * dy) for k in (-2, -1, 0, 1)]
            ok = (at[1] != self.N) & (at[2] != self.N) & (((fl[at[1]] | fl[at[2]]) & 2) != 0)
            ok &= L.rows == at[2]
            l2, l1, r1, r2 = (a[ok] for a in at)
            m2, p2 = l2 != self.N, r2 != self.N
            far_l, far_r = torch.where(m2, l2, r2), torch.where(p2, r2, l2)
            # tangential neighbours of both cells, for the viscous flux
            X, Y = L.x[ok], L.y[ok]
            tang = [L.at(X + a * dx + s * dy, Y + a * dy + s * dx) for s in (1, -1) for a in (-1, 0)]
            # the face on the high side of each normal cell, by its high cell
            sel = (fl[L.rows] & 2) != 0
            hi = L.at(L.x[sel] + dx, L.y[sel] + dy)
            sides.append((far_l, l1, r1, far_r, tang, hi))
        return normal, sides

    def _waves(self):
        """The boundary list in groups that keep the sequential order's results."""
        M, g = self.M, self.M["bc"]
        out = []
        for l in range(self.P["nlevels"]):
            rows = np.nonzero((g[:, 0] == l) & (g[:, 6] != -99) & (g[:, 6] != -125))[0]
            G = self.levels[l].at(*(torch.from_numpy(g[rows, k].astype(np.int64)).to(self.dev) for k in (1, 2))).tolist()
            R = self.levels[l].at(*(torch.from_numpy(g[rows, k].astype(np.int64)).to(self.dev) for k in (3, 4))).tolist()
            wrote, read, wave = {}, {}, []
            for a, b in zip(G, R):
                w = max(wrote.get(b, -1) + 1, read.get(a, -1) + 1, wrote.get(a, -1) + 1)
                wave.append(w)
                wrote[a] = w
                read[b] = max(read.get(b, -1), w)
            wave = np.array(wave, int)
            groups = []
            for w in range(wave.max() + 1 if len(wave) else 0):
                for t in np.unique(g[rows, 6]):
                    for f in np.unique(g[rows, 5]):
                        m = np.nonzero((wave == w) & (g[rows, 6] == t) & (g[rows, 5] == f))[0]
                        if len(m):
                            groups.append((w, int(t), int(f), torch.tensor([G[i] for i in m], device=self.dev),
                                           torch.tensor([R[i] for i in m], device=self.dev)))
            out.append(groups)
        return out

    def _recover(self, rho, u, v, e):
        p = (e - 0.5 * (u * u + v * v)) * (self.P["gama"] - 1) * rho
        return [rho, u, v, p, e, p / (rho * self.P["Rg"])]

    def _store(self, Q, rows, new):
        for q, x in zip(Q, new):
            q[rows] = x

    def _exchange(self, ts):
        P, Q = self.P, self.Q
        for l in range(P["nlevels"] - 1):
            (c, *_), sons = self.pairs["res", l]
            if len(c) and ts % P["average_step"][l + 1] == P["average_left"][l + 1]:
                rho = sum(Q[0][s] for s in sons)
                u, v, e = (sum(Q[k][s] * Q[0][s] for s in sons) / rho for k in (1, 2, 4))
                self._store(Q, c, self._recover(0.25 * rho, u, v, e))
        for l in range(P["nlevels"] - 1):
            nb, sons = self.pairs["pro", l]
            if len(nb[0]) and ts % P["prolong_step"][l + 1] == P["prolong_left"][l + 1]:
                U = [[Q[0][s]] + [Q[0][s] * Q[k][s] for k in (1, 2, 4)] for s in nb]
                for k, s in enumerate(sons):
                    a, b = (-0.25, 0.25)[k // 2], (-0.25, 0.25)[k % 2]
                    f = [U[0][c] + a * 0.5 * (U[2][c] - U[1][c]) + b * 0.5 * (U[4][c] - U[3][c])
                         for c in range(4)]
                    self._store(Q, s, self._recover(f[0], f[1] / f[0], f[2] / f[0], f[3] / f[0]))

    def _image(self, cells, w):
        return [sum(w[:, k] * self.Q[f][cells[k]] for k in range(8)) for f in (5, 3, 1, 2)]

    def _body(self):
        P = self.P
        row, cells, f = self.ib
        T, p, hu, hv = self._image(cells, f[:, 2:10])
        sd, hg, wall = f[:, 0], f[:, 1], f[:, 13:16]
        r0 = torch.where(sd < 0, torch.full_like(sd, -1.0), sd / (sd + hg))
        u, v, w = (torch.where(sd < 0, 2 * wall[:, k] - h, wall[:, k] + (h - wall[:, k]) * r0)
                   for k, h in enumerate((hu, hv, torch.zeros_like(hu))))
        e = P["Cv"] * T + 0.5 * (u * u + v * v + w * w)
        self._store(self.Q, row, [p / (P["Rg"] * T), u, v, p, e, T])

    def _boundaries(self, l):
        P, Q = self.P, self.Q
        fv = self.M["facevar"]
        back, angle = self.M["bc_scalars"]
        for _, kind, face, ghost, ref in sorted(self.waves[l], key=lambda t: t[0]):
            rho, u, v, p, e, T = (q[ref] for q in Q)
            if kind == -12:
                p = torch.full_like(p, float(fv[face][4] + back))
                rho = p / (P["Rg"] * T)
            elif kind == -13:
                speed = torch.sqrt(u * u + v * v)
                u, v = speed * math.cos(angle), speed * math.sin(angle)
                T = float(fv[face][5]) - 0.5 * (u * u + v * v) / P["Cp"]
                p = float(fv[face][4]) * (T / float(fv[face][5])) ** 3.5
                rho = p / (P["Rg"] * T)
                e = P["Cv"] * T + 0.5 * (u * u + v * v)
            elif kind != -50:
                raise ValueError("boundary type %d" % kind)
            self._store(Q, ghost, [rho, u, v, p, e, T])

    def _geometry(self, l):
        dx, dy, dz = self.P["dh"][l]
        return dx, dy, dz, (dy * dz, dz * dx)

    def _viscous(self, l):
        P = self.P
        u, v, T = self.Q[1], self.Q[2], self.Q[5]
        dx, dy, _, areas = self._geometry(l)
        out = []
        for d, (_, a, b, _, (ua, ub, da, db), _) in enumerate(self.lists[l][1]):
            n = [q[b] - q[a] for q in (u, v, T)]
            t = [0.25 * (q[ua] + q[ub] - q[da] - q[db]) for q in (u, v, T)]
            X, Y = (n, t) if d == 0 else (t, n)
            ux, vx, Tx = (q / dx for q in X)
            uy, vy, Ty = (q / dy for q in Y)
            Tm = 0.5 * (T[a] + T[b])
            mu = Tm ** 1.5 * (1 + P["s_over_t"]) / (Tm + P["s_over_t"])
            div = (ux + vy) / 3
            txx, tyy = 2 * mu * (ux - div) / P["Re"], 2 * mu * (vy - div) / P["Re"]
            txy = mu / P["Re"] * (uy + vx)
            um, vm, k = 0.5 * (u[a] + u[b]), 0.5 * (v[a] + v[b]), P["qk"] * mu
            tn = (txx, txy, um * txx + vm * txy + k * Tx) if d == 0 else \
                (txy, tyy, um * txy + vm * tyy + k * Ty)
            F = torch.zeros(3, self.N + 1, dtype=torch.float64, device=self.dev)
            for c in range(3):
                F[c, b] = areas[d] * tn[c]
            out.append(F)
        normal, sides = self.lists[l]
        return [sum(F[c, s[5]] - F[c, normal] for F, s in zip(out, sides)) for c in range(3)]

    def _residual(self, l, W):
        P = self.P
        areas = self._geometry(l)[3]
        normal, sides = self.lists[l]
        res = 0
        for d, (l2, l1, r1, r2, _, hi) in enumerate(sides):
            order = (0, 1, 2, 3) if d == 0 else (0, 2, 1, 3)
            S = []
            for k in order:
                a, b, c, e = (W[k][i] for i in (l2, l1, r1, r2))
                S.append((b + _limited(self.lim, b - a, c - b), c - _limited(self.lim, c - b, e - c)))
            f = _roe(P, areas[d], [s[0] for s in S], [s[1] for s in S])
            F = torch.zeros(4, self.N + 1, dtype=torch.float64, device=self.dev)
            for c, k in enumerate(order):
                F[k, r1] = f[c]
            res = res + (F[:, normal] - F[:, hi])
        return res

    def step(self, ts, dt):
        P, Q = self.P, self.Q
        self._exchange(ts)
        if self.ib:
            self._body()
        if ts % P["dt_var_step"] == 0:
            best = 1e4
            for l in range(P["nlevels"]):
                dx, dy, dz, (ax, ay) = self._geometry(l)
                n = self.lists[l][0]
                if len(n):
                    c = torch.sqrt(P["gama"] * P["Rg"] * Q[5][n])
                    b = P["cfl"] * dx * dy * dz / ((Q[1][n].abs() + c) * ax + (Q[2][n].abs() + c) * ay + c * dx * dy)
                    best = min(best, float(b.min()))
            dt = min(best, dt * P["dt_ratio"])
        on = [l for l in range(P["nlevels"]) if ts % P["march_step"][l] == P["march_left"][l]]
        for l in on if self.waves else ():
            self._boundaries(l)
        norm = torch.zeros(4, dtype=torch.float64, device=self.dev)
        for l in on:
            normal = self.lists[l][0]
            if not len(normal):
                continue
            vis = self._viscous(l) if P["viscous"] else None
            f = self.fl[normal]
            upd = ((f & 4) != 0) & ((f & 8) != 0)
            wr, reset = normal[upd], normal[((f & 16) != 0) & ~upd]
            U = [Q[0][wr]] + [Q[0][wr] * Q[k][wr] for k in (1, 2, 4)]
            dx, dy, dz, _ = self._geometry(l)
            W = [q.clone() for q in Q[:4]]
            for tp in P["tp"]:
                res = self._residual(l, W)
                for c in range(3) if vis else ():
                    res[c + 1] += vis[c]
                cv = [U[c] + res[c][upd] * (tp * dt * P["step_num"][l]) / (dx * dy * dz) for c in range(4)]
                new = self._recover(cv[0], cv[1] / cv[0], cv[2] / cv[0], cv[3] / cv[0])
                self._store(W, wr, new[:4])
                init = P["initvar"]
                self._store(W, reset, [init[0], init[1], init[2], init[4]])
            self._store(Q, wr, new)
            self._store(Q, reset, [init[k] for k in (0, 1, 2, 4, 6, 5)])
            counted = (f & 32) != 0
            if counted.any():
                norm = torch.maximum(norm, res[:, counted].abs().max(1).values)
        self.norm = norm
        return dt

    def rows(self, compact):
        q = [x[:self.N] for x in self.Q]
        if compact:
            return torch.stack(q[:4], 1)
        return torch.stack([q[0], q[1], q[2], torch.zeros_like(q[0]), q[3], q[5], q[4]], 1)

    def forces(self):
        M, P = self.M, self.P
        B = self.levels[-1]
        t = torch.from_numpy(np.asarray(M["patch"], np.int64)).to(self.dev)
        f = torch.from_numpy(np.asarray(M["patch_f"], np.float64)).to(self.dev)
        _, p, hu, hv = self._image([B.at(t[:, 1 + 2 * k], t[:, 2 + 2 * k]) for k in range(8)], f[:, 8:16])
        pc, nv, area, hg, pv = f[:, :3], f[:, 3:6], f[:, 6:7], f[:, 7:8], f[:, 16:19]
        arm = pc - torch.from_numpy(np.asarray(M["body_center"])).to(self.dev)[t[:, 0]]
        du = torch.stack([hu, hv, torch.zeros_like(hu)], 1) - pv
        shear = (du - nv * (du * nv).sum(1, keepdim=True)) / hg * P["mu"] * area * P["shear_ref"]
        push = -p[:, None] * area * nv * P["p_ref"]
        force = (push + shear) * P["area_ref"]
        both = torch.cat([force, torch.cross(arm, force, dim=1) * P["L_ref"]], 1)
        return torch.zeros(len(M["body_center"]), 6, dtype=torch.float64, device=self.dev).index_add(0, t[:, 0], both)


def _exact_flow(M, steps, compact):
    R = _Reference(M)
    dt = 1.0
    for ts in range(steps):
        dt = R.step(ts, dt)
    n = [float(x) for x in R.norm]
    got = dict(rows=R.rows(compact).cpu(), dt=dt, res=np.array([n[0], n[1], n[2], 0.0, n[3]]))
    if "bc" in M:
        got["forces"] = R.forces().cpu().numpy()
    return got


def _exact_network(case, seed):
    P, X, y, m, v = _network(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    P = P.double().to(dev).requires_grad_()
    X = X.to(dev)
    W = torch.split(P, [64 * 112, 64, 64 * 64, 64, 3 * 64, 3])

    def logits(rows):
        h = torch.nn.functional.gelu(rows.double() @ W[0].view(64, 112).T + W[1], approximate="tanh")
        h = torch.nn.functional.gelu(h @ W[2].view(64, 64).T + W[3], approximate="tanh")
        return h @ W[4].view(3, 64).T + W[5]

    z = logits(X)
    if case["kind"] == "forward":
        return dict(cls=None, logits=z.detach().cpu())
    y = y.to(dev).long()
    w = torch.tensor(WEIGHTS, dtype=torch.float32).double().to(dev)[y]
    loss = (w * torch.nn.functional.cross_entropy(z, y, reduction="none")).mean()
    loss.backward()
    g = P.grad.cpu()
    m, v, k, lr = m.double(), v.double(), 61, float(np.float32(3e-3))
    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
    step = lr * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
    return dict(grad=g, params=P.detach().cpu() - step, m=m, v=v,
                stats=torch.tensor([float(loss), float((z.argmax(1) == y).sum())], dtype=torch.float64))


def exact(case, seed):
    kind = case["kind"]
    if kind == "tag":
        return None  # tag bits only
    if kind in ("train", "forward"):
        return _exact_network(case, seed)
    if kind == "step":
        return _exact_flow(_vortex(case, seed, case["nx"], case["ny"]), 1, False)
    if kind == "coupled":
        return _exact_flow(_meshes(case, seed)[0], 1, True)
    if kind == "run":
        return _exact_flow(_meshes(case, seed)[0], case["steps"], case["mesh"] == "vortex")
    each = [_exact_flow(M, case["steps"], False) for M in _meshes(case, seed)]
    return dict(rows=[e["rows"] for e in each], forces=[e["forces"] for e in each],
                dt=[e["dt"] for e in each])

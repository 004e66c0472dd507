"""Performance cases of the reconstruction library: the calls a program makes,
over the sizes, shapes and options it makes them with.

Particle sets come from the seeded generators of
particleisosurface_gb300.synth (the benchmark's own workloads).  A case is a
dict with a "kind":

  mesh    particles in pinned host memory -> mesh in pinned host memory,
          through pi_reconstruct (the one call of a frame), with a context
          that the program keeps from frame to frame
  varr    the same with per-particle radii, through a frame's stages
  field   the particle state of a new frame (hash grid, anisotropy, normals)
          and the field with its gradient at host points
  grid    the particle state of a new frame and the uniform lattice of field
          values, left on the device
  serve   a burst of frames through the request loop
"""
import ctypes as C
import json
import math

import numpy as np
import torch

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import synth


def listed():
    return [
        # one droplet: the smallest call, where launches and host round trips count
        {"name": "ball_2k", "kind": "mesh", "shape": "ball", "n": 2000, "radius": 0.025, "qef": False, "splash": False},
        # the plain single frame of the CPU-runnable configuration
        {"name": "slab_20k", "kind": "mesh", "shape": "slab", "n": 20000, "radius": 0.025, "qef": False, "splash": False},
        # an ordinary frame of the batched and served streams, of an odd size
        {"name": "mixed_151k", "kind": "mesh", "shape": "mixed", "n": 151237, "radius": 0.01, "qef": False, "splash": False},
        # the 1M dam-break frame on the reference's active path
        {"name": "dam_1m", "kind": "mesh", "shape": "dam", "n": 1000000, "radius": 0.01, "qef": False, "splash": False},
        # the headline frame: the same with a QEF vertex per leaf
        {"name": "dam_1m_qef", "kind": "mesh", "shape": "dam", "n": 1000000, "radius": 0.01, "qef": True, "splash": False},
        # thin sheets and filaments with the QEF: degenerate neighbourhoods
        {"name": "sheets_500k_qef", "kind": "mesh", "shape": "sheets", "n": 500000, "radius": 0.01, "qef": True,
         "splash": False},
        # a large frame of the batched stream
        {"name": "mixed_1700k", "kind": "mesh", "shape": "mixed", "n": 1700003, "radius": 0.01, "qef": False,
         "splash": False},
        # spray above a slab, loose particles written as icosahedra
        {"name": "spray_60k_splash", "kind": "mesh", "shape": "spray", "n": 60001, "radius": 0.02, "qef": False,
         "splash": True},
        # particles of two sizes: the variable-radius path
        {"name": "two_radius_50k", "kind": "varr", "n": 50000},
        # Evaluator use: field and gradient at points around a new frame's particles
        {"name": "field_200k", "kind": "field", "shape": "dam", "n": 200000, "radius": 0.01, "m": 300007, "grad": True},
        # dense-grid mode on a new frame
        {"name": "grid_150k", "kind": "grid", "shape": "dam", "n": 150000, "radius": 0.01},
        # continuous batching: a burst of frames of mixed sizes on 8 slots
        {"name": "serve_10", "kind": "serve", "count": 10, "n_min": 20000, "n_max": 300000, "radius": 0.01, "slots": 8},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesh"] * 6 + ["varr", "field", "grid", "serve"])
    if kind == "mesh":
        shape = rng.choice(["ball", "slab", "mixed", "dam", "sheets", "spray"])
        qef = rng.random() < 0.4
        top = {"ball": 60000, "slab": 250000, "mixed": 1500000, "dam": 1400000, "sheets": 500000, "spray": 200000}[shape]
        return {"kind": "mesh", "shape": shape, "n": _logint(rng, 2000, min(top, 800000) if qef else top),
                "radius": rng.choice([0.005, 0.01, 0.02, 0.025]), "qef": qef,
                "splash": shape == "spray" and rng.random() < 0.7}
    if kind == "varr":
        return {"kind": "varr", "n": _logint(rng, 4000, 150000)}
    if kind == "field":
        return {"kind": "field", "shape": rng.choice(["dam", "slab", "mixed", "sheets"]), "n": _logint(rng, 5000, 200000),
                "radius": rng.choice([0.005, 0.01, 0.02]), "m": _logint(rng, 1000, 500000), "grad": rng.random() < 0.5}
    if kind == "grid":
        return {"kind": "grid", "shape": rng.choice(["dam", "slab"]), "n": _logint(rng, 5000, 200000),
                "radius": rng.choice([0.005, 0.01, 0.02])}
    return {"kind": "serve", "count": rng.randint(3, 12), "n_min": 10000, "n_max": _logint(rng, 30000, 300000),
            "radius": rng.choice([0.005, 0.01, 0.02]), "slots": rng.choice([2, 4, 8])}


_SHAPES = {"ball": synth.small_blob, "slab": synth.slab_and_sphere, "dam": synth.dam_break, "spray": synth.spray_frame,
           "sheets": synth.sheets_and_filaments}


def _particles(shape, n, radius, seed):
    if shape == "mixed":
        return synth.mixed_frame(seed, n, radius).xyz
    return _SHAPES[shape](n=n, radius=radius, seed=seed).xyz


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


# What a program keeps for all its frames: one context (or request loop) per
# case, as a process that reconstructs a stream of frames has it.
_kept = {}


def _keep(case, make):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


# Room for mesh vertices of n particles: at most 60 a particle (loose ones),
# else a surface part and one that grows with n; a program of this kind allots
# twice as many triangles.
_ROOM = {"ball": 6, "slab": 13, "mixed": 3, "dam": 4, "sheets": 6, "spray": 9, "two_radius": 3}


def _room(shape, n):
    """Pinned host buffers for the mesh of n particles, filled up to the
    counts a pass returns."""
    nv = min(60 * n, 600000 + _ROOM[shape] * n)
    return {"verts": torch.zeros((nv, 3), dtype=torch.float32).pin_memory(),
            "tris": torch.zeros((int(2.1 * nv), 3), dtype=torch.int32).pin_memory()}


def _serve_sizes(case):
    k = case["count"]
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [int(math.exp(lo + (hi - lo) * (i + 0.5) / k)) | 1 for i in range(k)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        kept = _keep(case, lambda: {"ctx": N.Context(0)})
        return dict(_room(case["shape"], case["n"]), kind=kind, ctx=kept["ctx"],
                    xyz=_pinned(_particles(case["shape"], case["n"], case["radius"], seed)),
                    params=N.default_params(case["radius"], qef=case["qef"], splash=case["splash"]))
    if kind == "varr":
        kept = _keep(case, lambda: {"ctx": N.Context(0)})
        fr = synth.two_radius_frame(n=case["n"], seed=seed)
        return dict(_room("two_radius", case["n"]), kind=kind, frame=N.Frame(kept["ctx"], N.default_params(fr.radius)),
                    xyz=_pinned(fr.xyz), radii=fr.radii)
    if kind == "field":
        kept = _keep(case, lambda: {"ctx": N.Context(0)})
        xyz = _particles(case["shape"], case["n"], case["radius"], seed)
        return {"kind": kind, "frame": N.Frame(kept["ctx"], N.default_params(case["radius"])), "xyz": _pinned(xyz),
                "pts": _pinned(_points(case, xyz, seed)), "grad": case["grad"]}
    if kind == "grid":
        kept = _keep(case, lambda: {"ctx": N.Context(0)})
        frame = N.Frame(kept["ctx"], N.default_params(case["radius"]))
        xyz = _pinned(_particles(case["shape"], case["n"], case["radius"], seed))
        return {"kind": kind, "frame": frame, "xyz": xyz,
                "values": torch.zeros(_lattice_room(case), dtype=torch.float32, device="cuda")}
    kept = _keep(case, lambda: {"server": N.Server(0, slots=case["slots"])})
    frames = [synth.mixed_frame(seed * 64 + i, n, case["radius"]).xyz for i, n in enumerate(_serve_sizes(case))]
    return {"kind": kind, "server": kept["server"], "frames": frames, "params": N.default_params(case["radius"]),
            "rooms": [_room("mixed", len(x)) for x in frames]}


def _lattice_room(case):
    """Values a program of this kind makes room for: the lattice's extent
    follows the particles, about 64 points each, more where they are few."""
    return 100 * case["n"] + 400000


def _points(case, xyz, seed):
    """Points around the particles, within a few radii of them."""
    rng = np.random.default_rng(seed + 1)
    at = xyz[rng.integers(0, len(xyz), case["m"])]
    return (at + rng.normal(0.0, 2.0 * case["radius"], at.shape)).astype(np.float32)


def _float_ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def _int_ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_int32))


def _mesh(nv, nt, room):
    return {"counts": np.array([nv.value, nt.value]), "verts": room["verts"], "tris": room["tris"]}


def _checked(nv, nt, room):
    if nv.value > len(room["verts"]) or nt.value > len(room["tris"]):
        raise RuntimeError("mesh buffers too small")


def run(state):
    kind, lib = state["kind"], N.lib()
    nv, nt = C.c_int64(), C.c_int64()
    if kind == "mesh":
        v, t, xyz = state["verts"], state["tris"], state["xyz"]
        N.check(lib.pi_reconstruct(state["ctx"].h, C.byref(state["params"]), _float_ptr(xyz), len(xyz), _float_ptr(v),
                                   len(v), _int_ptr(t), len(t), C.byref(nv), C.byref(nt)))
        return _mesh(nv, nt, state)
    if kind == "varr":
        f = state["frame"].upload(state["xyz"].numpy()).upload_radii(state["radii"]).run()
        N.check(lib.pi_mesh_counts(f.h, C.byref(nv), C.byref(nt)))
        _checked(nv, nt, state)
        N.check(lib.pi_mesh_get(f.h, _float_ptr(state["verts"]), _int_ptr(state["tris"]), None))
        return _mesh(nv, nt, state)
    if kind == "field":
        f = state["frame"].upload(state["xyz"].numpy()).hashgrid().aniso().normals()
        r = f.eval(state["pts"].numpy(), grad=state["grad"])
        return {"value": r[0], "grad": r[1]} if state["grad"] else {"value": r}
    if kind == "grid":
        f = state["frame"].upload(state["xyz"].numpy()).hashgrid().aniso().normals()
        f.grid_sample_device(state["values"].data_ptr(), state["values"].numel())
        return {"values": state["values"]}
    srv, out = state["server"], []
    tickets = [srv.submit(x, state["params"]) for x in state["frames"]]
    ms, wait = C.c_double(), C.c_double()
    for k, room in zip(tickets, state["rooms"]):
        N.check(lib.pi_server_wait(srv.h, k, C.byref(nv), C.byref(nt), C.byref(ms), C.byref(wait)))
        _checked(nv, nt, room)
        N.check(lib.pi_server_fetch(srv.h, k, _float_ptr(room["verts"]), _int_ptr(room["tris"])))
        out.append(_mesh(nv, nt, room))
    return out


# Distinct field evaluations and mesh vertices per particle of each shape at
# the listed sizes (the library's own frame counters, rounded), leaves per
# evaluation with the QEF, and the particles whose kernel reaches a point: the
# operations a frame cannot do without follow from them.
_EVALS = {"ball": 31, "slab": 72, "mixed": 7, "dam": 18, "sheets": 12, "spray": 32, "two_radius": 30}
_EVALS_QEF = {"ball": 90, "slab": 250, "mixed": 22, "dam": 66, "sheets": 42, "spray": 100}
_VERTS = {"ball": 2.5, "slab": 9.9, "mixed": 0.7, "dam": 2.2, "sheets": 1.8, "spray": 3.6, "two_radius": 0.7}
_REACH = 18  # particles whose kernel reaches a point
_PAIR = 38   # operations of one particle's kernel at one point
_LEAF = 960  # operations of one leaf's QEF


def work(case):
    kind = case["kind"]
    if kind == "serve":
        parts = [work({"kind": "mesh", "shape": "mixed", "n": n, "qef": False}) for n in _serve_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["n"]
    state = n * 2 * 40 * 36  # smoothed centre and covariance over about 40 neighbours, twice
    if kind in ("mesh", "varr"):
        shape = case.get("shape", "two_radius")
        evals = n * (_EVALS_QEF if case.get("qef") else _EVALS)[shape]
        solve = evals / 15 * _LEAF if case.get("qef") else 0
        nv = n * _VERTS[shape]
        return {"bytes": 12 * n + 12 * nv + 24 * nv, "flops": state + evals * _REACH * _PAIR + solve}
    if kind == "field":
        m = case["m"]
        return {"bytes": 12 * n + 12 * m + (16 if case["grad"] else 4) * m, "flops": state + m * _REACH * _PAIR}
    points = n * 64
    return {"bytes": 12 * n + 4 * points, "flops": state + n * 8 * _REACH * _PAIR}


# ---------------------------------------------------------------------------
# The field in 64 bits: the reference's formulas over the 27-cell candidate
# lists of the float hash grid, written with torch alone.
# ---------------------------------------------------------------------------
def _cells(xyz, r):
    """The hash grid over the particles: its origin, cell and size (float32
    arithmetic, as the grid is defined), and a table [cells + 1, cap] of the
    particles of each cell (n where empty; the last row is an empty cell)."""
    f = np.float32
    cell = f(r) * f(4)
    lo, size = [], []
    for a in range(3):
        mn, mx = xyz[:, a].min(), xyz[:, a].max()
        length = np.ceil((mx - mn) / cell) * cell
        centre = (mn + mx) / f(2)
        lo.append(centre - length / f(2))
        size.append(max(int(np.ceil(((centre + length / f(2)) - lo[a]) / cell)), 1))
    grid = (np.array(lo, f), cell, size)
    key = _keys(grid, xyz)
    if (key < 0).any():
        return grid, None
    order = np.argsort(key, kind="stable")
    skey = key[order]
    first = np.searchsorted(skey, skey, side="left")
    place = np.arange(len(xyz)) - first
    table = np.full((size[0] * size[1] * size[2] + 1, int(place.max()) + 1), len(xyz), np.int32)
    table[skey, place] = order
    return grid, torch.from_numpy(table).cuda()


def _coords(grid, pts):
    lo, cell, _ = grid
    return ((pts - lo) / cell).astype(np.int64)  # truncation toward zero


def _keys(grid, pts):
    c, size = _coords(grid, pts), grid[2]
    ok = np.all((c >= 0) & (c < np.array(size)), axis=1)
    return np.where(ok, (c[:, 2] * size[1] + c[:, 1]) * size[0] + c[:, 0], -1)


def _candidates(grid, table, pts):
    """Chunks (slice of the points, [m, 27 cap] particle indices, n = none)."""
    size = grid[2]
    c = torch.from_numpy(_coords(grid, pts)).cuda()
    cap = table.shape[1]
    step = max(1, (1 << 24) // (27 * cap))
    for s in range(0, len(pts), step):
        cc = c[s:s + step]
        rows = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    x, y, z = cc[:, 0] + dx, cc[:, 1] + dy, cc[:, 2] + dz
                    ok = (x >= 0) & (x < size[0]) & (y >= 0) & (y < size[1]) & (z >= 0) & (z < size[2])
                    rows.append(torch.where(ok, (z * size[1] + y) * size[0] + x, table.shape[0] - 1))
        yield slice(s, s + cc.shape[0]), table[torch.stack(rows, 1)].reshape(cc.shape[0], 27 * cap).long()


def _weight(d, h):
    t = h - d
    return torch.where(d < h / 2, 1 - 6 * d * d * t / h ** 3, 2 * t ** 3 / h ** 3) * (d < h)


def _state64(xyz, r):
    """Smoothed centres, G and det of every particle; None where a particle
    lies outside the hash grid."""
    grid, table = _cells(xyz, r)
    if table is None:
        return None
    n, r = len(xyz), float(np.float32(r))
    none = torch.full((1, 3), 1e30, dtype=torch.float64, device="cuda")
    p = torch.from_numpy(xyz).cuda().double()
    pp = torch.cat([p, none])
    mean = torch.empty_like(p)
    index = torch.arange(n, device="cuda")
    for s, cand in _candidates(grid, table, xyz):
        d = pp[cand] - p[s][:, None]
        w = _weight(d.norm(dim=2), 4 * r) * (cand != index[s][:, None])
        ws = w.sum(1, keepdim=True)
        off = (w[:, :, None] * torch.where(w[:, :, None] > 0, d, 0.0)).sum(1) / ws
        use = ((cand < n).sum(1, keepdim=True) > 2) & (ws > 0)
        mean[s] = p[s] + torch.where(use, float(np.float32(0.9)) * off, 0.0)
    mm = torch.cat([mean, none])
    cov = torch.empty((n, 3, 3), dtype=torch.float64, device="cuda")
    for s, cand in _candidates(grid, table, xyz):
        d = mm[cand] - mean[s][:, None]
        w = _weight(d.norm(dim=2), 4 * r)
        d = torch.where(w[:, :, None] > 0, d, 0.0)
        cov[s] = ((d * w[:, :, None]).transpose(1, 2) @ d + torch.eye(3, device="cuda", dtype=torch.float64) *
                  (2 * r) ** 2) / w.sum(1)[:, None, None]
    w, v = np.linalg.eigh(cov.cpu().numpy())
    w = np.maximum(w, w.max(1, keepdims=True) / 4)
    scale = np.cbrt(w.prod(1))[:, None] / w
    g = np.einsum("nik,nk,njk->nij", v, scale, v)
    return grid, table, mm, torch.from_numpy(g).cuda(), torch.from_numpy(scale.prod(1)).cuda()


def _field64(case, xyz, pts, grad):
    got = _state64(xyz, case["radius"])
    if got is None:
        return None
    grid, table, mm, g, det = got
    h = 2 * float(np.float32(case["radius"]))
    sigma = h ** -6
    a = torch.cat([g / h, torch.zeros_like(g[:1])])
    wd = torch.cat([det * sigma, torch.zeros_like(det[:1])])
    q = 0.01
    iso = sigma * (1 - 1.5 * q * q + 0.75 * q ** 3)
    value = torch.empty(len(pts), dtype=torch.float64, device="cuda")
    slope = torch.empty((len(pts), 3), dtype=torch.float64, device="cuda") if grad else None
    for s, cand in _candidates(grid, table, pts):
        at = torch.from_numpy(pts[s]).cuda().double()
        d = torch.where((cand < len(xyz))[:, :, None], at[:, None] - mm[cand], 1e3 * h)
        u = (a[cand] @ d[..., None])[..., 0]
        q = u.norm(dim=2)
        k = torch.where(q <= 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q) ** 3) * (q < 2)
        value[s] = iso - (wd[cand] * k).sum(1)
        if grad:
            t = wd[cand] * (1 - q * q) ** 2 * (q < 1)
            slope[s] = -6 * h ** 5 * (t[:, :, None] * u).sum(1)
    return value, slope


def exact(case, seed):
    # a mesh follows from comparisons of float values: it has no 64-bit counterpart
    if case["kind"] not in ("field", "grid"):
        return None
    xyz = _particles(case["shape"], case["n"], case["radius"], seed)
    if case["kind"] == "field":
        got = _field64(case, xyz, _points(case, xyz, seed), case["grad"])
        if got is None:
            return None
        return {"value": got[0], "grad": got[1]} if case["grad"] else {"value": got[0]}
    pts = _lattice(xyz, case["radius"])
    if len(pts) > 12_000_000:
        return None
    got = _field64(case, xyz, pts, False)
    if got is None:
        return None
    out = torch.zeros(_lattice_room(case), dtype=torch.float64, device="cuda")
    out[:len(pts)] = got[0]
    return {"values": out}


def _lattice(xyz, radius):
    """The uniform grid's points: spacing r over the particles' box grown by
    4r, coordinates in the float arithmetic that defines them."""
    f = np.float32
    r, axes = f(radius), []
    for a in range(3):
        mn, mx = xyz[:, a].min(), xyz[:, a].max()
        centre, length = (mn + mx) / f(2), mx - mn
        grown = np.ceil(length / r) * r + r * f(4)
        lo, hi = centre - grown / f(2), centre + grown / f(2)
        steps = int(grown / r)
        i = np.arange(steps + 1)
        axes.append((steps - i).astype(f) / f(steps) * lo + i.astype(f) / f(steps) * hi)
    z, y, x = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    return np.stack([x, y, z], -1).reshape(-1, 3)

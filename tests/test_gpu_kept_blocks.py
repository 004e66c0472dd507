"""Frames of changing sizes on one context reuse each other's device blocks, and
the counters of all stages come to the host in one copy: meshes and counts are the
ones a context without kept blocks (one with a budget) gives, stage by stage, with
a stage run again, and with a context per thread."""
import threading

import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

pytestmark = pytest.mark.gpu

COUNTS = ("num_invalid_keys", "num_nodes", "num_leaves", "num_dual_cells", "num_vertices", "num_triangles",
          "field_evals", "bisection_evals", "fp64_eigen", "field_evals_performed",
          "qef_accepted", "qef_singular")


def _frames(qef):
    out = []
    for n in (2000, 60000, 3000, 60000, 2500, 20000):
        s = synth.slab_and_sphere(n, seed=n)
        out.append((s.xyz, N.default_params(s.radius, qef=qef)))
    return out


def _result(f):
    v, t = f.mesh()[:2]
    info = f.info()
    return {k: info[k] for k in COUNTS}, v, t


def _run_all(ctx, frames, staged):
    got = []
    for xyz, p in frames:
        f = N.Frame(ctx, p).upload(xyz)
        if staged:
            f.hashgrid().aniso().normals().octree().octree().extract()
        else:
            f.run()
        got.append(_result(f))
        f.close()
    return got


def _same(a, b):
    for (ia, va, ta), (ib, vb, tb) in zip(a, b):
        assert ia == ib
        assert np.array_equal(va, vb) and np.array_equal(ta, tb)


@pytest.mark.parametrize("qef", [False, True])
def test_reused_blocks_change_nothing(qef):
    B.build()
    frames = _frames(qef)
    plain = N.Context(0, budget_bytes=64 << 30)
    want = _run_all(plain, frames, False)
    assert all(w[0]["num_triangles"] > 0 for w in want)
    plain.close()
    got = [None, None]

    def work(k):
        c = N.Context(0)
        _same(_run_all(c, frames, False), want)
        _same(_run_all(c, frames, True), want)
        got[k] = c.stats()
        c.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(g is not None for g in got)
    assert all(g["bytes"] == 0 for g in got)

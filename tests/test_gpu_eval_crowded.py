"""pi_eval_field at many points that share few hash cells, or have none: all in one
cell, all beyond the grid's reach on one side or on any, on the last cells that
still reach the grid, and a few or half of the points among such ones.  Values and gradients are
those of small calls, which take the points as they come, bit for bit (the sign of
a zero gradient too)."""
import ctypes as C

import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth
from test_gpu_kept_eviction import Pool

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def frame():
    B.build()
    fr = synth.dam_break(n=6000, seed=8)
    c = N.Context(0)
    f = N.Frame(c, N.default_params(fr.radius)).upload(fr.xyz).hashgrid().aniso().normals()
    yield fr, f
    f.close()
    c.close()


def _points(fr, f, kind, m):
    rng = np.random.default_rng(m)
    lo, hi = fr.xyz.min(0), fr.xyz.max(0)
    cell = 4 * fr.radius
    if kind == "one_cell":
        return fr.xyz[17] + rng.uniform(0, 0.2 * cell, (m, 3))
    if kind == "corner":
        return hi + 1.0 + rng.uniform(0, 1, (m, 3))
    if kind == "around":
        return rng.uniform(lo - 5 * (hi - lo), hi + 5 * (hi - lo), (m, 3))
    if kind == "shell":  # on both sides of where the reach ends
        p = rng.uniform(lo - 3 * cell, hi + 3 * cell, (m, 3))
        b = np.array(f.info()["bounding"])
        p[::3, 0] = b[1] + rng.choice([0.999, 1.0, 1.001, 2.0], len(p[::3])) * cell
        p[1::3, 1] = b[2] - rng.choice([0.999, 1.0, 1.001, 2.0], len(p[1::3])) * cell
        return p
    p = hi + 1.0 + rng.uniform(0, 1, (m, 3))
    if kind.startswith("half"):  # the other half scattered over the frame
        if kind == "half_one_cell":
            p = fr.xyz[17] + rng.uniform(0, 0.2 * cell, (m, 3))
        p[::2] = fr.xyz[rng.integers(0, fr.n, len(p[::2]))] + rng.normal(0, fr.radius, p[::2].shape)
        return p
    p[rng.integers(0, m, 40)] = fr.xyz[:40]
    return p


@pytest.mark.parametrize("m", [16384, 20011])
@pytest.mark.parametrize("kind", ["one_cell", "corner", "around", "shell", "few_inside", "half_outside",
                                  "half_one_cell"])
def test_values_are_those_of_small_calls(frame, kind, m):
    fr, f = frame
    p = _points(fr, f, kind, m).astype(np.float32)
    val, grad = f.eval(p, grad=True)
    parts = [f.eval(p[k:k + 4000], grad=True) for k in range(0, m, 4000)]
    assert np.array_equal(val.view(np.uint32), np.concatenate([x[0] for x in parts]).view(np.uint32))
    assert np.array_equal(grad.view(np.uint32), np.concatenate([x[1] for x in parts]).view(np.uint32))
    assert np.array_equal(val.view(np.uint32), f.eval(p).view(np.uint32))
    if kind not in ("corner", "around"):
        assert (val != np.float32(f.info()["iso_value"])).any()


def test_without_device_memory_for_the_ordering(frame):
    """Scattered points whose own arrays fit the device's memory and the ordering's
    do not are evaluated as they come."""
    fr, f = frame
    m = 16_000_000
    rng = np.random.default_rng(m)
    p = (fr.xyz[rng.integers(0, fr.n, 4000)] + rng.normal(0, fr.radius, (4000, 3))).astype(np.float32)
    want = f.eval(p)
    p = np.tile(p, (m // 4000, 1))
    assert np.array_equal(f.eval(p[:40000]), np.tile(want, 10))
    pool = Pool()
    assert pool.cu.cuCtxSynchronize() == 0 and pool.cu.cuMemPoolTrimTo(pool.pool, C.c_size_t(0)) == 0
    free, total = C.c_size_t(), C.c_size_t()
    assert pool.cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    block = C.c_uint64()
    # 16 bytes a point for its coordinates and value, 12 for its place
    assert pool.cu.cuMemAlloc_v2(C.byref(block), C.c_size_t(free.value - 16 * m - (96 << 20))) == 0
    try:
        took = pool.taken_by(lambda: np.testing.assert_array_equal(f.eval(p), np.tile(want, m // 4000)))
    finally:
        assert pool.cu.cuMemFree_v2(block) == 0
    assert 16 * m <= took < 28 * m

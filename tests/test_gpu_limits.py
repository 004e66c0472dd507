"""Frames whose sample buckets pass the range of an int: buckets by whole cells
where cell octants do not fit, coarser ones with per-particle radii, and
PI_ERR_LIMIT where the cells themselves do not, with the context usable
afterwards.  The buckets only order the evaluations, so every leaf's value stays
the point evaluation's, bit for bit."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

pytestmark = pytest.mark.gpu

INT_MAX = 2**31 - 1
T_LEAF = 2


@pytest.fixture(scope="module")
def ctx():
    B.build()
    c = N.Context(0)
    yield c
    c.close()


def _pair(xyz, shift):
    x = xyz.astype(np.float64) - xyz.mean(0)
    s = np.asarray(shift, np.float64) / 2
    return np.concatenate([x - s, x + s]).astype(np.float32)


def _leaves_are_point_values(f, qef=False):
    nodes = f.dump(N.DUMP_NODES)
    leaves = nodes[nodes["type"] == T_LEAF]
    if qef:  # a QEF vertex moves the leaf's point
        leaves = leaves[np.all(leaves["node"][:, :3] == leaves["center"], axis=1)]
    assert len(leaves) > 1000 and len(np.unique(leaves["depth"])) >= 2
    val = f.eval(np.ascontiguousarray(leaves["node"][:, :3]))
    assert np.array_equal(val.view(np.uint32), leaves["node"][:, 3].view(np.uint32))
    v, t = f.mesh()
    assert len(t) > 1000 and np.isfinite(v).all()


@pytest.mark.parametrize("qef", [False, True])
def test_octants_beyond_an_int_use_whole_cells(ctx, qef):
    fr = synth.small_blob(n=2000, seed=3)
    cell = 4 * fr.radius
    f = N.Frame(ctx, N.default_params(fr.radius, qef=qef)).upload(_pair(fr.xyz, (8000 * cell, 4000 * cell, 0))).run()
    d = [n + 4 for n in f.info()["xyz_cell_num"]]
    assert d[0] * d[1] * d[2] <= INT_MAX < 8 * d[0] * d[1] * d[2]
    _leaves_are_point_values(f, qef)
    f.close()


def test_cells_beyond_an_int_are_refused(ctx):
    r = 0.025
    rng = np.random.default_rng(7)
    x = _pair(rng.uniform(0, 3 * r, (60, 3)), (21000 * 4 * r, 21000 * 4 * r, 0))
    f = N.Frame(ctx, N.default_params(r)).upload(x).hashgrid().aniso().normals()
    d = [n + 4 for n in f.info()["xyz_cell_num"]]
    assert d[0] * d[1] * d[2] > INT_MAX
    with pytest.raises(N.PiError) as e:
        f.octree()
    assert e.value.code == N.PI_ERR_LIMIT
    f.close()
    fr = synth.small_blob(n=2000, seed=3)
    f = N.Frame(ctx, N.default_params(fr.radius)).upload(fr.xyz).run()
    _leaves_are_point_values(f)
    f.close()


def test_variable_radius_buckets_are_coarsened(ctx):
    fr = synth.two_radius_frame(n=4000, seed=6)
    rmax = float(fr.radii.max())
    x = _pair(fr.xyz, (5500 * rmax, 0, 0))
    rad = np.concatenate([fr.radii, fr.radii])
    f = N.Frame(ctx, N.default_params(float(fr.radii.min()))).upload(x).upload_radii(rad).run()
    n = int(np.ceil(2 * f.info()["root_half"] / (4 * rmax))) + 4
    assert n**3 > INT_MAX
    _leaves_are_point_values(f)
    f.close()

"""Frames whose tree is deep and thin run under the budgets that hold their nodes
and their stages' scratch: nothing is sized by what a level could hold.  The budgets are
0.2 % above the least that level-by-level growth of the nodes and sorted corners of
the leaves take."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

pytestmark = pytest.mark.gpu

R = 0.01


def _rod(length):
    """4000 particles in a rod of 4 x 4 radii, `length` radii long."""
    x = np.random.default_rng(5).uniform(0, 1, (4000, 3))
    x[:, 0] *= length * R
    x[:, 1:] *= 4 * R
    return x.astype(np.float32)


@pytest.mark.parametrize("length,depth,qef,budget", [
    (1200, 11, False, 34_700_000), (1200, 11, True, 73_370_000), (5000, 13, False, 254_300_000),
    (5000, 13, True, 258_300_000), (20000, 15, False, 95_760_000), (20000, 15, True, 140_770_000)])
def test_rod_runs_under_its_budget(length, depth, qef, budget):
    B.build()
    c = N.Context(0, budget_bytes=budget)
    f = N.Frame(c, N.default_params(R, qef=qef)).upload(_rod(length)).run()
    assert f.info()["depth_max"] == depth and f.info()["num_triangles"] > 0
    f.close()
    c.close()


def test_far_blobs_run_under_their_budget():
    """Two blobs 40000 radii apart: D_max 16, corners by sorted keys, and half of the
    budget for the hash grid's table."""
    B.build()
    b = synth.small_blob(n=3000, seed=21)
    x = b.xyz - b.xyz.mean(0)
    x = np.concatenate([x, x + np.array([40000, 0, 0]) * b.radius]).astype(np.float32)
    c = N.Context(0, budget_bytes=477_600_000)
    f = N.Frame(c, N.default_params(b.radius)).upload(x).run()
    assert f.info()["depth_max"] == 16 and f.info()["num_triangles"] > 0
    f.close()
    c.close()

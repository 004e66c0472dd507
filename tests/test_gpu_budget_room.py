"""Frames whose tree is deep and thin run under the budgets that hold their nodes
and their stages' scratch: nothing is sized by what a level could hold.  The budgets are
0.2 % above the least that level-by-level growth of the nodes and sorted corners of
the leaves take."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

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
    (5000, 13, True, 258_300_000)])
def test_rod_runs_under_its_budget(length, depth, qef, budget):
    B.build()
    c = N.Context(0, budget_bytes=budget)
    f = N.Frame(c, N.default_params(R, qef=qef)).upload(_rod(length)).run()
    assert f.info()["depth_max"] == depth and f.info()["num_triangles"] > 0
    f.close()
    c.close()

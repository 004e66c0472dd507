"""The octree levels above D_min, written from the tested paths of all of
them: against the oracle for every number of such levels the kernels take (the
deepest path level, one more, several more: the level loop goes on there), with
the tree's links and order checked node by node."""
import numpy as np
import pytest

import parity as PR
import pyoracle as O
from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

pytestmark = pytest.mark.gpu


def _clusters(gap):
    """Three jittered lattice balls of radius 5r (r = 0.01), up to `gap`
    apart: few particles in a box of about gap / r leaf cells."""
    rng = np.random.default_rng(11)
    g = np.arange(-0.05, 0.0501, 0.02)
    p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    p = p[(p ** 2).sum(1) <= 0.05 ** 2]
    at = [np.zeros(3), np.array([gap, 0.4 * gap, 0.1 * gap]), np.array([0.2 * gap, 0.9 * gap, 0.7 * gap])]
    return np.concatenate([p + rng.uniform(-0.003, 0.003, p.shape) + c for c in at]).astype(np.float32)


@pytest.fixture(scope="module")
def ctx():
    B.build()
    O.build()
    c = N.Context(0)
    yield c
    c.close()


# D_max 4 to 11, D_min = D_max - 3 (path levels 0 .. min(D_min - 1, 5))
@pytest.mark.parametrize("gap", [0.0, 0.1, 0.3, 0.8, 2.0, 4.5, 9.0, 18.0])
def test_coarse_levels_match_oracle(ctx, gap):
    xyz, r = _clusters(gap), 0.01
    o = O.OracleFrame(xyz, r).run()
    f = N.Frame(ctx, N.default_params(r)).upload(xyz).run()
    d = o.depths()
    assert (f.info()["depth_max"], f.info()["depth_min"]) == (d["depth_max"], d["depth_min"])
    n = f.dump(N.DUMP_NODES)
    rep = PR.compare_octrees(o.nodes(), n, o, o.scalars()["max_scalar"], d["depth_min"])
    # the parity rule of every octree test: a type may differ only where a
    # sampled level's sign or curvature is a tie; above D_min none may
    assert not rep["unexplained"] and rep["type_mismatch"] == rep["explained"]
    a, b = PR.node_table(o.nodes()), PR.node_table(n)
    assert {k: v[0] for k, v in a.items() if k[0] < d["depth_min"]} == \
           {k: v[0] for k, v in b.items() if k[0] < d["depth_min"]}
    # links: a parent's children are consecutive, in octant order, and name it
    par = n["first_child"] >= 0
    assert np.array_equal(par, n["type"] == 1)
    kids = n["first_child"][par][:, None] + np.arange(8)
    assert np.array_equal(n["parent"][kids], np.repeat(np.nonzero(par)[0][:, None], 8, 1))
    assert np.array_equal(n["id"][kids], n["id"][par][:, None] * np.uint64(8) + np.arange(8, dtype=np.uint64))
    assert np.array_equal(n["depth"][kids], np.repeat(n["depth"][par][:, None] + 1, 8, 1))
    # order: level after level, each in path order
    assert np.all(np.diff(n["depth"].astype(int)) >= 0)
    for k in range(d["depth_max"] + 1):
        assert np.all(np.diff(n["id"][n["depth"] == k].astype(np.int64)) > 0)
    f.close()

"""The QEF's normal equations in integers: leaves whose values are integers of
the iso value's grid, of a coarser grid of their own (dense particles), and of
neither (the FP64 sums), at radii whose field values lie near both ends of the
float range, against the FP64 NumPy solve of the same 27 samples."""
import numpy as np
import pytest

import parity as PR
from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

pytestmark = pytest.mark.gpu


def _frame(r, spacing, n, seed):
    """A jittered ball of the given spacing (in radii) in a thin slab of spacing
    2: the values' range on the ball's leaves follows its density."""
    rng = np.random.default_rng(seed)
    k = int(round(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k) * spacing] * 3, indexing="ij"), -1).reshape(-1, 3)
    ball = g[((g - g.mean(0)) ** 2).sum(1) <= (0.5 * k * spacing) ** 2]
    s = np.stack(np.meshgrid(np.arange(14) * 2.0, np.arange(3) * 2.0, np.arange(14) * 2.0, indexing="ij"), -1)
    p = np.concatenate([ball, s.reshape(-1, 3) + [0.0, -6.0, 0.0]])
    return ((p + rng.uniform(-0.25, 0.25, p.shape)) * r).astype(np.float32)


@pytest.fixture(scope="module")
def ctx():
    B.build()
    c = N.Context(0)
    yield c
    c.close()


# spacing 2: lattice density; 1: eight times that; 0.6: 37 times
@pytest.mark.parametrize("r", [2.5e-6, 0.01, 3.0e5])
@pytest.mark.parametrize("spacing", [2.0, 1.0, 0.6])
def test_vertices_match_fp64_solve(ctx, r, spacing):
    f = N.Frame(ctx, N.default_params(r, qef=True)).upload(_frame(r, spacing, 1500, int(spacing * 10))).run()
    nodes, samp, info = f.dump(N.DUMP_NODES), f.dump(N.DUMP_QEF_SAMPLES), f.info()
    leaves = np.nonzero(nodes["type"] == 2)[0]
    # the property the integers rest on
    iso = np.float32(info["iso_value"])
    unit = np.float64(np.nextafter(iso, np.float32(np.inf)) - iso) / 2
    m = samp[leaves].astype(np.float64) / unit
    assert np.array_equal(m, np.rint(m))
    x, in_cell, sing = PR.qef_solve_f64_batch(nodes["center"][leaves], nodes["half"][leaves], samp[leaves])
    want = in_cell & ~sing
    got = (nodes["node"][leaves][:, :3] != nodes["center"][leaves]).any(1)
    both = want & got
    err = np.abs(nodes["node"][leaves][both][:, :3] - x[both][:, :3]).max(1) / r
    print("r %g spacing %g: leaves %d, range %.3g..%.3g of 2^28, accepted %d, differ %d, max %.2e r" %
          (r, spacing, len(leaves), m.min() / 2 ** 28, m.max() / 2 ** 28, both.sum(), (want != got).sum(),
           err.max() if len(err) else 0))
    assert both.any()
    assert err.max() <= PR.QEF_VERT_TOL
    assert (want != got).sum() <= max(2, len(leaves) // 1000)
    f.close()

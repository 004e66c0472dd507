"""pi_eval_field puts many points in hash-cell order before it evaluates them:
the same values bit for bit as in small calls, which take them as they come,
on both sides of the counts where the ordering starts, with points outside the
grid, on its bounds and not finite among them, with and without gradients, and
under a budget that has no room for the ordering."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

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


def _points(fr, m):
    rng = np.random.default_rng(m)
    p = fr.xyz[rng.integers(0, fr.n, m)] + rng.normal(0.0, 2.0 * fr.radius, (m, 3))
    p[:: 997] = rng.uniform(-50.0, 50.0, p[:: 997].shape)  # mostly outside the grid
    p[5] = fr.xyz.min(0)
    p[6] = fr.xyz.max(0)
    p[7] = 1e30
    p[8, 0] = np.inf
    p[9, 1] = np.nan
    return p.astype(np.float32)


@pytest.mark.parametrize("m", [4096, 16383, 16384, 16385, 40007])
@pytest.mark.parametrize("grad", [False, True])
def test_ordered_evaluation_is_the_same(frame, m, grad):
    fr, f = frame
    p = _points(fr, m)
    got = f.eval(p, grad=grad)
    parts = [f.eval(p[k:k + 4000], grad=grad) for k in range(0, m, 4000)]
    if grad:
        assert np.array_equal(got[0], np.concatenate([x[0] for x in parts]), equal_nan=True)
        assert np.array_equal(got[1], np.concatenate([x[1] for x in parts]), equal_nan=True)
        # the value does not depend on whether gradients are asked for
        assert np.array_equal(got[0], f.eval(p), equal_nan=True)
    else:
        assert np.array_equal(got, np.concatenate(parts), equal_nan=True)


def test_without_room_for_the_ordering(frame):
    fr, f = frame
    p = _points(fr, 40007)
    want = f.eval(p)
    probe = N.Context(0)
    g = N.Frame(probe, N.default_params(fr.radius)).upload(fr.xyz).hashgrid().aniso().normals()
    used = probe.stats()["bytes"]
    g.close()
    probe.close()
    c = N.Context(0, budget_bytes=used + 16 * len(p) + 4096)  # the points and the values, no more
    g = N.Frame(c, N.default_params(fr.radius)).upload(fr.xyz).hashgrid().aniso().normals()
    assert np.array_equal(g.eval(p), want, equal_nan=True)
    g.close()
    c.close()

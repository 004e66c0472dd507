"""A frame whose stages fail for want of memory (PI_ERR_NOMEM under a budget)
stays usable: its info can be read, and a later attempt finds every node array
and counts from zero."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

pytestmark = pytest.mark.gpu


def _nomem(call):
    with pytest.raises(N.PiError) as e:
        call()
    assert e.value.code == N.PI_ERR_NOMEM


def _bytes(fr, stages):
    c = N.Context(0)
    f = N.Frame(c, N.default_params(fr.radius)).upload(fr.xyz)
    for s in stages:
        getattr(f, s)()
    b = c.stats()["bytes"]
    f.close()
    c.close()
    return b


def test_info_after_two_failed_attempts():
    """The first attempt fails behind the hash stage and leaves its count of valid
    keys unread; the second one fails in the hash stage, at a table of 10^8 cells."""
    B.build()
    fr = synth.small_blob(n=2000, seed=3)
    c = N.Context(0, budget_bytes=_bytes(fr, ["hashgrid"]) + 16384)
    f = N.Frame(c, N.default_params(fr.radius)).upload(fr.xyz)
    _nomem(f.run)
    wide = fr.xyz.copy()
    wide[0] = wide.max(0) + 500 * 4 * fr.radius
    f.upload(wide)
    _nomem(f.run)
    info = f.info()
    assert info["num_particles"] == fr.n and info["num_triangles"] == 0
    f.upload(fr.xyz).hashgrid()
    assert f.info()["num_invalid_keys"] == int(np.sum(f.dump(N.DUMP_KEYS) < 0))
    f.close()
    c.close()


@pytest.mark.parametrize("value,code", [(np.nan, N.PI_ERR_INVALID), (np.inf, N.PI_ERR_INVALID), (1e9, N.PI_ERR_LIMIT)])
def test_refusals_do_not_depend_on_the_memory_left(value, code):
    """Positions that are not finite, or too far apart for the grid, are refused as
    such under a budget that the particles alone take."""
    B.build()
    fr = synth.small_blob(n=20000, seed=3)
    xyz = fr.xyz.copy()
    xyz[7, 1] = value
    for budget in (12 * fr.n + 4096, 0):
        c = N.Context(0, budget_bytes=budget)
        f = N.Frame(c, N.default_params(fr.radius)).upload(xyz)
        with pytest.raises(N.PiError) as e:
            f.hashgrid()
        assert e.value.code == code
        f.close()
        c.close()


def _state(call):
    with pytest.raises(N.PiError) as e:
        call()
    assert e.value.code == N.PI_ERR_STATE


def test_failed_uploads_leave_no_results():
    """The results of a frame are of the particles it had before an upload that fails;
    none can be asked for until there are particles again."""
    B.build()
    fr = synth.two_radius_frame(n=2000, seed=6)
    p = N.default_params(float(fr.radii.min()))
    probe = N.Context(0)
    f = N.Frame(probe, p).upload(fr.xyz).upload_radii(fr.radii).hashgrid().aniso()
    used = probe.stats()["bytes"]
    want = f.dump(N.DUMP_XMEANS)
    f.close()
    probe.close()
    c = N.Context(0, budget_bytes=used + (1 << 20))
    f = N.Frame(c, p).upload(fr.xyz).upload_radii(fr.radii).hashgrid().aniso()
    _nomem(lambda: f.upload(np.zeros((1 << 20, 3), np.float32)))
    _state(lambda: f.dump(N.DUMP_XMEANS))
    _state(f.hashgrid)
    f.upload(fr.xyz).upload_radii(fr.radii).hashgrid().aniso()
    assert np.array_equal(f.dump(N.DUMP_XMEANS), want)
    g = N.Frame(c, p)  # one that has never held any
    _nomem(lambda: g.upload(np.zeros((1 << 20, 3), np.float32)))
    _state(lambda: g.upload_radii(fr.radii))
    _state(g.hashgrid)
    g.close()
    f.close()
    c.close()


COUNTS = ("num_nodes", "num_leaves", "num_dual_cells", "num_vertices", "num_triangles", "field_evals",
          "candidate_pairs", "bisection_evals", "fp64_eigen", "field_evals_performed", "qef_accepted", "qef_singular")


def _least_budget(fr, p):
    """The least budget of the whole frame, and its counts."""
    lo, hi = _bytes(fr, ["hashgrid", "aniso", "normals"]), 1 << 30
    whole = None
    while hi - lo > 1 << 16:
        b = (lo + hi) // 2
        c = N.Context(0, budget_bytes=b)
        f = N.Frame(c, p).upload(fr.xyz)
        try:
            info = f.run().info()
            whole, hi = {k: info[k] for k in COUNTS}, b
        except N.PiError as e:
            assert e.code == N.PI_ERR_NOMEM
            lo = b
        f.close()
        c.close()
    return hi, whole


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("qef", [False, True])
@pytest.mark.parametrize("share", [0.1, 0.3, 0.6, 0.9])
def test_counts_after_a_failed_attempt(qef, share, staged):
    """Another frame takes the memory that the octree or the extraction needs; when
    it is gone the stage runs again, at once or after its info was read, and every
    count is a first run's."""
    B.build()
    fr = synth.slab_and_sphere(n=20000, seed=1)
    p = N.default_params(fr.radius, qef=qef)
    least, whole = _least_budget(fr, p)
    base = _bytes(fr, ["hashgrid", "aniso", "normals"])
    # node arrays that have grown stay: a second attempt may need more than a first
    c = N.Context(0, budget_bytes=2 * least)
    other = N.Frame(c, p)
    f = N.Frame(c, p).upload(fr.xyz).hashgrid().aniso().normals()
    rest = (lambda: f.octree().extract()) if staged else f.run
    # 12 bytes a particle: what the other frame leaves is `share` of what the rest needs
    other.upload(np.zeros((int(least + (1 - share) * (least - base)) // 12, 3), np.float32))
    _nomem(rest)
    if share != 0.6:
        f.info()
    other.close()
    info = rest().info()
    assert {k: info[k] for k in COUNTS} == whole
    f.close()
    c.close()

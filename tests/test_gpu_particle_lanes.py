"""Anisotropy and normals of a small frame, whose particles have four lanes each,
against those of the same particles in a frame too large for that: equal bits.

The larger frame adds particles more than 12 r from the first ones, inside the same
box, so the hash grid and the candidates of the first ones, and their order, stay."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

pytestmark = pytest.mark.gpu

R = 0.0078125  # a power of two: the box arithmetic is exact


def _points(n, extra, seed):
    """n particles of one region (a ragged blob, a sheet, lone ones), the box's
    corners, then `extra` in the other half of the box."""
    rng = np.random.default_rng(seed)
    blob = rng.uniform(0.0, 0.3, (n, 3)) * np.array([1.0, 1.0, np.cbrt(n) / 40])
    blob[: n // 8, 2] = 0.15
    corners = np.array([[0.0, 0.0, 0.0], [2.0, 1.0, 1.0]])
    far = rng.uniform(0.0, 1.0, (extra, 3)) * np.array([0.9, 0.9, 0.9]) + np.array([1.0, 0.0, 0.0])
    return np.concatenate([corners, blob, far]).astype(np.float32)


def _state(ctx, xyz, radii, splash):
    f = N.Frame(ctx, N.default_params(R, splash=splash)).upload(xyz)
    if radii is not None:
        f.upload_radii(radii)
    f.hashgrid().aniso().normals()
    out = {k: f.dump(k) for k in (N.DUMP_XMEANS, N.DUMP_G, N.DUMP_DET, N.DUMP_NORMALS, N.DUMP_FP64_FLAGS)}
    f.close()
    return out


@pytest.mark.parametrize("n,varr,splash", [
    (1, False, False), (31, False, True), (1000, False, False), (5003, False, True), (20000, False, False),
    (7001, True, False)])
def test_small_frames_have_the_large_frames_bits(n, varr, splash):
    B.build()
    ctx = N.Context(0)
    extra = 120000
    xyz = _points(n, extra, n)
    radii = None
    if varr:
        radii = np.where(np.random.default_rng(n).uniform(size=len(xyz)) < 0.3, R, 2 * R).astype(np.float32)
        radii[:2], radii[-2:] = R, (R, 2 * R)
        # both bins' boxes are the same in both frames
        xyz[n + 1], xyz[n] = xyz[1], xyz[0]
        radii[n + 1] = radii[n] = 2 * R
    m = n + 2
    # the second corner takes part in the extra particles' region: leave it out
    keep = np.r_[0, 2:m - (2 if varr else 0)] if n > 2 else np.r_[0]
    small = _state(ctx, xyz[:m], None if radii is None else radii[:m], splash)
    large = _state(ctx, xyz, radii, splash)
    for k in small:
        assert np.array_equal(small[k][keep], large[k][keep]), k
    ctx.close()

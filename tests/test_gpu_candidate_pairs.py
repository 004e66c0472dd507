"""The work counters of the kernels whose points share their candidates: the
candidate pairs that the leaf values and the edge bisection report are the sums
of their points' 27-cell list lengths (pi_hashgrid_neighbors), on meshes of few
vertices (4 to a warp), some and many, and with last warps that are partly
filled."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth
from test_gpu_consistency import bisect_f32

pytestmark = pytest.mark.gpu

FRAMES = {
    "blob_150": lambda: synth.small_blob(n=150, seed=5),
    "blob_700": lambda: synth.small_blob(n=700, seed=6),
    "blob_4000": lambda: synth.small_blob(n=4000, seed=7),
    "slab_9001": lambda: synth.slab_and_sphere(n=9001, seed=8),
    "slab_20000": lambda: synth.slab_and_sphere(n=20000, seed=1),
    "spray_20000": lambda: synth.spray_frame(n=20000, seed=23, radius=0.01),
    "sheets_30000": lambda: synth.sheets_and_filaments(n=30000, seed=9),
}


@pytest.mark.parametrize("case", list(FRAMES))
def test_pairs_are_the_candidates_of_every_point(case):
    B.build()
    fr = FRAMES[case]()
    ctx = N.Context(0)
    ctx.profile(True)
    f = N.Frame(ctx, N.default_params(fr.radius)).upload(fr.xyz).hashgrid().aniso().normals().octree()
    before = f.info()["candidate_pairs"]
    info = f.extract().info()
    groups = ctx.kernel_groups()
    nodes = f.dump(N.DUMP_NODES)

    finest = nodes[(nodes["type"] == 2) & (nodes["depth"] == info["depth_max"])]["node"][:, :3]
    assert groups["leaf_values"]["units"] == len(finest) > 0
    assert groups["leaf_values"]["pairs"] == f.neighbors(finest)[0][-1]

    e = f.dump(N.DUMP_VERTEX_EDGES)
    mids = []

    def value(p):
        mids.append(p)
        return f.eval(p)

    bisect_f32(nodes["node"][e[:, 0]], nodes["node"][e[:, 1]], np.float32(fr.radius) / np.float32(2), value)
    mids = np.concatenate(mids)
    want = int(f.neighbors(mids)[0][-1])
    assert info["bisection_evals"] == groups["bisection"]["units"] == len(mids) > 0
    assert groups["bisection"]["pairs"] == want
    assert info["candidate_pairs"] - before == want
    f.close()
    ctx.close()

"""The frame's hash order with cells of every size the sort treats differently:
empty, small, just below and above the block-sorted size, thousands of particles,
and particles on the grid's upper bounds (key -1, at the front): IndexList is the
stable sort by key, and the positions follow it."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

pytestmark = pytest.mark.gpu

R = 0.0078125  # a power of two: the box arithmetic is exact


@pytest.fixture(scope="module")
def ctx():
    B.build()
    c = N.Context(0)
    yield c
    c.close()


def _points(counts, outside, seed):
    """counts[c] particles in cell c of a line of cells, and `outside` more on
    the upper bound of the x axis, all in a seeded order."""
    rng = np.random.default_rng(seed)
    cell = 4 * R
    parts = [np.array([[0.0, 0.0, 0.0]])]
    for c, k in enumerate(counts):
        parts.append(np.stack([(c + rng.uniform(0.05, 0.95, k)) * cell, rng.uniform(0.0, 0.5 * cell, k),
                               rng.uniform(0.0, 0.5 * cell, k)], -1))
    end = len(counts) * cell
    parts.append(np.stack([np.full(max(outside, 1), end), rng.uniform(0, 0.5 * cell, max(outside, 1)),
                           np.zeros(max(outside, 1))], -1))
    p = np.concatenate(parts).astype(np.float32)
    return p[rng.permutation(len(p))]


@pytest.mark.parametrize("counts,outside", [
    ((1,), 0), ((0, 3, 0, 8, 1), 1), ((255, 0, 256, 257, 2), 5), ((300, 300, 300, 300), 400),
    ((5000, 1, 0, 70000, 12, 258), 1000), (tuple([9] * 3000), 40)])
def test_index_list_is_the_stable_order(ctx, counts, outside):
    xyz = _points(counts, outside, len(counts) + outside)
    f = N.Frame(ctx, N.default_params(R)).upload(xyz).hashgrid()
    keys = f.dump(N.DUMP_KEYS)
    assert (keys == -1).sum() == f.info()["num_invalid_keys"] >= max(outside, 1)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(f.dump(N.DUMP_INDEX_LIST), order)
    cells = f.info()["cell_num"]
    want = np.concatenate([[0], np.cumsum(np.bincount(keys[keys >= 0], minlength=cells))])
    assert np.array_equal(f.dump(N.DUMP_CELL_OFFSETS), want)
    f.close()

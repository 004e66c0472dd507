"""The hash order's cells above the block-sorted size, which are put in order by
windows of particle indices: at the size where that starts, at every alignment of
the cell's range, beside other listed cells, with all particles in one cell or
outside the grid but two, and with windows as wide as their bits allow."""
import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from test_gpu_cell_sort import R, _points

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    B.build()
    c = N.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("counts,outside", [
    ((4095, 4096, 4097, 1, 4098, 2, 4099, 3, 4100), 3), ((5000,), 0), ((4097, 300, 0, 12000, 257, 4096, 9000), 4098),
    ((1, 1), 20000), ((8200, 8201, 8202, 8203) * 8, 8204), ((31,) * 50 + (200000,) + (7,) * 50, 30301),
    ((2_000_000, 3, 3_500_000), 1_000_000), ((9,) * 600_000 + (6000,), 5)])
def test_index_list_is_the_stable_order(ctx, counts, outside):
    xyz = _points(counts, outside, len(counts) + outside)
    f = N.Frame(ctx, N.default_params(R)).upload(xyz).hashgrid()
    keys = f.dump(N.DUMP_KEYS)
    assert (keys == -1).sum() == f.info()["num_invalid_keys"] >= max(outside, 1)
    order = f.dump(N.DUMP_INDEX_LIST)
    assert np.array_equal(order, np.argsort(keys, kind="stable"))
    # the positions follow the order: a query's candidates are the cell's particles
    q = xyz[[0, len(xyz) // 2, len(xyz) - 1]]
    off, idx = f.neighbors(q)
    assert np.all(np.diff(off) >= 0) and idx.size == off[-1]
    f.close()

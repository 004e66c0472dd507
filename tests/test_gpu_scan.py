"""The exclusive scan behind the cell offsets, at the sizes where its launches
change (one block, a cluster with 4 and with 32 elements a thread, tiles, tiles
whose sums are scanned too) and on an output that is not 16-byte aligned, against
the counts of the cell keys."""
import ctypes as C

import numpy as np
import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B

pytestmark = pytest.mark.gpu

R = 0.0078125  # a power of two: the box arithmetic is exact, so the cell counts are those asked for


def _cells(dims, n, seed):
    """n particles in a box of exactly `dims` hash cells, most in a few cells."""
    rng = np.random.default_rng(seed)
    size = (np.array(dims) - 0.5) * 4 * R
    p = rng.uniform(0.0, 1.0, (n, 3)) ** rng.choice([0.2, 1.0, 5.0], (n, 1)) * size
    p[0], p[1] = 0.0, size
    return p.astype(np.float32)


def _offsets(keys, cells):
    return np.concatenate([[0], np.cumsum(np.bincount(keys[keys >= 0], minlength=cells))])


@pytest.fixture(scope="module")
def ctx():
    B.build()
    c = N.Context(0)
    yield c
    c.close()


# the scan has cells + 1 elements
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 9, 7), (13, 15, 21), (16, 16, 16), (7, 31, 151), (32, 32, 32),
                                  (64, 64, 31), (510, 257, 1), (512, 256, 1), (64, 64, 66), (331, 320, 317)])
def test_cell_offsets(ctx, dims):
    xyz = _cells(dims, 5000, sum(dims))
    f = N.Frame(ctx, N.default_params(R)).upload(xyz).hashgrid()
    cells = f.info()["cell_num"]
    assert tuple(f.info()["xyz_cell_num"]) == dims
    assert np.array_equal(f.dump(N.DUMP_CELL_OFFSETS), _offsets(f.dump(N.DUMP_KEYS), cells))
    f.close()


@pytest.mark.parametrize("dims", [(5, 9, 7), (20, 20, 20), (40, 50, 60), (60, 70, 80)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_unaligned_offsets(dims, shift):
    torch = pytest.importorskip("torch")
    B.build()
    xyz = torch.from_numpy(_cells(dims, 4000, 3)).cuda()
    n, cells = len(xyz), int(np.prod(dims))
    keys = torch.empty(n, dtype=torch.int32, device="cuda")
    idx = torch.empty(n, dtype=torch.int32, device="cuda")
    room = torch.full((cells + 1 + shift + 8,), -7, dtype=torch.int32, device="cuda")
    b, d, cn = np.zeros(6, np.float32), np.zeros(3, np.int32), C.c_int64()
    fn = N.lib().pi_hashgrid_build_noalloc
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64,
                   C.POINTER(C.c_float), C.POINTER(C.c_int32), C.POINTER(C.c_int64), C.c_void_p]
    torch.cuda.synchronize()
    N.check(fn(xyz.data_ptr(), n, R, keys.data_ptr(), idx.data_ptr(), room[shift:].data_ptr(), cells + 1,
               N.ptr(b, C.c_float), N.ptr(d, C.c_int32), C.byref(cn), None))
    got = room.cpu().numpy()
    assert cn.value == cells
    assert np.array_equal(got[shift:shift + cells + 1], _offsets(keys.cpu().numpy(), cells))
    assert (got[:shift] == -7).all() and (got[shift + cells + 1:] == -7).all()

"""What a context keeps of released device blocks serves the frames that follow:
small frames take next to nothing from the pool after a large frame has filled
the list, and a context gets the memory that an idle one keeps.  Seen through the
pool's own counters."""
import ctypes as C

import pytest

from particleisosurface_gb300 import _native as N
from particleisosurface_gb300 import build as B
from particleisosurface_gb300 import synth

pytestmark = pytest.mark.gpu

RESERVED, USED_CURRENT, USED_HIGH = 5, 7, 8  # CU_MEMPOOL_ATTR_RESERVED_MEM_CURRENT, ..._USED_MEM_...


class Pool:
    """The device's default memory pool."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        assert self.cu.cuInit(0) == 0
        dev, self.pool = C.c_int(), C.c_void_p()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def get(self, attr):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def taken_by(self, call):
        """Bytes in use at most during the call, above those before it."""
        zero = C.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(zero)) == 0
        before = self.get(USED_CURRENT)
        call()
        return self.get(USED_HIGH) - before


def _frame(ctx, fr):
    f = N.Frame(ctx, N.default_params(fr.radius)).upload(fr.xyz).run()
    f.close()


@pytest.mark.parametrize("first", [300_000, 600_000, 1_000_000])
def test_small_frames_after_a_large_one(first):
    B.build()
    large, small = synth.dam_break(n=first, seed=2), synth.slab_and_sphere(n=2000, seed=1)
    pool = Pool()
    ctx = N.Context(0)
    whole = pool.taken_by(lambda: _frame(ctx, small))  # the first one: everything comes from the pool
    assert whole > 1 << 20
    ctx.close()
    ctx = N.Context(0)
    for _ in range(2):
        _frame(ctx, large)
    _frame(ctx, small)
    _frame(ctx, small)
    assert pool.taken_by(lambda: _frame(ctx, small)) < whole // 20
    ctx.close()


def test_an_idle_context_gives_its_blocks():
    B.build()
    fr = synth.dam_break(n=300_000, seed=2)
    idle, other, probe = N.Context(0), N.Context(0), N.Context(0)
    pool = Pool()
    need = pool.taken_by(lambda: _frame(probe, fr))
    probe.close()
    _frame(idle, synth.dam_break(n=600_000, seed=2))
    kept = pool.get(USED_CURRENT)
    assert kept > 200 << 20
    assert pool.cu.cuCtxSynchronize() == 0 and pool.cu.cuMemPoolTrimTo(pool.pool, C.c_size_t(0)) == 0
    # the device's memory goes but for 100 MB less than the frame needs, which the
    # idle context keeps twice over
    left = need - (pool.get(RESERVED) - kept) - (100 << 20)
    if left <= 0:
        pytest.skip("the pool holds enough beside the kept blocks")
    free, total = C.c_size_t(), C.c_size_t()
    assert pool.cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    block = C.c_uint64()
    assert pool.cu.cuMemAlloc_v2(C.byref(block), C.c_size_t(free.value - left)) == 0
    try:
        _frame(other, fr)
    finally:
        assert pool.cu.cuMemFree_v2(block) == 0
    other.close()
    idle.close()

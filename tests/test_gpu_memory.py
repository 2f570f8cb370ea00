"""Device blocks kept for reuse: sizes, contents, limits, misuse."""
import ctypes

import numpy
import pytest

from kelvin_gb300 import _lib

pytestmark = pytest.mark.gpu


def alloc(ctx, nbytes):
    p = _lib.vp()
    ctx.check(ctx.L.kvft_alloc(ctx.h, nbytes, ctypes.byref(p)), "kvft_alloc")
    return p.value


def test_blocks_are_reused_by_size():
    ctx, other = _lib.Context(0), _lib.Context(0)
    try:
        # blocks kept by the rest of the process go back first (a request that
        # cannot be met releases them): the smallest kept block that fits is
        # taken, and one of theirs may fit better than this test's
        p = _lib.vp()
        assert ctx.L.kvft_alloc(ctx.h, 2 * ctx.mem_info()[1], ctypes.byref(p)) == 2
        a = alloc(ctx, 40 << 20)
        b = alloc(ctx, 40 << 20)
        assert a != b
        free0 = ctx.mem_info()[0]
        assert ctx.L.kvft_free(ctx.h, a) == 0
        # a kept block counts as free memory
        assert ctx.mem_info()[0] >= free0 + (40 << 20)
        # an eighth smaller still takes it, from another context too; half does not
        c = alloc(other, 20 << 20)
        assert c != a
        d = alloc(other, 36 << 20)
        assert d == a
        assert ctx.L.kvft_free(ctx.h, a) == 0         # the same block, whoever asked for it
        assert ctx.L.kvft_free(ctx.h, a) == 1         # twice: KVFT_EINVAL
        for p in (b, c):
            assert ctx.L.kvft_free(ctx.h, p) == 0
        assert ctx.L.kvft_free(ctx.h, None) == 0
    finally:
        other.close()
        ctx.close()


def test_a_kept_block_is_not_larger_than_the_limit():
    ctx = _lib.Context(0)
    try:
        total = ctx.mem_info()[1]
        big = alloc(ctx, total // 32 + (1 << 20))
        assert ctx.L.kvft_free(ctx.h, big) == 0
        p = _lib.vp()
        # more than exists fails cleanly and gives back what was kept
        assert ctx.L.kvft_alloc(ctx.h, 2 * total, ctypes.byref(p)) == 2   # KVFT_ENOMEM
        x = _lib.DeviceArray.from_host(ctx, numpy.arange(5.0))
        assert numpy.array_equal(x.to_host(), numpy.arange(5.0))
        x.free()
    finally:
        ctx.close()

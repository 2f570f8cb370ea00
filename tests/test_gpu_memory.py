"""Device blocks kept for reuse: sizes, contents, limits, misuse."""
import ctypes
import threading

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


def test_free_leaves_another_threads_capture_alone():
    """A block freed while another thread captures a graph: the capture goes
    on, the block is kept, and the freeing thread's next launch is fine."""
    torch = pytest.importorskip("torch")
    ctx = _lib.Context(0)
    try:
        a = alloc(ctx, 48 << 20)
        y = _lib.DeviceArray.from_host(ctx, numpy.arange(4096.0).reshape(64, 64))
        z = _lib.DeviceArray(ctx, (64, 64))
        x = torch.zeros(8, device="cuda")
        side = torch.cuda.Stream()
        x.add_(1)
        torch.cuda.synchronize()
        status = []

        def free():
            status.append(ctx.L.kvft_free(ctx.h, a))
            status.append(ctx.L.kvft_gemm(ctx.h, 64, 64, 64, 1, _lib.PREC_FP64, 7, y.ptr, y.ptr,
                                          z.ptr))

        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side, capture_error_mode="relaxed"):
            x.add_(1)
            t = threading.Thread(target=free)
            t.start()
            t.join()
            x.add_(1)
        assert status == [0, 0]
        g.replay()
        torch.cuda.synchronize()
        assert (x == 3).all()
        h = numpy.arange(4096.0).reshape(64, 64)
        assert numpy.allclose(z.to_host(), h @ h, rtol=1e-13)
        b = alloc(ctx, 48 << 20)
        assert b == a
        assert ctx.L.kvft_free(ctx.h, b) == 0
        y.free()
        z.free()
    finally:
        ctx.close()


def test_free_waits_for_every_stream():
    """A freed block is not handed out while a stream of the caller's own may
    still use it."""
    torch = pytest.importorskip("torch")
    ctx = _lib.Context(0)
    try:
        a = alloc(ctx, 8 << 20)
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(40 * 1000 * 1000)          # clocks: about 20 ms
        done = side.record_event()
        assert not done.query()
        assert ctx.L.kvft_free(ctx.h, a) == 0
        assert done.query()
    finally:
        ctx.close()


@pytest.mark.parametrize("nbytes", [2 ** 64 - 1, 2 ** 64 - 511, 2 ** 64 - 512, 2 ** 63, 2 ** 48 + 1])
def test_sizes_beyond_the_address_space_are_refused(nbytes):
    """Sizes that rounding up to whole blocks would wrap, and beside them."""
    ctx = _lib.Context(0)
    try:
        p = _lib.vp()
        assert ctx.L.kvft_alloc(ctx.h, nbytes, ctypes.byref(p)) != 0
        assert not p.value
    finally:
        ctx.close()


def test_kept_blocks_are_given_back_on_request():
    """What is kept for reuse returns to the driver, where others find it."""
    torch = pytest.importorskip("torch")
    ctx, other = _lib.Context(0), _lib.Context(0)
    try:
        a = alloc(ctx, 640 << 20)
        assert ctx.L.kvft_free(ctx.h, a) == 0
        free = torch.cuda.mem_get_info()[0]
        other.release_memory()                          # any context of the device
        assert torch.cuda.mem_get_info()[0] >= free + (640 << 20)
        ctx.release_memory()                            # nothing kept: nothing happens
        x = _lib.DeviceArray.from_host(ctx, numpy.arange(5.0))
        assert numpy.array_equal(x.to_host(), numpy.arange(5.0))
        x.free()
    finally:
        other.close()
        ctx.close()

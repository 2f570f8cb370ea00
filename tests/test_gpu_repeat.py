"""Sums that repeat to the bit: products whose K is at most 2048 (tensor cores,
four and more levels) or 64 (FP64) give the same result in every run, however
few their output tiles are."""
import numpy
import pytest

from conftest import random_system
from kelvin_gb300 import _lib, ft_cc_equations

pytestmark = pytest.mark.gpu


# The last K of one range and of eight, odd and even extents, a batch, several
# tiles; the error bound is that of the digit count.
@pytest.mark.parametrize("digits,tol", [(4, 5e-7), (5, 5e-9), (6, 5e-11), (7, 5e-12)])
@pytest.mark.parametrize("M,N,K,batch", [(37, 21, 2048, 1), (1, 70, 2047, 1), (70, 40, 513, 1),
                                         (19, 19, 1900, 3), (130, 100, 1025, 2), (129, 1, 777, 5)])
def test_tensor_core_products_repeat(ctx, M, N, K, batch, digits, tol):
    rng = numpy.random.default_rng(M + N + K)
    A, B = rng.standard_normal((batch, M, K)), rng.standard_normal((batch, K, N))
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray.from_host(ctx, numpy.full((batch, M, N), numpy.nan))

    def run():
        ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                                  dC.ptr), "kvft_gemm")
        return dC.to_host()

    C = run()
    bound = abs(A).max(2)[:, :, None] * abs(B).max(1)[:, None, :] * K
    assert (abs(C - A @ B) <= tol * bound).all()
    assert all((run() == C).all() for _ in range(30))


# A residual whose longest sums have 64 terms: products that add into C.
def test_fp64_residual_repeats(ctx, nv=4, no=4):
    rng = numpy.random.default_rng(nv + no)
    F, I = random_system(rng, no, nv)
    t1 = rng.standard_normal((nv, no)) * 0.05
    t2 = rng.standard_normal((nv, nv, no, no)) * 0.05
    t2 = t2 - t2.transpose(1, 0, 2, 3)
    t2 = t2 - t2.transpose(0, 1, 3, 2)
    ctx.set_precision(_lib.PREC_FP64, 7)
    first = None
    for _ in range(200):
        T1, T2 = -F.vo.copy(), -I.vvoo.copy()
        ft_cc_equations.stanton_residual(T1, T2, F, I, t1, t2, ctx=ctx)
        first = first or (T1, T2)
        assert (T1 == first[0]).all() and (T2 == first[1]).all()

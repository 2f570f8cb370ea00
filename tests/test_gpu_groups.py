"""Products that share one launch (the spin blocks of a contraction), and the
FP64 kernel's free tile extents."""
import numpy
import pytest

from conftest import random_system, random_T
from kelvin_gb300 import _lib, ft_cc_equations, systems
from kelvin_gb300.cc_utils import F_ORDER, I_ORDER, DeviceSolver
from kelvin_gb300.quadrature import ft_quad
from oracle import ft_ccsd as oft
from oracle import ft_utils

pytestmark = pytest.mark.gpu


# One output, single rows and columns, extents around the 64 and 128 tile
# limits and around each thread's output counts, one k and k around the block
# of 16, K split over blocks (few outputs, long K), odd batches.
@pytest.mark.parametrize("M,N,K,batch", [
    (1, 1, 1, 1), (1, 129, 3, 2), (129, 1, 17, 1), (13, 2197, 13, 3), (2197, 13, 13, 3),
    (19, 19, 6859, 2), (8, 8, 512, 10), (64, 65, 16, 1), (65, 64, 15, 1), (127, 33, 33, 5),
    (361, 361, 361, 1), (57, 4000, 57, 1), (2, 300, 1000, 1),
    # a row per thread: 128-, 64- and 32-row blocks, 1 to 24 columns, several
    # column tiles (25, 49, 64), K around its block of 16, either side big
    (40000, 1, 16, 2), (33000, 24, 17, 4), (20011, 25, 15, 3), (9000, 49, 31, 3),
    (64, 7777, 9, 5), (8, 512, 8, 60), (5000, 13, 13, 20),
    # K in two or four slices of a block: 32, 33, 64 and 65 outputs a tile, K
    # below the slice count and around the block of 32
    (4, 8, 1, 2), (4, 8, 3, 2), (8, 4, 33, 2), (3, 11, 31, 1), (8, 8, 5, 3), (8, 8, 65, 3),
    (5, 13, 34, 1),
    # 64 x 64 tiles: full ones, ragged by one and two in each direction, K
    # around its block of 16, a batch; just too few tiles; a long K whose ranges
    # count as blocks
    (2048, 2048, 17, 1), (2047, 2046, 31, 1), (1024, 1023, 48, 4), (1920, 1920, 20, 1),
    (57, 57, 9000, 2), (300, 57, 1024, 2), (200, 130, 1023, 1)])
def test_gemm_fp64_tiles(ctx, M, N, K, batch):
    rng = numpy.random.default_rng(M + 3 * N + 7 * K + batch)
    A = rng.standard_normal((batch, M, K))
    B = rng.standard_normal((batch, K, N))
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, (batch, M, N))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64, 7, dA.ptr, dB.ptr, dC.ptr),
              "kvft_gemm")
    # each of the two sums (numpy's and the kernel's) is within K units of
    # roundoff of the exact one, relative to the sum of magnitudes
    bound = 2.0 * (K + 2) * 2.0 ** -53 * (abs(A) @ abs(B))
    assert (abs(dC.to_host() - A @ B) <= bound).all()


# Odd alpha halves, so that every block's offset is odd: 3 (all products on
# the FP64 pipe), 13 and 17 (both engines), against the oracle's full sums.
@pytest.mark.parametrize("pw,prec,digits,tol", [
    (3, _lib.PREC_FP64, 7, 1e-12), (3, _lib.PREC_FP64_TC, 7, 1e-12),
    (13, _lib.PREC_FP64, 7, 1e-12), (17, _lib.PREC_FP64_TC, 7, 1e-10)])
def test_grouped_update_vs_oracle(ctx, pw, prec, digits, tol):
    s = systems.ueg_recipe(2, 2.0, pw, 0.5)
    beta, ng = 1.0 / s.T, 4
    en = s.g_energies_tot()
    n = en.shape[0]
    ti, g, G = ft_quad(ng, beta, "lin")
    F, I = oft.ft_integrals(s.g_fock_tot(), s.g_aint_tot(), en, beta, s.mu)
    D1, D2 = ft_utils.D1(en, en), ft_utils.D2(en, en)
    rng = numpy.random.default_rng(pw)
    sp = numpy.arange(n) >= n // 2
    t1 = rng.standard_normal((ng, n, n)) * 0.05 * (sp[:, None] == sp)
    t2 = rng.standard_normal((ng, n, n, n, n)) * 0.05
    t2 = t2 - t2.transpose(0, 2, 1, 3, 4)
    t2 = (t2 - t2.transpose(0, 1, 2, 4, 3)) * (
        sp[:, None, None, None].astype(int) + sp[None, :, None, None]
        == sp[None, None, :, None].astype(int) + sp)
    r1, r2 = oft.ccsd_stanton(F, I, t1, t2, D1, D2, ti, ng, G)
    ctx.set_precision(prec, digits)
    try:
        o1, o2 = ft_cc_equations.ccsd_stanton(F, I, t1, t2, D1, D2, ti, ng, G, ctx=ctx)
    finally:
        ctx.set_precision(_lib.PREC_FP64, 7)
    assert abs(o1 - r1).max() <= tol * max(1.0, abs(r1).max())
    assert abs(o2 - r2).max() <= tol * max(1.0, abs(r2).max())


# The Lambda path's groups write beta = 0 outputs without a separate pass over
# them; a device buffer that held NaN before must come out clean.
def test_grouped_lambda_leaves_no_stale_blocks(ctx):
    s = systems.ueg_recipe(2, 2.0, 7, 0.5)
    beta = 1.0 / s.T
    ti, g, G = ft_quad(4, beta, "lin")
    sv = DeviceSolver.from_system(ctx, s.g_energies_tot(), s.g_fock_tot(), s.g_aint_tot(), beta,
                                  s.mu, ti, g, G)
    try:
        sv.guess(1)
        conv = {"max_iter": 2, "damp": 0.2, "tconv": 1e-14}
        on = sv.lambda_solve(conv)
        sv.spin_blocks(False)
        off = sv.lambda_solve(conv)
    finally:
        sv.close()
    for a, b in zip(on, off):
        assert numpy.isfinite(a).all()
        assert abs(a - b).max() <= 1e-12 * max(1.0, abs(b).max())


# A big tensor with a small matrix (K, N <= 64): k and column edges of the 32-
# and 64-deep tiles and of the 16-column MMA steps, one column, partial row
# tiles, the big operand on either side (its rows or k contiguous), every
# digit count.  Norm-wise bounds by digit count as for the general kernel.
@pytest.mark.parametrize("M,N,K,batch", [(2049, 1, 16, 1), (700, 16, 17, 3), (1100, 33, 32, 2),
                                         (1025, 64, 33, 2), (2100, 57, 57, 1), (900, 31, 64, 4)])
@pytest.mark.parametrize("digits", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("big_left", [True, False])
def test_thin_contraction(ctx, M, N, K, batch, digits, big_left):
    rng = numpy.random.default_rng(M + 3 * N + 7 * K + digits)
    A = rng.standard_normal((batch, M, K)) * numpy.exp(rng.standard_normal((batch, M, 1)) * 3)
    B = rng.standard_normal((batch, K, N)) * numpy.exp(rng.standard_normal((batch, 1, N)) * 3)
    A[:, 5] = 0.0
    if not big_left:
        A, B = (numpy.ascontiguousarray(x.transpose(0, 2, 1)) for x in (B, A))
    m, n = A.shape[1], B.shape[2]
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, (batch, m, n))
    ctx.check(ctx.L.kvft_gemm(ctx.h, m, n, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    C = dC.to_host()
    tol = {2: 2e-3, 3: 5e-5, 4: 5e-7, 5: 5e-9, 6: 5e-11, 7: 5e-12}[digits]
    bound = abs(A).max(2)[:, :, None] * abs(B).max(1)[:, None, :] * K
    assert (abs(C - A @ B) <= tol * (256 / K) ** 0.5 * bound).all()


def test_group_of_a_large_batch(ctx, n=8, nb=11000, digits=7):
    """The sub-blocks of a group times its batch exceed 65535, a single
    product's batch does not: each entry is what it is in a batch of three.
    The tolerance is the rounding of FP64 additions in another order."""
    rng = numpy.random.default_rng(3)
    h = n // 2
    s = numpy.arange(n) >= h
    F, I = random_system(rng, n, n)
    for b in ("oo", "ov", "vo", "vv"):
        getattr(F, b)[s[:, None] != s] = 0.0
    cons = (s[:, None, None, None].astype(int) + s[:, None, None]) == (s[:, None].astype(int) + s)
    for b in ("vvvv", "vvvo", "vovv", "vvoo", "vovo", "oovv", "vooo", "ooov", "oooo"):
        getattr(I, b)[~cons] = 0.0
    t1, t2 = random_T(rng, 3, n, n)
    t1[:, s[:, None] != s] = 0.0
    t2[:, ~cons] = 0.0
    dF = [_lib.DeviceArray.from_host(ctx, getattr(F, k)) for k in F_ORDER]
    dI = [_lib.DeviceArray.from_host(ctx, getattr(I, k)) for k in I_ORDER]
    out = []
    ctx.set_precision(_lib.PREC_FP64_TC, digits)
    ctx.set_residual_spin_blocks(h)
    try:
        for idx in (numpy.arange(3), numpy.arange(nb) % 3):
            d1, d2 = _lib.DeviceArray.from_host(ctx, t1[idx]), _lib.DeviceArray.from_host(ctx, t2[idx])
            o1 = _lib.DeviceArray.from_host(ctx, numpy.zeros((len(idx), n, n)))
            o2 = _lib.DeviceArray.from_host(ctx, numpy.zeros((len(idx),) + (n,) * 4))
            ctx.check(ctx.L.kvft_stanton_residual(ctx.h, len(idx), n, n, _lib.ptr_array(dF),
                                                  _lib.ptr_array(dI), d1.ptr, d2.ptr, 1.0, o1.ptr,
                                                  o2.ptr), "kvft_stanton_residual")
            out.append((o1.to_host(), o2.to_host()))
    finally:
        ctx.set_residual_spin_blocks(0)
        ctx.set_precision(_lib.PREC_FP64, 7)
    (a1, a2), (b1, b2) = out
    for y in (0, 1, 2, 5461, 10921, 10922, 10923, nb - 1):
        assert abs(b1[y] - a1[y % 3]).max() <= 1e-11 * abs(a1).max()
        assert abs(b2[y] - a2[y % 3]).max() <= 1e-11 * abs(a2).max()

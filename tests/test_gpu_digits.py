"""The wide digits of seven levels (nine-bit, read out every 128 terms) are at
least as accurate as seven-bit digits of the same level count: the error of the device product is at most that of seven-bit
digits with exact sums, computed here, in the 2-norm and for the largest
element.  Operands: normal, A A^T (equal signs in every square), few-valued,
constant, wide-range; K below, at and above the read-out length and the
kernels' k-blocks."""
import numpy
import pytest

from kelvin_gb300 import _lib

pytestmark = pytest.mark.gpu


def operands(kind, K, M=48):
    rng = numpy.random.default_rng(K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, M))
    if kind == "aat":
        B = A.T.copy()
    elif kind == "few":
        A, B = 1.0 / rng.integers(1, 12, (M, K)), 1.0 / rng.integers(1, 9, (K, M))
    elif kind == "const":
        A, B = numpy.full((M, K), 0.3), numpy.full((K, M), 0.7)
    elif kind == "wide":
        A, B = A * numpy.exp(3 * A), B * numpy.exp(3 * B)
    return A, B


def seven_bit(A, D):
    """Balanced base-128 digits (D - 1 of them) of the rows of A, as FP64
    values, and the row exponents."""
    S = D - 1
    e = numpy.floor(numpy.log2(abs(A).max(1))) + 2
    Y = numpy.floor(abs(A) * 2.0 ** (7 * S - e)[:, None] + 0.5).astype(numpy.int64)
    d = []
    for s in range(S, 1, -1):
        low = ((Y + 64) & 127) - 64
        d.insert(0, low * 2.0 ** (-7 * s))
        Y = (Y - low) >> 7
    d.insert(0, Y * 2.0 ** -7)
    return [x * numpy.sign(A) for x in d], e


@pytest.mark.parametrize("kind", ["normal", "aat", "few", "const", "wide"])
@pytest.mark.parametrize("K", [33, 57, 64, 300, 512, 545, 3249])
def test_wide_digits_no_less_accurate_than_seven_bit(ctx, K, kind, digits=7):
    A, B = operands(kind, K)
    ref = A.astype(numpy.longdouble) @ B.astype(numpy.longdouble)
    (a, ea), (b, eb) = seven_bit(A, digits), seven_bit(B.T, digits)
    old = sum((a[s - 1] @ b[t - 1].T).astype(numpy.longdouble)
              for s in range(1, digits) for t in range(1, digits) if s + t <= digits)
    old = old * numpy.longdouble(2) ** (ea[:, None] + eb[None, :])
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, ref.shape)
    ctx.check(ctx.L.kvft_gemm(ctx.h, A.shape[0], B.shape[1], K, 1, _lib.PREC_FP64_TC, digits,
                              dA.ptr, dB.ptr, dC.ptr), "kvft_gemm")
    bound = abs(A).max(1)[:, None] * abs(B).max(0)[None, :]
    err, err7 = abs(dC.to_host() - ref) / bound, abs(old - ref) / bound
    assert (err ** 2).sum() <= (err7 ** 2).sum()
    assert err.max() <= err7.max()


# Few output tiles: with four or more levels K is cut into ranges of 256 and
# more that add into C.  Either side of the first cut (512), one k-block more,
# a long K with one, several and enough tiles, a batch.  Tolerances: those of
# the digit counts (norm-wise), which do not depend on how K is cut.
@pytest.mark.parametrize("digits,tol", [(4, 5e-7), (5, 5e-9), (6, 5e-11), (7, 5e-12)])
@pytest.mark.parametrize("M,N,K,batch", [(70, 40, 511, 1), (70, 40, 512, 1), (70, 40, 545, 1),
                                         (37, 21, 16317, 1), (130, 100, 2049, 3),
                                         (600, 1, 700, 1), (2000, 700, 600, 1)])
def test_split_k_with_few_tiles(ctx, M, N, K, batch, digits, tol):
    rng = numpy.random.default_rng(M + N + K)
    A, B = rng.standard_normal((batch, M, K)), rng.standard_normal((batch, K, N))
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray.from_host(ctx, numpy.full((batch, M, N), numpy.nan))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    bound = abs(A).max(2)[:, :, None] * abs(B).max(1)[:, None, :] * K
    assert (abs(dC.to_host() - A @ B) <= tol * bound).all()


# Rows of 257 to 4096 values are packed by clusters, longer ones in two
# passes: K at the edges of both, of the cluster sizes and of the slabs (odd
# K, one value in the last slab), rows at the edges of the 16- and 32-row tiles, an
# all-zero row on each side, one operand contiguous along its rows and one
# along K.  A row scaled by a power of two gives exactly the scaled product.
@pytest.mark.parametrize("digits,tol", [(3, 5e-5), (6, 5e-11), (7, 5e-12)])
@pytest.mark.parametrize("M,N,K,batch", [(31, 33, 257, 1), (64, 97, 511, 3), (33, 40, 513, 1),
                                         (777, 130, 777, 1), (65, 32, 2047, 2), (40, 70, 2049, 1),
                                         (32, 65, 3249, 2), (17, 16, 4095, 1), (64, 33, 4096, 1),
                                         (33, 64, 4097, 1), (5000, 40, 361, 4)])
def test_pack_long_rows(ctx, M, N, K, batch, digits, tol):
    rng = numpy.random.default_rng(M + N + K)
    A = rng.standard_normal((batch, M, K)) * numpy.exp(3 * rng.standard_normal((batch, M, 1)))
    B = rng.standard_normal((batch, K, N)) * numpy.exp(3 * rng.standard_normal((batch, 1, N)))
    A[:, 2] = 0.0
    B[:, :, 1] = 0.0
    A[:, 5] = A[:, 4] * 2.0 ** 40
    A[:, 7] = 0.0
    A[:, 7, K - 1] = 3.0                          # the last value alone sets the exponent
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, (batch, M, N))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    C = dC.to_host()
    bound = abs(A).max(2)[:, :, None] * abs(B).max(1)[:, None, :] * K
    assert (abs(C - A @ B) <= tol * bound).all()
    assert not C[:, 2].any() and not C[:, :, 1].any()
    if digits == 3 and K <= 2048:                 # one K range: one fixed order
        assert (C[:, 5] == C[:, 4] * 2.0 ** 40).all()


# A long K against few rows: one operand is converted inside the contraction
# (not packed).  Rows and columns at the edges (1, 48 / 49, 64, and 65, which
# packs), K just beyond the packed lengths, odd, at and beside the k-blocks and
# ranges; either side converted (the other one has more than 64 rows or both
# fit); products that give every SM a K range and just too few or too many;
# zero rows.  Tolerances: those of the digit counts.
@pytest.mark.parametrize("digits,tol", [(2, 2e-3), (3, 5e-5), (5, 5e-9), (6, 5e-11), (7, 5e-12)])
@pytest.mark.parametrize("M,N,K,batch", [(57, 57, 4097, 60), (1, 64, 4129, 51), (64, 1, 5000, 60),
                                         (48, 49, 6143, 60), (49, 48, 6144, 51),
                                         (64, 65, 4999, 52), (65, 64, 5001, 52),
                                         (19, 19, 6859, 60), (8, 9, 70001, 6),
                                         (57, 57, 4097, 50), (37, 21, 28749, 1),
                                         (3, 5, 4200, 303), (3, 5, 4200, 304)])
def test_converted_operand(ctx, M, N, K, batch, digits, tol):
    rng = numpy.random.default_rng(M + N + K)
    A = rng.standard_normal((batch, M, K)) * numpy.exp(3 * rng.standard_normal((batch, M, 1)))
    B = rng.standard_normal((batch, K, N)) * numpy.exp(3 * rng.standard_normal((batch, 1, N)))
    A[:, M // 2] = 0.0
    B[0, :, N // 2] = 0.0
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray.from_host(ctx, numpy.full((batch, M, N), numpy.nan))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    C = dC.to_host()
    bound = abs(A).max(2)[:, :, None] * abs(B).max(1)[:, None, :] * K
    assert (abs(C - A @ B) <= tol * bound).all()
    assert not C[:, M // 2].any() and not C[0, :, N // 2].any()


# Rows whose values lie close together: their leading digits agree, so the
# products of a level all have one sign and a level's sum grows with K times
# the largest product.  Kinds by the digits that agree: two, three and four of
# the wide ones, and values of a few close-by numbers.  K at and beside the
# read-out length, in one range and several, packed and (the batch)
# converted inside the contraction.  The bound is the one of the test above.
def close_operands(kind, K, batch, M):
    rng = numpy.random.default_rng(K + batch)

    def draw(shape):
        n, u = rng.standard_normal(shape), rng.random(shape)
        return {"rel 1e-4": lambda: 1.9605 * (1 + 1e-4 * n), "rel 1e-6": lambda: 1.9605 * (1 + 1e-6 * n),
                "half": lambda: 0.49 + 2e-4 * u, "one": lambda: 0.98 + 5e-4 * n,
                "pi": lambda: numpy.pi * (1 + 1e-3 * u),
                "three": lambda: numpy.array([1.9591, 1.9602, 1.9608])[rng.integers(0, 3, shape)],
                # leading digits 127, 255, 255
                "top": lambda: 127 * 2.0 ** -8 + 255 * 2.0 ** -17 + 255 * 2.0 ** -26 + 2.0 ** -35 * u,
                }[kind]()

    return draw((batch, M, K)), draw((batch, K, M))


@pytest.mark.parametrize("kind", ["rel 1e-4", "rel 1e-6", "half", "one", "pi", "three", "top"])
@pytest.mark.parametrize("K,batch,M", [(128, 1, 48), (129, 1, 48), (257, 1, 48), (361, 1, 48),
                                       (512, 1, 48), (1024, 1, 48), (3249, 1, 24), (4129, 60, 8)])
def test_wide_digits_of_close_values(ctx, K, batch, M, kind, digits=7):
    A, B = close_operands(kind, K, batch, M)
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, (batch, M, M))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, M, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    C = dC.to_host()
    s = s7 = m = m7 = 0.0
    for b in range(batch):
        ref = A[b].astype(numpy.longdouble) @ B[b].astype(numpy.longdouble)
        (x, ex), (y, ey) = seven_bit(A[b], digits), seven_bit(B[b].T, digits)
        old = sum((x[i - 1] @ y[j - 1].T).astype(numpy.longdouble)
                  for i in range(1, digits) for j in range(1, digits) if i + j <= digits)
        old = old * numpy.longdouble(2) ** (ex[:, None] + ey[None, :])
        bound = abs(A[b]).max(1)[:, None] * abs(B[b]).max(0)[None, :]
        err, err7 = abs(C[b] - ref) / bound, abs(old - ref) / bound
        s, s7 = s + (err ** 2).sum(), s7 + (err7 ** 2).sum()
        m, m7 = max(m, err.max()), max(m7, err7.max())
    assert s <= s7
    assert m <= m7


# Integers whose digits and products the kept levels hold in full: the running
# sums are integers, so the product is exact, up to the last bit of a rounding
# to FP64 that does not happen.  K at and beside the read-out length, in one range
# and several; rows and columns scaled by powers of two, whose product is then
# exactly the scaled one, or zero or not finite where FP64 ends.
@pytest.mark.parametrize("M,N,K,batch", [(48, 48, 65, 1), (48, 33, 128, 1), (130, 50, 129, 2),
                                         (48, 48, 361, 1), (300, 200, 1025, 1), (64, 64, 2049, 60),
                                         (33, 17, 4097, 60), (2000, 700, 600, 1)])
def test_wide_digits_of_integers(ctx, M, N, K, batch, digits=7):
    rng = numpy.random.default_rng(M + N + K)
    A = rng.integers(-2 ** 20 + 1, 2 ** 20, (batch, M, K)).astype(float)
    B = rng.integers(-2 ** 20 + 1, 2 ** 20, (batch, K, N)).astype(float)
    B[:, :, 0] = abs(B[:, :, 0])
    A[:, 0] = abs(A[:, 0])                           # the largest sums
    ref = A @ B                                      # below 2^53: exact
    a = rng.integers(-300, 300, (batch, M, 1)).astype(float)
    b = rng.integers(-300, 300, (batch, 1, N)).astype(float)
    a[:, 1], b[:, :, 1], a[:, 2], b[:, :, 2] = -560, -560, 560, 560
    A, B = A * 2.0 ** a, B * 2.0 ** b
    dA, dB = _lib.DeviceArray.from_host(ctx, A), _lib.DeviceArray.from_host(ctx, B)
    dC = _lib.DeviceArray(ctx, (batch, M, N))
    ctx.check(ctx.L.kvft_gemm(ctx.h, M, N, K, batch, _lib.PREC_FP64_TC, digits, dA.ptr, dB.ptr,
                              dC.ptr), "kvft_gemm")
    with numpy.errstate(over="ignore", under="ignore"):
        ref = numpy.ldexp(ref, (a + b).astype(int))
    ref[abs(ref) < 2.0 ** -1022] = 0.0
    C, fin = dC.to_host(), numpy.isfinite(ref)
    assert (C[fin] == ref[fin]).all()
    # sums of K ranges that each end beyond FP64 may have both signs
    assert not numpy.isfinite(C[~fin]).any()


def test_wide_digits_of_a_long_sum(ctx, K=600001, batch=304):
    """A sum that runs through every read-out of a K no unit shares, with the
    largest terms of one sign.  Tolerance: that of the digit count."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    A, B = (0.49 + 0.0099 * torch.rand((batch, K), generator=g, device="cuda", dtype=torch.float64)
            for _ in range(2))
    C = torch.full((batch,), float("nan"), device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    a, b, c = (_lib.DeviceArray(ctx, t.shape, ptr=t.data_ptr(), owner=t) for t in (A, B, C))
    ctx.check(ctx.L.kvft_gemm(ctx.h, 1, 1, K, batch, _lib.PREC_FP64_TC, 7, a.ptr, b.ptr, c.ptr),
              "kvft_gemm")
    ref = (A * B).sum(1)
    assert (abs(C - ref) <= 5e-12 * 0.25 * K).all()

// Contractions of a big tensor with a small matrix on the tensor cores: the
// n^5 class of the residual, C[r, j] (+)= alpha sum_k A[r, k] B[k, j] with r a
// composite of up to three orbital indices (10^4..10^6 values) and k, j single
// ones (K, N <= 64).  The arithmetic is the digit splitting of kvft_tc.cu,
// product for product.
//
// Such a contraction reads and writes a big tensor once and does little in
// between, so nothing may pass over memory twice: the FP64 rows of A are
// packed inside the kernel (a row has at most 64 values, so its exponent is
// known when it is read), where the general kernel reads digit planes that
// two other launches wrote.  The small matrices (N rows of K) come as digit
// planes from kv_tc_pack.
//
// One CTA walks a contiguous range of items (block of C, batch entry, 128-row
// tile); per tile
//   1. all threads turn the FP64 values they hold in registers into digits,
//      stored straight into the swizzled shared-memory layout that the MMA
//      reads (K-major);
//   2. one thread issues the tile's MMAs (every level of every k-step) and the
//      TMA load of the next small matrix;
//   3. all threads issue the global loads of their next A values (they arrive
//      while the tile is finished);
//   4. all threads wait for the accumulators and write C: level sums to FP64,
//      stored, or added by L2 reductions.
// A tau-independent A (the integrals) is packed once per tile and used for
// every tau point of the range.
//
// A's values are read along whichever of its row index and k is contiguous,
// and C is written along whichever of its row index and j is (through a
// per-warp transpose in shared memory for j), so both streams coalesce.
//
// K > 32 takes 64-deep tiles (128-byte swizzle), else 32-deep ones (64-byte);
// two CTAs of 256 threads per SM where shared memory and TMEM allow (K <= 32,
// or up to three levels), else one of 512.
//
// What bounds it: the chain of each tile (convert, MMA, drain, write; 8000 to
// 11000 clocks with two CTAs per SM overlapping theirs), of which the writes
// and the conversions are instructions and the MMAs are latency (dependent
// accumulations, about 250 clocks each).  Memory traffic would allow 3-4x.
// Measured, ten contractions of one update, packing included, before (digit
// planes through memory, general tiles) and now: 54 spin orbitals, 10 tau
// points, seven levels 8.9 -> 2.3 ms; 66, 16 points, three levels 11.8 -> 5.9;
// 38, 16 points, six levels 5.4 -> 1.3; 114, 3 points, three levels 12.7 ->
// 8.4, six levels 22 -> 13.8.
#include "kvft_tc.h"

namespace {

constexpr int KMAX = 64, NMAX = 64;
constexpr int MMAS = 10;                     // MMAs of a k-step (at most two per A plane)

struct ThinParams {
    int M, N, K, TN;             // TN: N rounded up to 16 (columns of one level)
    int items, batch, mt;
    int shared_a;                // A does not depend on the batch entry
    int a_rows_fast, c_rows_fast;
    int nbuf;                    // shared-memory buffers of the small matrix
    const double *A;
    KIdx Ar;
    long long ks, a_bst;         // stride of k
    double *C;
    KIdx Cr;
    long long cs, c_bst;         // stride of j
    double alpha, beta;
    int store;                   // first source: 0 adds (beta = 1), 1 stores, 2 general beta
    int alpha_pow2;
    int krow0;                   // row part of a value's exponent field, see f64_hi
    unsigned alpha_sign;
    const int *eb;               // exponents of the small matrices' rows
    int eb_bst, b_batch_rows, b_plane_rows;
    int *err;
    FastDiv dv_mt, dv_batch;
    KIdxDiv dv_ar, dv_cr;
    int beg[KV_MAXPROD + 1];
    long long coff[KV_MAXPROD], oa[KV_MAXPROD];
    int brow[KV_MAXPROD], bex[KV_MAXPROD];
};

// High word of x 2^k (x a finite FP32 value, its low word is the bits << 29):
// the exponent and top mantissa bits of x moved to their FP64 place plus kk =
// (k + 1023 - 127) << 20, then x's sign.  Zero for x = 0 and for results
// below 2^-1022.  All integer operations: the FP64 pipe (16 clocks a warp)
// is left to the additions that need it.
__device__ __forceinline__ double f64_of(float x, int kk, uint32_t sgn) {
    const uint32_t u = __float_as_uint(x);
    int h = (int)((u & 0x7FFFFFFFu) >> 3) + kk;
    if (x == 0.f || h < (1 << 20)) h = 0;
    return __hiloint2double((int)((uint32_t)h | ((u ^ sgn) & 0x80000000u)), (int)(u << 29));
}

// One step of a CTA: source `src` of the item (cb, b, mt).
struct Step {
    int item, src, cb, b, mt;
    __device__ __forceinline__ void at(const ThinParams &p, int it) {
        item = it;
        const int q = p.shared_a ? p.dv_batch.div(it) : p.dv_mt.div(it);
        const int fast = it - q * (p.shared_a ? p.batch : p.mt);
        cb = p.shared_a ? p.dv_mt.div(q) : p.dv_batch.div(q);
        const int slow = q - cb * (p.shared_a ? p.mt : p.batch);
        b = p.shared_a ? fast : slow;
        mt = p.shared_a ? slow : fast;
        src = p.beg[cb];
    }
    __device__ __forceinline__ void next(const ThinParams &p) {
        if (++src < p.beg[cb + 1]) return;
        item++;
        int &fast = p.shared_a ? b : mt;
        if (++fast < (p.shared_a ? p.batch : p.mt)) src = p.beg[cb];
        else if (item < p.items) at(p, item);
    }
};

__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w)
                 : "memory");
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t x) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}

// Shared-memory bytes: 1 KB alignment slack, A planes, B buffers, per-warp
// transpose tiles (32 x 9 doubles), row maxima, row exponents, column
// exponents of two buffers, barriers, four words and the MMA table.
__host__ __device__ constexpr size_t thin_smem(int kbt, int S, int nt, int TN, int nbuf) {
    return 1024 + (size_t)S * kbt * 2 * (TM + nbuf * TN) + (size_t)(nt / 32) * 32 * 9 * 8 +
           (size_t)(nt / 128 + 1) * TM * 4 + 2 * NMAX * 4 + 4 * 8 + 16 + MMAS * 16;
}

__host__ __device__ constexpr int thin_threads(int kbt, int D) {
    return kbt == 64 && D > 3 ? 512 : 256;
}

template <int KBT, int DL>
__global__ void __launch_bounds__(thin_threads(KBT, DL), thin_threads(KBT, DL) == 512 ? 1 : 2)
tc_thin_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ ThinParams p) {
    if (!kv_depend()) return;
    constexpr int NT = thin_threads(KBT, DL);
    using G = Dig<DL>;
    constexpr int S = G::S, nl = G::NL;
    constexpr int PLANE = TM * KBT * 2;
    constexpr int NKP = NT / TM;                 // threads per row (a_rows_fast)
    constexpr int VP = KBT / NKP;                // values of A per thread
    constexpr int NW = NT / 32;
    constexpr bool FF = DL > 3;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bplane = p.TN * KBT * 2;
    uint8_t *sA = smem, *sB = smem + S * PLANE;
    double *tr = (double *)(sB + (size_t)p.nbuf * S * bplane);      // [NW][32][9]
    int *rmax = (int *)(tr + NW * 32 * 9);                           // [NKP][TM]
    int *rexp = rmax + NKP * TM;                                     // [TM]
    int *cexp = rexp + TM;                                           // [2][NMAX]
    uint64_t *bars = (uint64_t *)(cexp + 2 * NMAX);                  // B full x 2, accumulators
    uint32_t *tmem_slot = (uint32_t *)(bars + 4);
    volatile int *s_fail = (volatile int *)(tmem_slot + 1);
    uint4 *mma = (uint4 *)(tmem_slot + 4);                           // [MMAS]
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int ncols = nl * p.TN <= 32 ? 32 : nl * p.TN <= 64 ? 64 : nl * p.TN <= 128 ? 128
                      : nl * p.TN <= 256 ? 256 : 512;
    // The MMAs of one 16-deep k-step: A plane q against B planes t0.. (adjacent
    // in shared memory) into levels q + t0.. (adjacent in TMEM), N <= 256.
    // The widths are run-time values, so the issuing thread reads them from a
    // table: deriving them per tile took it 300 clocks an MMA.
    const int pmax = 256 / p.TN;
    int nmma = 0;
#pragma unroll
    for (int q = 1; q <= S; q++) {
        const int tmax = nl + 1 - q;
        for (int t0 = 1; t0 <= tmax; t0 += pmax, nmma++)
            if (tid == 0)
                mma[nmma] = make_uint4((q + t0 - 2) * p.TN, ((q - 1) * PLANE) >> 4,
                                       ((t0 - 1) * bplane) >> 4,
                                       idesc_of(min(pmax, tmax - t0 + 1) * p.TN) |
                                           (q > 1 ? 0x80000000u : 0u));
    }
    if (tid == 0) {
        *s_fail = 0;
        for (int i = 0; i < 3; i++) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    const int row = (warp & 3) * 32 + lane;      // A row (a_rows_fast) and TMEM lane
    const int part = warp >> 2;                  // k part / column part
    const int kpad = (p.K + 15) & ~15;
    const uint32_t sA32 = smem_u32(sA), sB32 = smem_u32(sB);
    const uint64_t dA0 = desc_of<KBT>(sA32), dB0 = desc_of<KBT>(sB32);

    // ---- this CTA's range ----
    const int i0 = (int)((long long)p.items * blockIdx.x / gridDim.x);
    const int i1 = (int)((long long)p.items * (blockIdx.x + 1) / gridDim.x);

    unsigned long long pre[VP];                  // the next tile's A values
    // values of one tile: a_rows_fast -- row `row`, the 8-deep k chunks c NKP +
    // part; otherwise rows of this warp, a pair of k per lane (half a warp per
    // row at KBT = 32)
    constexpr int RW = TM / NW;                  // rows per warp
    constexpr int RI = KBT == 64 ? 1 : 2;        // rows per load step
    auto fetch = [&](const Step &s) {
        const double *base = p.A + p.oa[s.src] + (p.shared_a ? 0 : (long long)s.b * p.a_bst);
        const int m0 = s.mt * TM;
        if (p.a_rows_fast) {
            const int m = m0 + row;
            const bool ok = m < p.M;
            const double *q0 = base + (ok ? p.dv_ar.off(p.Ar, m) : 0);
            const int kn = ok ? p.K : 0;
#pragma unroll
            for (int c = 0; c < VP / 8; c++) {
                const int k0 = (c * NKP + part) * 8;
                const double *q = q0 + (long long)k0 * p.ks;
#pragma unroll
                for (int v = 0; v < 8; v++) {
                    pre[8 * c + v] = k0 + v < kn
                                         ? (unsigned long long)__double_as_longlong(__ldg(q)) : 0ull;
                    q += p.ks;
                }
            }
        } else {
            const int r = m0 + warp * RW + (lane % RW);
            const long long ro = r < p.M ? p.dv_ar.off(p.Ar, r) : -1;
            const int k = 2 * (KBT == 64 ? lane : lane % 16);
            const long long ko = (long long)k * p.ks;
#pragma unroll
            for (int v = 0; v < VP / 2; v++) {
                const long long o = __shfl_sync(0xffffffffu, ro,
                                                v * RI + (KBT == 64 ? 0 : lane / 16));
                const double *q = base + o + ko;
                pre[2 * v] = o >= 0 && k < p.K
                                 ? (unsigned long long)__double_as_longlong(__ldg(q)) : 0ull;
                pre[2 * v + 1] = o >= 0 && k + 1 < p.K
                                     ? (unsigned long long)__double_as_longlong(__ldg(q + p.ks))
                                     : 0ull;
            }
        }
    };
    // swizzled byte offset of 16-byte chunk c of row r within a plane
    auto chunk = [&](int r, int c) -> uint32_t {
        return (uint32_t)(r * KBT * 2 + ((c ^ (KBT == 64 ? r & 7 : (r >> 1) & 3)) << 4));
    };
    auto load_b = [&](int buf, const Step &s) {  // one thread
        mbar_expect_tx(smem_u32(&bars[buf]), (uint32_t)(S * bplane));
        const int y = p.brow[s.src] + s.b * p.b_batch_rows;
        for (int t = 0; t < S; t++)
            tma_load_2d(sB32 + (uint32_t)((buf * S + t) * bplane), &tmB, 0, y + t * p.b_plane_rows,
                        smem_u32(&bars[buf]));
    };
    auto bkey = [&](const Step &s) { return p.bex[s.src] + s.b * p.eb_bst; };
    auto same_a = [&](const Step &x, const Step &y) {
        return x.mt == y.mt && p.oa[x.src] == p.oa[y.src] && (p.shared_a || x.b == y.b);
    };

    uint32_t phB = 0, phD = 0;                   // phB: one bit per buffer
    int curB = -1, buf = p.nbuf - 1;
    bool pendB = false;                          // the next B is already on its way
    bool newA = true;
    int nMma = 0;
    Step s;
    if (i0 < i1) {
        s.at(p, i0);
        fetch(s);
    }
    while (i0 < i1 && s.item < i1) {
        // ---- operands of this step ----
        const int kb = bkey(s);
        const bool newB = kb != curB;
        if (newB) {
            buf = p.nbuf == 2 ? buf ^ 1 : 0;
            if (!pendB && tid == 0) load_b(buf, s);
            pendB = false;
            curB = kb;
            if (tid < p.N) cexp[buf * NMAX + tid] = exp_of(p.eb[kb + tid]) * (1 << 20);
        }
        if (newA) {
            if (p.a_rows_fast) {
                int e = -2000;
#pragma unroll
                for (int v = 0; v < VP; v++) e = max(e, raw_exp(pre[v]));
                rmax[part * TM + row] = e;
                __syncthreads();
                e = rmax[row];
#pragma unroll
                for (int q = 1; q < NKP; q++) e = max(e, rmax[q * TM + row]);
                e = exp_of(e);
                if (part == 0) rexp[row] = p.krow0 + e * (1 << 20);
#pragma unroll
                for (int c = 0; c < VP / 8; c++) {
                    if ((c * NKP + part) * 8 >= kpad) break;
                    uint32_t w[4][S];
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        digit_words<DL>(pre[8 * c + 2 * j], pre[8 * c + 2 * j + 1], e, w[j]);
                    const uint32_t a = sA32 + chunk(row, c * NKP + part);
#pragma unroll
                    for (int t = 0; t < S; t++)
                        sts128(a + t * PLANE, w[0][t], w[1][t], w[2][t], w[3][t]);
                }
            } else {
                const int kp = KBT == 64 ? lane : lane % 16;          // pair of k
#pragma unroll
                for (int v = 0; v < VP / 2; v++) {
                    const int r = warp * RW + v * RI + (KBT == 64 ? 0 : lane / 16);
                    int e = max(raw_exp(pre[2 * v]), raw_exp(pre[2 * v + 1]));
                    if constexpr (KBT == 64) {
                        e = __reduce_max_sync(0xffffffffu, e);
                    } else {
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1)
                            e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
                    }
                    e = exp_of(e);
                    if (kp == 0) rexp[r] = p.krow0 + e * (1 << 20);
                    if (2 * kp < kpad) {
                        uint32_t w[S];
                        digit_words<DL>(pre[2 * v], pre[2 * v + 1], e, w);
                        const uint32_t a = sA32 + chunk(r, kp >> 2) + (kp & 3) * 4;
#pragma unroll
                        for (int t = 0; t < S; t++) sts32(a + t * PLANE, w[t]);
                    }
                }
            }
        }
        Step n = s;
        n.next(p);
        const bool more = n.item < i1;
        const bool nextB = more && bkey(n) != curB && p.nbuf == 2;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        // ---- the tile's MMAs ----
        if (tid == 0) {
            bool ok = *s_fail == 0;
            if (newB && !mbar_wait(smem_u32(&bars[buf]), (phB >> buf) & 1)) {
                ok = false;
                mbar_wait(smem_u32(&bars[buf]), (phB >> buf) & 1);   // once more: it must land
            }
            if (ok) {
                fence_after();
                const uint64_t dB = dB0 + (((uint32_t)(buf * S * bplane)) >> 4);
#pragma unroll
                for (int kk = 0; kk < KBT / 16; kk++) {
                    if (kk * 16 >= kpad) break;
                    for (int i = 0; i < nmma; i++) {
                        const uint4 d = mma[i];
                        umma(tmem + d.x, dA0 + d.y + 2 * kk, dB + d.z + 2 * kk, d.w & 0x7FFFFFFFu,
                             (kk > 0 || d.w >> 31) ? 1u : 0u);
                    }
                }
                umma_commit(smem_u32(&bars[2]));
            } else {
                atomicExch(p.err, 7);
                *s_fail = 1;
            }
            if (nextB) load_b(buf ^ 1, n);
        }
        if (newB) phB ^= 1u << buf;
        if (nextB) pendB = true;
        nMma++;
        // ---- the next tile's loads ----
        newA = more && !same_a(s, n);
        if (newA) fetch(n);
        // ---- C ----
        const int m = s.mt * TM + row;
        const long long roff = m < p.M ? p.dv_cr.off(p.Cr, m) : -1;
        double *Cb = p.C + p.coff[s.cb] + (long long)s.b * p.c_bst;
        const int store = s.src == p.beg[s.cb] ? p.store : 0;
        const int krow = rexp[row];
        const int4 *ce = (const int4 *)(cexp + buf * NMAX);
        {
            const bool got = *s_fail == 0 && mbar_wait(smem_u32(&bars[2]), phD);
            phD ^= 1;
            // one verdict per warp: tcgen05.ld below needs every lane
            if (__any_sync(0xffffffffu, !got)) {
                if (lane == 0) {
                    atomicExch(p.err, 8);
                    *s_fail = 1;
                }
            }
            __syncwarp();
            if (!__any_sync(0xffffffffu, !got)) {
                fence_after();
                const uint32_t tb = tmem + ((uint32_t)((warp & 3) * 32) << 16);
                for (int g = part; g * 8 < p.N; g += NKP) {
                    uint32_t r[nl][8];
#pragma unroll
                    for (int l = 0; l < nl; l++) tmem_ld<8>(tb + l * p.TN + g * 8, r[l]);
                    tmem_wait_ld();
                    const int4 c0 = ce[2 * g], c1 = ce[2 * g + 1];
                    const int kc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                    double v[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int kk = krow + kc[j];
                        float hi = __uint_as_float(r[0][j]);
                        if constexpr (!FF) {
                            if (nl > 1) hi += __uint_as_float(r[nl > 1 ? 1 : 0][j]);
                            v[j] = f64_of(hi, kk, p.alpha_sign);
                        } else {
                            float lo = 0.f, e;
#pragma unroll
                            for (int l = 1; l < nl; l++) {
                                two_sum(hi, __uint_as_float(r[l][j]), hi, e);
                                lo += e;
                            }
                            v[j] = f64_of(hi, kk, p.alpha_sign) + f64_of(lo, kk, p.alpha_sign);
                        }
                    }
                    if (!p.alpha_pow2) {
#pragma unroll
                        for (int j = 0; j < 8; j++) v[j] *= p.alpha;
                    }
                    const int jn = min(8, p.N - g * 8);
                    if (p.c_rows_fast) {
                        double *d = Cb + roff + (long long)(g * 8) * p.cs;
                        if (roff >= 0) {
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                if (j < jn) {
                                    if (store == 0) atomicAdd(d, v[j]);
                                    else *d = store == 1 ? v[j] : fma(p.beta, *d, v[j]);
                                }
                                d += p.cs;
                            }
                        }
                    } else {
                        // transpose 32 rows x 8 columns: 8 lanes then write
                        // one row's adjacent columns
                        double *tw = tr + warp * 32 * 9;
#pragma unroll
                        for (int j = 0; j < 8; j++) tw[lane * 9 + j] = v[j];
                        __syncwarp();
                        const int j = lane % 8;
                        const long long co = (long long)(g * 8 + j) * p.cs;
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const int rr = i * 4 + lane / 8;
                            const long long ro = __shfl_sync(0xffffffffu, roff, rr);
                            if (ro >= 0 && j < jn) {
                                double *d = Cb + ro + co;
                                const double x = tw[rr * 9 + j];
                                if (store == 0) atomicAdd(d, x);
                                else *d = store == 1 ? x : fma(p.beta, *d, x);
                            }
                        }
                        __syncwarp();
                    }
                }
            }
        }
        fence_before();
        __syncthreads();
        fence_after();
        if (*s_fail) break;
        s = n;
    }
    // a B load still on its way lands before the CTA leaves; the MMAs issued
    // have completed (bars[2] was waited for) unless a wait expired, and then
    // the commit gets one more bounded wait
    if (tid == 0) {
        if (pendB && !mbar_wait(smem_u32(&bars[buf ^ 1]), (phB >> (buf ^ 1)) & 1))
            atomicExch(p.err, 9);
        if (*s_fail && nMma > 0 && !mbar_wait(smem_u32(&bars[2]), phD ^ 1)) atomicExch(p.err, 10);
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols)
                     : "memory");
    }
}

constexpr size_t THIN_SMEM_CAP = 226 * 1024;

template <int KBT, int DL>
int launch_thin(kvft_ctx *ctx, const CUtensorMap &mb, ThinParams &p) {
    constexpr int S = Dig<DL>::S, NT = thin_threads(KBT, DL);
    auto kern = tc_thin_kernel<KBT, DL>;
    p.nbuf = 2;
    if (thin_smem(KBT, S, NT, p.TN, 2) > THIN_SMEM_CAP) p.nbuf = 1;
    size_t smem = thin_smem(KBT, S, NT, p.TN, p.nbuf);
    // CTAs that share an SM must fit its TMEM together
    const int cols = Dig<DL>::NL * p.TN;
    int per = NT == 512 || cols > 256 ? 1 : 2;
    if (per == 1) smem = std::max(smem, (size_t)118 * 1024);
    else if (2 * smem > THIN_SMEM_CAP) per = 1;
    KV_TRY(kv_smem_optin(ctx, kern, THIN_SMEM_CAP));
    const int grid = std::min(p.items, per * ctx->sm_count);
    KvProfScope prof(ctx, ctx->gemm_cat, ctx->gemm_work);
    kv_launch(ctx, kern, grid, NT, smem, mb, p);
    return kv_launch_check(ctx, "tc_thin");
}

bool single(const KIdx &x) { return x.size[0] == 1 && x.size[1] == 1; }

}  // namespace

// The shapes it takes: K and N single indices of at most 64 values, and
// enough rows that a tile per SM exists (below that the general kernel's
// launches cost the same and it splits K where that is long).  An operand
// that is contiguous along neither its rows nor k (t1 <mn||je>, rows (m, e,
// j)) is read in 32-byte sectors of which 8 bytes count; with K > 32 that
// costs more than reading packed planes (114 spin orbitals, three tau points,
// three levels: 1.41 against 0.84 ms; with K = 27 it is 0.30 against 0.55).
bool kv_thin_fits(int M, int N, int K, int batch, const KMat &A, const KMat &B, const KOut &C) {
    if (K > 32 && A.c.st[2] != 1 && kidx_fast_stride(A.r) != 1) return false;
    return K >= 16 && K <= KMAX && N <= NMAX && M > NMAX && M >= 4 * N && single(A.c) &&
           single(B.r) && single(B.c) && single(C.c) && (long long)M * batch >= 2048;
}

int kv_gemm_thin(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
                 const KMat &B, double beta, const KOut &C, int D, const KvProds &g) {
    const int S = dig_planes(D);
    const int kbt = K <= 32 ? 32 : 64;
    const int nbB = B.bst ? batch : 1;
    int wb[KV_MAXPROD];
    const PackView vb = kv_tc_group_view(B.p, B.c, B.r, B.bst, B.stable, nbB, g.n, g.ob, wb);
    Packed pb;
    KV_TRY(kv_tc_pack(ctx, "tc_pack_b", vb, N, K, vb.nsub * nbB, D, &pb));
    const long long rows = (long long)vb.nsub * nbB * S * N;
    const KvGroupTab tab = kv_group_tab(g, false);
    ThinParams p;
    p.M = M, p.N = N, p.K = K;
    p.TN = (N + 15) & ~15;
    p.batch = batch;
    p.mt = (M + TM - 1) / TM;
    const long long items = (long long)tab.ncb * batch * p.mt;
    if (rows > 0x7FFFFFFFLL || items > 0x7FFFFFFFLL)
        return kv_fail(ctx, KVFT_EINVAL, "tensor-core gemm: operand too large");
    p.items = (int)items;
    p.shared_a = A.bst == 0;
    p.ks = A.c.st[2];
    p.a_rows_fast = !(p.ks == 1 && kidx_fast_stride(A.r) != 1);
    p.cs = C.c.st[2];
    p.c_rows_fast = !(p.cs == 1 && kidx_fast_stride(C.r) != 1);
    p.A = A.p, p.Ar = A.r, p.a_bst = A.bst;
    p.C = C.p, p.Cr = C.r, p.c_bst = C.bst;
    p.alpha = alpha, p.beta = beta;
    p.store = beta == 1.0 ? 0 : beta == 0.0 ? 1 : 2;
    int alpha_exp = 0;
    p.alpha_pow2 = kv_tc_pow2(alpha, &alpha_exp, &p.alpha_sign);
    const int c2 = 2 * (D == 7 ? Dig<7>::C : Dig<6>::C);
    p.krow0 = (1023 - 127 - c2 + alpha_exp) * (1 << 20);
    p.eb = pb.ex;
    p.eb_bst = nbB > 1 ? N : 0;
    p.b_batch_rows = nbB > 1 ? S * N : 0;
    p.b_plane_rows = N;
    p.err = ctx->dflag;
    p.dv_mt = fastdiv(p.mt);
    p.dv_batch = fastdiv(batch);
    p.dv_ar = kidx_div(A.r), p.dv_cr = kidx_div(C.r);
    for (int c = 0; c <= tab.ncb; c++) p.beg[c] = tab.beg[c];
    for (int c = 0; c < tab.ncb; c++) p.coff[c] = tab.coff[c];
    for (int q = 0; q < g.n; q++) {
        const int y = wb[tab.prod[q]];
        p.oa[q] = g.oa[tab.prod[q]];
        p.brow[q] = y * nbB * S * N;
        p.bex[q] = y * nbB * N;
    }
    // bytes it must move: A as FP64, the small matrices' planes, C
    ctx->gemm_work = 8.0 * M * K * (p.shared_a ? 1.0 : batch) * g.n + 2.0 * S * N * K * nbB * g.n +
                     8.0 * M * N * (double)batch * g.n * (beta != 0.0 ? 2 : 1);
    CUtensorMap mb;
    KV_TRY(kv_tc_map(ctx, &mb, pb.planes, pb.K, pb.ld, rows, kbt, p.TN));
#define KV_THIN(d_)                                                       \
    case d_: return kbt == 64 ? launch_thin<64, d_>(ctx, mb, p) : launch_thin<32, d_>(ctx, mb, p);
    switch (D) {
        KV_THIN(2) KV_THIN(3) KV_THIN(4) KV_THIN(5) KV_THIN(6)
    default: return kbt == 64 ? launch_thin<64, 7>(ctx, mb, p) : launch_thin<32, 7>(ctx, mb, p);
    }
#undef KV_THIN
}

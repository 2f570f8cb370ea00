// FP64-accurate contractions on the 5th-generation tensor cores.
//
// GB300 issues ~2 FP64 FMAs per clock per SM but ~3600 BF16 MACs, so an FP64
// GEMM is rebuilt from exact BF16 digit products (an Ozaki-style error-free
// splitting):
//
//   * packing: every row r of A (and every column of B) is scaled by 2^-e_r
//     so that |y| < 1/2, then y = 2^-C sum_{s=1..S} P_s with balanced digits
//     P_s = d_s 2^(C - pos(s)), exact in BF16 (kvft_tc.h: digit schemes; base
//     128 up to D = 6, nine-bit digits at D = 7).  The digits are extracted
//     with integer arithmetic from the FP64 bit pattern.
//   * products: A B = 2^(e_m + e_n - 2 C) sum_{s,t} P_s^A P_t^B.  Pairs of one
//     level s + t have one weight; levels up to NL + 1 are kept.  A base-128
//     product is an integer below 2^12 (times a power of two), so an FP32
//     accumulator over K <= 2048 terms and two pairs is exact; nine-bit digits
//     are read out after 128 terms (kvft_tc.h: which levels that keeps exact).
//     Every level l = s + t has its own TMEM accumulator, at column
//     (l - 2) TN of the set, and the digit planes of a B tile lie one after
//     another in shared memory, so a single tcgen05.mma of A plane s against
//     B planes t0..t0+k-1 (N = k TN <= 256) adds each product into its own
//     level: 5 MMAs per 16-deep k-step for D = 7 instead of 15 pair MMAs,
//     which keeps the tensor core's shared-memory reads of A below the SM's
//     shared-memory bandwidth.
//   * epilogue: the accumulators are read from TMEM (tcgen05.ld), the K
//     chunks (K > KCHUNK) are summed in registers, and the tile is scaled by
//     2^(e_m + e_n - 2 C) alpha and written to the FP64 output view once.
// With D = 7 (15 pair products, five digits) the error is ~1e-13 of K max|A|
// max|B|, far inside the 1e-8 amplitude / 1e-10 Ha parity bounds; D = 3..5 is the
// mixed-precision form.
//
// Kernel: persistent, one CTA per SM walking output tiles; warp 0 = TMA
// producer, warp 1 = MMA issuer (and TMEM owner), warps 2..9 = epilogue; the
// epilogue of one tile overlaps the MMAs of the next.  Operands are staged by
// TMA (64-byte swizzle, 32-element k-blocks, every digit plane of a k-block
// per pipeline stage).  Every mbarrier wait is bounded by %globaltimer; on
// expiry the kernel records an error word and unwinds.
#include "kvft_tc.h"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

namespace {

constexpr int NEPI = 8;                       // epilogue warps: two per TMEM lane quadrant
constexpr int NTHREADS = 64 + 32 * NEPI;      // + TMA producer warp + MMA warp
constexpr int TMEM_COLS = 512;               // all of an SM's TMEM (one CTA per SM)
constexpr int KRANGE = 2048;                  // K range of a unit that adds by atomics
constexpr int GROUP_M = 8;                    // m-tiles per raster group (L2 reuse)
// Wide digits: unit 2^-WUNIT of the integer sums (level 2 has weight one; the
// last two levels are rounded to it, a sixteenth of their planes' own rounding
// over 128 terms), and the terms after which a sum (at most 2^14 a term) goes to
// C, below 2^63.
constexpr int WUNIT = 32, WFLUSH = 1 << 16;

// A converted in the kernel (CV): at most CV_M rows, NCV more warps that turn
// FP64 values into digits, CV_RING k-blocks of FP64 values in flight.
constexpr int CV_M = 64, NCV = 8;
constexpr int CV_RING = 3;

struct TcParams {
    int M, N;             // output extent
    int mt, nt;           // output tiles along M and N
    int units;            // work units: C blocks * mt * nt * batch * nsplit
    int nsplit;           // >1: each K range is its own unit, added into C by FP64 atomics
    long long c_split;    // or stored to its own copy of C, this far from the range before (0: added)
    int split_kb;         // k-blocks per K range
    int chunk_kb;         // k-blocks per K chunk (exactness bound)
    int flush_kb;         // wide digits: k-blocks after which the running sum goes to C
    int nkb_total;        // k-blocks of the padded K extent
    int S, D, NS;         // digit planes, levels, pipeline stages
    int Mp, Np;           // rows per digit plane of A / B
    int a_batch_rows, b_batch_rows;   // row offset between batch entries (0: shared)
    const int *ea, *eb;   // row exponents of A / column exponents of B
    int ea_bst, eb_bst;
    int batch;
    // the group's products by block of C: block c starts at coff[c] and its
    // sources are q = beg[c] .. beg[c + 1] - 1, each with the first plane row
    // (arow, brow) and first exponent (aex, bex) of its operand sub-blocks
    int beg[KV_MAXPROD + 1];
    long long coff[KV_MAXPROD];
    int arow[KV_MAXPROD], brow[KV_MAXPROD], aex[KV_MAXPROD], bex[KV_MAXPROD];
    double alpha, beta;
    int alpha_pow2;       // alpha = +-2^alpha_exp: folded into the exponent field
    int alpha_exp;
    unsigned alpha_sign;  // sign bit of alpha (bit 31 of the FP64 high word)
    KOut C;
    int *err;
    FastDiv dv_split, dv_perb, dv_gsz, dv_batch;   // nsplit, mt nt, GROUP_M nt, batch
    FastDiv dv_cr2, dv_cr1;               // C's row index: sizes of its fast components
    // converted A (CV): the FP64 operand, its products' offsets, its K index
    const double *A;
    long long ar;                         // stride of its rows
    KIdx Ac;
    KIdxDiv dv_ac;
    long long a_bst, oa[KV_MAXPROD];
    int K;
};

// A work unit: one output tile of one batch entry of one block of C over a
// k-block range, for every source of that block.  The sources run one after
// the other through the pipeline, each with its own accumulation and its own
// write to C (the first stores or scales, the others add): the same threads
// write the same elements, so the order is the program's.
struct Unit {
    int b, cb, m0, n0, kb0, kb1;
};

// Units are numbered split-fastest, then in raster groups of GROUP_M m-tiles
// (n-tiles walk inside a group), then by batch entry, then by block of C, so
// the CTAs that run at the same time share a few A row panels and sweep B
// once per group.  With a converted A the batch entries come first: they share
// B (the integrals), which is then read from memory once.
template <bool CV>
__device__ __forceinline__ Unit unit_of(const TcParams &p, int u, int tn) {
    static_assert(GROUP_M == 8, "raster groups of 8 m-tiles (shift and mask below)");
    Unit w;
    if constexpr (CV) {                   // one m-tile and one n-tile
        const int t = p.dv_batch.div(u);
        w.b = u - t * p.batch;
        w.cb = p.dv_split.div(t);
        w.m0 = w.n0 = 0;
        w.kb0 = (t - w.cb * p.nsplit) * p.split_kb;
        w.kb1 = min(w.kb0 + p.split_kb, p.nkb_total);
        return w;
    }
    const int t = p.dv_split.div(u);
    const int split = u - t * p.nsplit;
    const int per_b = p.mt * p.nt;
    const int bc = p.dv_perb.div(t);
    const int r = t - bc * per_b;
    w.cb = p.dv_batch.div(bc);
    w.b = bc - w.cb * p.batch;
    const int gsz = GROUP_M * p.nt;
    const int g = p.dv_gsz.div(r);
    const int first = g * GROUP_M;
    const int gm = min(GROUP_M, p.mt - first);
    const int rr = r - g * gsz;
    if (gm == GROUP_M) {
        w.m0 = (first + (rr & 7)) * TM;
        w.n0 = (rr >> 3) * tn;
    } else {                              // the last, short group
        w.m0 = (first + rr % gm) * TM;
        w.n0 = (rr / gm) * tn;
    }
    if (p.nsplit > 1) {
        w.kb0 = split * p.split_kb;
        w.kb1 = min(w.kb0 + p.split_kb, p.nkb_total);
    } else {
        w.kb0 = 0;
        w.kb1 = p.nkb_total;
    }
    return w;
}

// Shared-memory bytes of the kernel: 1 KB alignment slack, NS pipeline stages
// (S digit planes of A and of B per stage), the barriers, the epilogue's
// per-warp column tables and two words (TMEM base, failure flag).
__host__ __device__ constexpr size_t tc_smem(int S, int NS, int tn, int kb, bool cv = false) {
    return 1024 + (size_t)NS * S * ((cv ? CV_M : TM) + tn) * kb * 2 + 8 * (2 * NS + 5) +
           (size_t)NEPI * (tn / 2) * 12 + 16 + (cv ? (size_t)CV_RING * CV_M * kb * 8 + 16 : 0);
}

// Persistent kernel: each CTA walks the units blockIdx.x, blockIdx.x +
// gridDim.x, ...; the stage ring and the TMEM accumulator sets run on across
// units, so TMA, tensor core and epilogue of different units overlap.
//
//   warp 0      TMA producer: all S digit planes of A and B of one k-block per
//               stage.
//   warp 1      TMEM owner and MMA issuer: the level products of K chunk c
//               (at most KCHUNK deep, so the leading level sums are exact) go
//               to accumulator set c % NSET; a commit marks the set full.
//   warps 2-9   epilogue: warp w reads TMEM lanes 32 (w % 4).. of column half
//               (w - 2) / 4, frees the set, and carries the sum over the
//               unit's K chunks in registers -- one FP32 value per element
//               when D <= 3 (the few-digit form), an unevaluated FP32 pair
//               (error-free two-sums) at D = 4 to 6, a 64-bit integer at D = 7
//               (the level sums are integers).  After the last chunk the
//               tile goes to C once: FP64 built from bit patterns with the
//               scale 2^(e_m + e_n - 2 C) (and a power-of-two alpha) in the
//               exponent field, old values of C loaded 8 at a time.
//
// D <= 3: TN = 128, two levels (256 columns) per set, two sets, so the MMAs
// of one chunk run while the epilogue drains the other.  D >= 4: TN = 64, three
// to five levels, two sets up to D = 5; at D = 6 there is room for one, which
// the epilogue frees as soon as the levels are in registers (a few percent of
// a 2048-deep chunk's MMA time).  D = 7 reads out sixteen times as often and so
// takes TN = 48, where two sets of five levels fit (against 64 columns and one
// set, both with read-outs every 512 terms: 1 % of an update of 54 spin
// orbitals and 10 tau points, 5 % of a residual of 21 occupied and 37 virtual
// spin orbitals; at D = 6 the narrower tile costs 4.5 % of a sweep of 114 spin
// orbitals and 3 tau points instead).
//
// DL (the digit levels D) is a template parameter: the MMA issue loop is then
// straight-line code whose descriptors are per-stage bases plus constant
// offsets, so the single issuing thread keeps up with the tensor core.
//
// CV (a small A that no cache holds, K > 4096; the caller's rule): A is not
// packed.  Warps 10-17 copy its FP64 values asynchronously into a ring of
// k-blocks in shared memory, CV_RING - 1 ahead, each warp its own rows and so
// without barriers, and write their digits into the stage that the TMA
// producer fills with B.  A's planes then have CV_M rows; the MMA reads 128, and
// the rows beyond are other planes' bytes, whose products no one reads.
template <int TN, bool FF, int KBT, int DL, bool CV>
__global__ void __launch_bounds__(NTHREADS + (CV ? 32 * NCV : 0), 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               TcParams p) {
    if (!kv_depend()) return;
    using G = Dig<DL>;
    constexpr int SD = G::S, nl = G::NL;     // digit planes and levels
    constexpr int PLANE_BYTES = (CV ? CV_M : TM) * KBT * 2;   // a digit plane of an A k-block
    constexpr int BPLANE = TN * KBT * 2;         // one digit plane of a B k-block
    constexpr bool WD = G::WIDE;             // running sums are 64-bit integers
    constexpr int WCOLS = TN / 2;            // columns per epilogue warp
    constexpr int LW = FF ? 4 : 16;          // columns per TMEM load (<= 32 registers in flight)
    constexpr int NG = WCOLS / LW;           // TMEM loads per level
    constexpr int WG = 8;                    // columns per store group
    constexpr int SET_COLS = nl * TN;        // TMEM columns of a set
    constexpr int NSET = 2 * SET_COLS <= TMEM_COLS ? 2 : 1;   // accumulator sets
    constexpr int PMAX = 256 / TN;           // B planes per MMA (N <= 256)
    static_assert(NSET * SET_COLS <= TMEM_COLS, "accumulator sets exceed TMEM");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int S = SD;
    const int NS = p.NS;
    constexpr uint32_t stage_a = S * PLANE_BYTES, stage_b = S * BPLANE;
    uint8_t *sA = smem;
    uint8_t *sB = smem + NS * stage_a;
    uint64_t *bars = (uint64_t *)(sB + NS * stage_b);
    uint64_t *full = bars, *empty = bars + NS;
    uint64_t *accf = bars + 2 * NS, *acce = accf + 2, *done = acce + 2;
    long long *s_coff = (long long *)(done + 1);            // [NEPI][WCOLS]
    int *s_cexp = (int *)(s_coff + NEPI * WCOLS);           // [NEPI][WCOLS]
    uint32_t *tmem_slot = (uint32_t *)(s_cexp + NEPI * WCOLS);
    volatile int *s_fail = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        *s_fail = 0;
        for (int i = 0; i < NS; i++) {
            mbar_init(smem_u32(&full[i]), CV ? 1 + NCV : 1);
            mbar_init(smem_u32(&empty[i]), 1);
        }
        for (int i = 0; i < NSET; i++) {
            mbar_init(smem_u32(&accf[i]), 1);
            mbar_init(smem_u32(&acce[i]), NEPI);
        }
        mbar_init(smem_u32(done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer ----
            const uint32_t bytes = (uint32_t)(CV ? stage_b : stage_a + stage_b);
            int st = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const Unit w = unit_of<CV>(p, u, TN);
                for (int q = p.beg[w.cb]; q < p.beg[w.cb + 1] && ok; q++) {
                    const int ya = p.arow[q] + w.b * p.a_batch_rows + w.m0;
                    const int yb = p.brow[q] + w.b * p.b_batch_rows + w.n0;
                    for (int kb = w.kb0; kb < w.kb1; kb++) {
                        if (!mbar_wait(smem_u32(&empty[st]), ph ^ 1) || *s_fail) {
                            atomicExch(p.err, 1);
                            *s_fail = 1;
                            ok = false;
                            break;
                        }
                        const uint32_t fb = smem_u32(&full[st]);
                        mbar_expect_tx(fb, bytes);
                        const int x = kb * KBT;
                        for (int s = 0; s < S; s++) {
                            if (!CV)
                                tma_load_2d(smem_u32(sA + st * stage_a + s * PLANE_BYTES), &tmA, x,
                                            ya + s * p.Mp, fb);
                            tma_load_2d(smem_u32(sB + st * stage_b + s * BPLANE), &tmB, x,
                                        yb + s * p.Np, fb);
                        }
                        issued++;
                        if (++st == NS) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                }
            }
            // drain: every issued stage must have landed before the CTA exits
            for (int i = 0; i < min(issued, NS); i++) {
                if (st == 0) {
                    st = NS - 1;
                    ph ^= 1;
                } else {
                    st--;
                }
                if (!mbar_wait(smem_u32(&full[st]), ph)) atomicExch(p.err, 2);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer ----
            // descriptors of stage 0's first planes; a stage or plane offset
            // adds (offset >> 4) to the address field (all of shared memory
            // fits its 14 bits)
            const uint64_t dA0 = desc_of<KBT>(smem_u32(sA)), dB0 = desc_of<KBT>(smem_u32(sB));
            int st = 0, gc = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const Unit w = unit_of<CV>(p, u, TN);
                const int nsrc = p.beg[w.cb + 1] - p.beg[w.cb];
                for (int q = 0; q < nsrc && ok; q++)
                for (int c0 = w.kb0; c0 < w.kb1 && ok; c0 += p.chunk_kb) {
                    const int c1 = min(c0 + p.chunk_kb, w.kb1);
                    const int set = gc % NSET;
                    if (!mbar_wait(smem_u32(&acce[set]), ((gc / NSET) & 1) ^ 1) || *s_fail) {
                        atomicExch(p.err, 3);
                        *s_fail = 1;
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t tacc = tmem + set * SET_COLS;
                    for (int kb = c0; kb < c1; kb++) {
                        if (!mbar_wait(smem_u32(&full[st]), ph) || *s_fail) {
                            atomicExch(p.err, 4);
                            *s_fail = 1;
                            ok = false;
                            break;
                        }
                        fence_after();
                        // A plane s against B planes t0.. (adjacent in shared
                        // memory) into levels s + t0.. (adjacent in TMEM); the
                        // first k-step of a chunk starts every level (s = 1
                        // reaches all of them) and later ones accumulate
                        const uint64_t dA = dA0 + ((st * stage_a) >> 4);
                        const uint64_t dB = dB0 + ((st * stage_b) >> 4);
                        const uint32_t later = (kb > c0) ? 1u : 0u;
#pragma unroll
                        for (int kk = 0; kk < KBT / 16; kk++) {
#pragma unroll
                            for (int s = 1; s <= S; s++) {
                                const int tmax = nl + 1 - s;
                                const uint32_t acc = (kk > 0 || s > 1) ? 1u : later;
                                const uint64_t da = dA + (((s - 1) * PLANE_BYTES + kk * 32) >> 4);
#pragma unroll
                                for (int t0 = 1; t0 <= tmax; t0 += PMAX) {
                                    const int np = min(PMAX, tmax - t0 + 1);
                                    const uint64_t db =
                                        dB + (((t0 - 1) * BPLANE + kk * 32) >> 4);
                                    umma(tacc + (s + t0 - 2) * TN, da, db,
                                         idesc_of(np * TN), acc);
                                }
                            }
                        }
                        umma_commit(smem_u32(&empty[st]));
                        if (++st == NS) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                    if (!ok) break;
                    umma_commit(smem_u32(&accf[set]));
                    gc++;
                }
            }
            // every MMA issued by this thread completes before TMEM is freed
            umma_commit(smem_u32(done));
            if (!mbar_wait(smem_u32(done), 0)) atomicExch(p.err, 5);
        }
    } else if (CV && warp >= 2 + NEPI) {
        // ---- A: FP64 values to digits ----
        // A warp's rows are w0 + y + i STEP, y < RPI, i < ni; it copies a row's
        // values with neighbouring lanes and converts a pair a lane.  Rows past
        // the last one repeat it: branches per row would serialise the loads
        // and the conversions (3800 clocks a k-block of 57 x 64 with them).
        constexpr int LPR = KBT / 2, RPI = 32 / LPR;   // lanes and rows of a conversion step
        constexpr int STEP = NCV * RPI, NI = CV_M / STEP, KPL = KBT / 32;
        const int w0 = (warp - 2 - NEPI) * RPI, r0 = w0 + lane / LPR, kp = 2 * (lane % LPR);
        const int ni = w0 < p.M ? (p.M - w0 + STEP - 1) / STEP : 0;
        double *ring = (double *)(((uintptr_t)(tmem_slot + 4) + 15) & ~(uintptr_t)15);
        // position in the sequence of k-blocks of this CTA's units
        struct Cursor {
            Unit w;
            int u, q, kb;
            const double *base;
            __device__ __forceinline__ void unit(const TcParams &p) {
                if (u >= p.units) return;
                w = unit_of<CV>(p, u, TN);
                q = p.beg[w.cb];
                kb = w.kb0;
                base = p.A + p.oa[q] + (long long)w.b * p.a_bst;
            }
            __device__ __forceinline__ bool next(const TcParams &p) {   // another source or unit
                if (++kb < w.kb1) return false;
                kb = w.kb0;
                if (++q >= p.beg[w.cb + 1]) {
                    u += gridDim.x;
                    unit(p);
                } else {
                    base = p.A + p.oa[q] + (long long)w.b * p.a_bst;
                }
                return true;
            }
        };
        auto fetch = [&](Cursor &c, int slot) {
            if (c.u < p.units) {
                const int k0 = c.kb * KBT + lane;
                const uint32_t d0 = smem_u32(ring + (slot * CV_M + w0) * KBT + lane);
                const double *g[KPL];
#pragma unroll
                for (int j = 0; j < KPL; j++)
                    g[j] = c.base + p.dv_ac.off(p.Ac, min(k0 + 32 * j, p.K - 1));
#pragma unroll
                for (int i = 0; i < NI; i++) {
                    if (i >= ni) break;
#pragma unroll
                    for (int y = 0; y < RPI; y++)
#pragma unroll
                        for (int j = 0; j < KPL; j++)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                             d0 + ((i * STEP + y) * KBT + 32 * j) * 8),
                                         "l"(g[j] + min(w0 + i * STEP + y, p.M - 1) * p.ar)
                                         : "memory");
                }
                c.next(p);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        Cursor f, c;
        f.u = c.u = blockIdx.x;
        f.unit(p);
        c.unit(p);
#pragma unroll
        for (int i = 0; i < CV_RING - 1; i++) fetch(f, i);
        int st = 0, slot = 0;
        uint32_t ph = 0;
        bool fresh = true;
        int ex[NI];
        // swizzled byte offset in a plane; rows STEP apart have the same swizzle
        static_assert(STEP % 8 == 0, "swizzle period");
        const uint32_t so =
            (uint32_t)(r0 * KBT * 2 + (((kp >> 3) ^ (KBT == 64 ? r0 & 7 : (r0 >> 1) & 3)) << 4) +
                       (kp & 7) * 2);
        while (c.u < p.units) {
            fetch(f, slot == 0 ? CV_RING - 1 : slot - 1);
            if (fresh) {
                const int *ea = p.ea + p.aex[c.q] + c.w.b * p.ea_bst;
#pragma unroll
                for (int i = 0; i < NI; i++) ex[i] = exp_of(ea[min(r0 + i * STEP, p.M - 1)]);
            }
            const bool tail = c.kb * KBT + KBT > p.K;
            asm volatile("cp.async.wait_group %0;" ::"n"(CV_RING - 1) : "memory");
            __syncwarp();                        // the other lanes' copies too
            const bool got = mbar_wait(smem_u32(&empty[st]), ph ^ 1);
            if (__any_sync(0xffffffffu, !got || *s_fail)) {
                if (lane == 0) {
                    atomicExch(p.err, 11);
                    *s_fail = 1;
                }
                break;
            }
            uint8_t *dst = sA + st * stage_a;
            const double *src = ring + (slot * CV_M + r0) * KBT + kp;
#pragma unroll
            for (int i = 0; i < NI; i += 2) {
                if (i >= ni) break;
                uint32_t wd[2][S];
#pragma unroll
                for (int y = 0; y < 2 && i + y < NI; y++) {
                    ulonglong2 x =
                        *reinterpret_cast<const ulonglong2 *>(src + (i + y) * STEP * KBT);
                    if (tail) {                  // beyond K
                        const int k = c.kb * KBT + kp;
                        if (k >= p.K) x.x = 0;
                        if (k + 1 >= p.K) x.y = 0;
                    }
                    digit_words<DL>(x.x, x.y, ex[i + y], wd[y]);
                }
#pragma unroll
                for (int y = 0; y < 2 && i + y < NI; y++)
#pragma unroll
                    for (int t = 0; t < S; t++)
                        *reinterpret_cast<uint32_t *>(dst + t * PLANE_BYTES + so +
                                                      (i + y) * STEP * KBT * 2) = wd[y][t];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full[st]));
            if (++st == NS) {
                st = 0;
                ph ^= 1;
            }
            slot = slot == CV_RING - 1 ? 0 : slot + 1;
            fresh = c.next(p);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ---- epilogue ----
        const int ew = warp - 2, q = warp & 3, h = ew >> 2;
        const int row = q * 32 + lane;
        long long *coff = s_coff + ew * WCOLS;
        int *cexp = s_cexp + ew * WCOLS;
        float rhi[WD ? 1 : WCOLS];
        float rlo[FF && !WD ? WCOLS : 1];
        unsigned long long sum[WD ? WCOLS : 1];      // in units of 2^-WUNIT
        int gc = 0;
        bool ok = true;
        int cached_n = -1, cached_e = -1;   // the columns coff / cexp hold (warp-uniform)
        for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            const Unit w = unit_of<CV>(p, u, TN);
            if (w.kb0 >= w.kb1) continue;
            const int q0 = p.beg[w.cb], q1 = p.beg[w.cb + 1];
            for (int src = q0; src < q1 && ok; src++) {
                const double beta = src == q0 ? p.beta : 1.0;
                // C addresses of this unit; for the read-modify-write of a
                // general beta the old values are prefetched into L2 now, while
                // the MMAs run, so that it is not bound by the few loads a warp
                // keeps in flight (the L2 reductions of beta = 1 fetch their lines
                // at L2 themselves: prefetching them too cost 6 of 82 ms per
                // 114-spin-orbital iteration in issue slots)
                const int nw = w.n0 + h * WCOLS;          // first column of this warp
                // column offsets and exponents: the same for every tile of this
                // column range (and batch entry, when B is per batch)
                const int ekey = p.bex[src] + w.b * p.eb_bst;
                if (nw != cached_n || ekey != cached_e) {
                    __syncwarp();                            // the last tile's reads are done
                    for (int i = lane; i < WCOLS; i += 32) {
                        const int n = nw + i;
                        coff[i] = (n < p.N) ? p.C.c.off(n) : 0;
                        cexp[i] = (n < p.N) ? exp_of(p.eb[ekey + n]) : 0;
                    }
                    cached_n = nw;
                    cached_e = ekey;
                }
                __syncwarp();
                const int m = w.m0 + row;
                const int nlim = p.N - nw;
                long long roff = 0;
                if (m < p.M) {                               // p.C.r.off(m), fast divisions
                    const int r1 = p.dv_cr2.div(m), i2 = m - r1 * p.C.r.size[2];
                    const int i0 = p.dv_cr1.div(r1), i1 = r1 - i0 * p.C.r.size[1];
                    roff = (long long)i0 * p.C.r.st[0] + (long long)i1 * p.C.r.st[1] +
                           (long long)i2 * p.C.r.st[2];
                }
                double *Cr = p.C.p + (long long)w.b * p.C.bst + p.coff[w.cb] + roff;
                if (p.c_split) Cr += w.kb0 / p.split_kb * p.c_split;
                const int krow = (m < p.M) ? exp_of(p.ea[p.aex[src] + w.b * p.ea_bst + m]) -
                                                 2 * G::C + p.alpha_exp
                                           : 0;
                if (!CV && m < p.M && p.nsplit == 1 && beta != 0.0 && beta != 1.0) {
                    for (int i = 0; i < min(WCOLS, nlim); i++)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(Cr + coff[i]));
                }
                for (int f0 = w.kb0, f1; f0 < w.kb1 && ok; f0 = f1) {
                f1 = WD ? min(f0 + p.flush_kb, w.kb1) : w.kb1;
                const double be = f0 == w.kb0 ? beta : 1.0;
                for (int c0 = f0; c0 < f1; c0 += p.chunk_kb) {
                    const int set = gc % NSET;
                    const bool got = mbar_wait(smem_u32(&accf[set]), (gc / NSET) & 1);
                    // one verdict per warp: tcgen05.ld below needs every lane
                    if (__any_sync(0xffffffffu, !got || *s_fail)) {
                        if (lane == 0) {
                            atomicExch(p.err, 6);
                            *s_fail = 1;
                        }
                        ok = false;
                        break;
                    }
                    fence_after();
                    const bool first = (c0 == f0);
                    const uint32_t tb =
                        tmem + ((uint32_t)(q * 32) << 16) + set * SET_COLS + h * WCOLS;
    #pragma unroll
                    for (int g = 0; g < NG; g++) {
                        uint32_t r[nl][LW];
    #pragma unroll
                        for (int l = 0; l < nl; l++)
                            tmem_ld<LW>(tb + l * TN + g * LW, r[l]);
                        tmem_wait_ld();
    #pragma unroll
                        for (int j = 0; j < LW; j++) {
                            const int i = g * LW + j;
                            float hi = __uint_as_float(r[0][j]);
                            if constexpr (!FF) {
                                if (nl > 1) hi += __uint_as_float(r[nl > 1 ? 1 : 0][j]);
                                rhi[i] = first ? hi : rhi[i] + hi;
                            } else if constexpr (WD) {
                                // level l holds an integer times 2^(18 - 9 l): the
                                // sum of all as one integer, exact but for the
                                // rounding of the last two levels' sum
                                const int i2 = __float2int_rn(hi);
                                const int i3 = __float2int_rn(__uint_as_float(r[1][j]) * 512.f);
                                const int i4 = __float2int_rn(__uint_as_float(r[2][j]) * 262144.f);
                                const int i5 = __float2int_rn(
                                    (__uint_as_float(r[3][j]) + __uint_as_float(r[nl > 4 ? 4 : 0][j])) *
                                    (float)(1ll << WUNIT));
                                sum[i] = (first ? 0ull : sum[i]) +
                                         (unsigned long long)((i2 * 512 + i3) * (1ll << (WUNIT - 9))) +
                                         (unsigned long long)(i4 * (1ll << (WUNIT - 18))) +
                                         (unsigned long long)(long long)i5;
                            } else {
                                // exact level sums, leading first: an FP32 pair
                                float lo = 0.f, e;
    #pragma unroll
                                for (int l = 1; l < nl; l++) {
                                    two_sum(hi, __uint_as_float(r[l][j]), hi, e);
                                    lo += e;
                                }
                                if (first) {
                                    rhi[i] = hi;
                                    rlo[i] = lo;
                                } else {
                                    float sm;
                                    two_sum(rhi[i], hi, sm, e);
                                    rlo[i] += lo + e;
                                    rhi[i] = sm;
                                }
                            }
                        }
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&acce[set]));
                    gc++;
                }
                if (!ok) break;
                // ---- the tile to C ----
                if (m < p.M) {
                    // value of column i of this thread's row
                    auto value = [&](int i) -> double {
                        const int k = krow + cexp[i];
                        double v;
                        if constexpr (WD) {
                            v = i64_scaled((long long)sum[i], k - WUNIT, p.alpha_sign);
                        } else {
                            v = f32_scaled(rhi[i], k, p.alpha_sign);
                            if constexpr (FF) v += f32_scaled(rlo[i], k, p.alpha_sign);
                        }
                        if (!p.alpha_pow2) v *= p.alpha;
                        return v;
                    };
                    if (CV || (p.nsplit > 1 && !p.c_split) || be == 1.0) {
                        // C += value: each element gets exactly one addition in
                        // this launch unless K chunks run as separate units, so a
                        // fire-and-forget reduction at L2 gives old + value
                        // rounded once, like a load-add-store, without the
                        // thread waiting for the old value (measured on the
                        // 114-spin-orbital n^5 class: 82 ms per iteration
                        // against 120 ms for the load-add-store ring below)
                        if constexpr (FF && !WD) {
                            if (p.alpha_pow2) {
                                // the FP32 pair as two reductions at L2: no FP64
                                // add on the SM (GB300's FP64 pipe bounded this
                                // write); C gets old + hi + lo in two roundings
    #pragma unroll
                                for (int i = 0; i < WCOLS; i++) {
                                    if (i < nlim) {
                                        const int k = krow + cexp[i];
                                        atomicAdd(Cr + coff[i], f32_scaled(rhi[i], k, p.alpha_sign));
                                        atomicAdd(Cr + coff[i], f32_scaled(rlo[i], k, p.alpha_sign));
                                    }
                                }
                            } else {
    #pragma unroll
                                for (int i = 0; i < WCOLS; i++)
                                    if (i < nlim) atomicAdd(Cr + coff[i], value(i));
                            }
                        } else {
    #pragma unroll
                            for (int i = 0; i < WCOLS; i++)
                                if (i < nlim) atomicAdd(Cr + coff[i], value(i));
                        }
                    } else if (be == 0.0) {
                        if (FF && !WD && p.alpha_pow2) {
                            // hi stored, lo added at L2: hi + lo rounded once,
                            // as the FP64 add gave, without it on the SM
    #pragma unroll
                            for (int i = 0; i < WCOLS; i++) {
                                if (i < nlim) {
                                    const int k = krow + cexp[i];
                                    Cr[coff[i]] = f32_scaled(rhi[WD ? 0 : i], k, p.alpha_sign);
                                    if constexpr (FF && !WD)
                                        atomicAdd(Cr + coff[i], f32_scaled(rlo[i], k, p.alpha_sign));
                                }
                            }
                        } else {
    #pragma unroll
                            for (int i = 0; i < WCOLS; i++)
                                if (i < nlim) Cr[coff[i]] = value(i);
                        }
                    } else {
                        // read-modify-write: the old values of the next RING
                        // groups of WG columns are in flight while one group is
                        // combined and stored
                        constexpr int NGW = WCOLS / WG, RING = FF ? 3 : 2;
                        double old[RING][WG];
    #pragma unroll
                        for (int q = 0; q < RING; q++)
    #pragma unroll
                            for (int j = 0; j < WG; j++)
                                old[q][j] = (q < NGW && q * WG + j < nlim) ? Cr[coff[q * WG + j]] : 0.0;
    #pragma unroll
                        for (int g = 0; g < NGW; g++) {
                            const int q = g % RING;
    #pragma unroll
                            for (int j = 0; j < WG; j++) {
                                const int i = g * WG + j;
                                const double v = fma(be, old[q][j], value(i));
                                if (i < nlim) Cr[coff[i]] = v;
                            }
                            if (g + RING < NGW) {
    #pragma unroll
                                for (int j = 0; j < WG; j++) {
                                    const int i = (g + RING) * WG + j;
                                    old[q][j] = (i < nlim) ? Cr[coff[i]] : 0.0;
                                }
                            }
                        }
                    }
                }
                __syncwarp();
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// Digit packing: FP64 strided view (rows x K) -> S BF16 planes [b][s][Rp][Kp]
// and row exponents [b][Rp].
// ---------------------------------------------------------------------------
// Operand tiles of 32 rows x 64 k go through shared memory so that global
// reads are coalesced along whichever operand index is contiguous in memory
// (the row index for some permuted views, k for others) and plane writes are
// coalesced along k.  The composite-index offsets of the tile's rows and k
// columns are computed once per tile (96 divisions instead of one per
// element) and kept in shared memory; -1 marks a row or column outside the
// view.
constexpr int PT_R = 32, PT_K = 64;

// The tile walk: offsets of tile rows r0.. and k columns k0.. in a shared
// table (threads 0-95), then each thread's 8 values -- row lane at k = w + 8 i
// (rows_fast), else rows w + 8 i at k = lane, lane + 32 -- loaded into
// registers, so a block can have the next tile's loads in flight while it
// works on the current one.
__device__ __forceinline__ void tile_offsets(const PackView &v, int r0, int k0, int R, int K,
                                             long long *off) {
    const int tid = threadIdx.x;
    if (tid < PT_R) {
        off[tid] = (r0 + tid < R) ? v.r.off(r0 + tid) : -1;
    } else if (tid < PT_R + PT_K) {
        const int k = k0 + tid - PT_R;
        off[tid] = (k < K) ? v.c.off(k) : -1;
    }
}

__device__ __forceinline__ void tile_fetch(const double *base, const long long *off,
                                           int rows_fast, unsigned long long (&pre)[8]) {
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    if (rows_fast) {
        const long long ro = off[lane];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const long long ko = off[PT_R + w + 8 * i];
            pre[i] = (ro >= 0 && ko >= 0)
                         ? (unsigned long long)__double_as_longlong(__ldg(base + ro + ko))
                         : 0ull;
        }
    } else {
        const long long ko0 = off[PT_R + lane], ko1 = off[PT_R + lane + 32];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const long long ro = off[w + 8 * i];
            pre[2 * i] = (ro >= 0 && ko0 >= 0)
                             ? (unsigned long long)__double_as_longlong(__ldg(base + ro + ko0))
                             : 0ull;
            pre[2 * i + 1] = (ro >= 0 && ko1 >= 0)
                                 ? (unsigned long long)__double_as_longlong(__ldg(base + ro + ko1))
                                 : 0ull;
        }
    }
}

// raw row exponents: max binary exponent over each row of `ktiles`
// consecutive 64-wide k tiles, one atomicMax per row and block.  The maxima
// are taken in registers from each thread's 8 values, and the next tile's
// loads are issued before the current tile's values are used.
__global__ void __launch_bounds__(256)
pack_exp_kernel(const __grid_constant__ PackView v, int R, int K, int rows_fast, int ktiles, int *__restrict__ ex) {
    if (!kv_depend()) return;
    __shared__ long long off[PT_R + PT_K];
    __shared__ int rmax[8][PT_R];
    const int b = blockIdx.z, r0 = blockIdx.y * PT_R;
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const double *base = v.base(b);
    const int kt0 = blockIdx.x * ktiles;
    const int nkt = min(ktiles, (K + PT_K - 1) / PT_K - kt0);
    // rows_fast: one row per thread (lane); otherwise four rows (w + 8 i)
    int em[4] = {-2000, -2000, -2000, -2000};
    unsigned long long pre[8];
    tile_offsets(v, r0, kt0 * PT_K, R, K, off);
    __syncthreads();
    tile_fetch(base, off, rows_fast, pre);
    for (int t = 0; t < nkt; t++) {
        unsigned long long cur[8];
#pragma unroll
        for (int i = 0; i < 8; i++) cur[i] = pre[i];
        if (t + 1 < nkt) {
            __syncthreads();                    // every thread has read the offsets
            tile_offsets(v, r0, (kt0 + t + 1) * PT_K, R, K, off);
            __syncthreads();
            tile_fetch(base, off, rows_fast, pre);
        }
        if (rows_fast) {
#pragma unroll
            for (int i = 0; i < 8; i++) em[0] = max(em[0], raw_exp(cur[i]));
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                em[i] = max(em[i], max(raw_exp(cur[2 * i]), raw_exp(cur[2 * i + 1])));
        }
    }
    if (rows_fast) {
        // row lane: combine the eight warps' maxima
        rmax[w][lane] = em[0];
        __syncthreads();
        if (w == 0) {
            int e = rmax[0][lane];
#pragma unroll
            for (int q = 1; q < 8; q++) e = max(e, rmax[q][lane]);
            if (e > -2000 && r0 + lane < R) atomicMax(&ex[(long long)b * R + r0 + lane], e);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            int e = em[i];
            for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
            const int row = r0 + w + 8 * i;
            if (lane == 0 && e > -2000 && row < R) atomicMax(&ex[(long long)b * R + row], e);
        }
    }
}

// Balanced base-128 digits of x 2^-e (|x 2^-e| < 1/2), most significant
// first, from the FP64 bit pattern with integer arithmetic only.
__device__ __forceinline__ void digits_of(unsigned long long bits, int e, int S, int *d) {
    for (int s = 0; s < S; s++) d[s] = 0;
    const int be = (int)((bits >> 52) & 0x7FF);
    if (be == 0) return;                        // zero / subnormal (< 2^-1022): zero
    const long long mant = (long long)((bits & 0xFFFFFFFFFFFFFull) | (1ull << 52));
    // |x| 2^-e 2^(7S) = mant 2^(be - 1023 - 52 - e + 7S), rounded to an integer
    const int sh = be - 1023 - 52 - e + 7 * S;
    long long Y;
    if (sh >= 0) Y = mant << sh;
    else if (sh > -63) Y = (mant + (1ll << (-sh - 1))) >> (-sh);
    else Y = 0;
    // digits in [-64, 63], least significant first; the top one takes the
    // remainder, which is in [0, 64]
    for (int s = S - 1; s >= 1; s--) {
        int dd = (int)(Y & 127);
        if (dd >= 64) dd -= 128;
        d[s] = dd;
        Y = (Y - dd) >> 7;
    }
    d[0] = (int)Y;
    if (bits >> 63)
        for (int s = 0; s < S; s++) d[s] = -d[s];
}

// Up to three planes take at most 21 bits of |x| 2^-e 2^(7S): the shift
// right is at least 33, so those bits and the rounding bit all lie in the
// high word of the significand, and 32-bit arithmetic on it gives the digits
// of the 64-bit form above exactly (adding the rounding bit 2^(n+31) cannot
// carry out of bits the low word decides).
template <int S>
__device__ __forceinline__ void digits_of_s(unsigned long long bits, int e, int *d) {
    if (S > 3) {
        digits_of(bits, e, S, d);
        return;
    }
#pragma unroll
    for (int s = 0; s < S; s++) d[s] = 0;
    const unsigned hi = (unsigned)(bits >> 32);
    const int be = (int)((hi >> 20) & 0x7FF);
    if (be == 0) return;
    const int n = 52 + e - (be - 1023) - 7 * S - 32;      // >= 1 since e >= be - 1021
    unsigned Y = n < 22 ? (((hi & 0xFFFFFu) | 0x100000u) + (1u << (n - 1))) >> n : 0u;
#pragma unroll
    for (int s = S - 1; s >= 1; s--) {
        int dd = (int)(Y & 127u);
        if (dd >= 64) dd -= 128;
        d[s] = dd;
        Y = (unsigned)((int)Y - dd) >> 7;
    }
    d[0] = (int)Y;
    if (hi >> 31)
#pragma unroll
        for (int s = 0; s < S; s++) d[s] = -d[s];
}

// bf16 pair (d0 2^-7s, d1 2^-7s), |d| <= 64: the float 1.5 2^23 + d is formed
// by an integer add on its bit pattern and the offset is removed, with the
// scaling, by one exact FMA; one conversion then packs both values.
template <int s>
__device__ __forceinline__ __nv_bfloat162 digit_pair(int d0, int d1) {
    constexpr float sc = 1.0f / (float)(1ull << (7 * s));     // 2^-7s, exact
    const float f0 = fmaf(__int_as_float(0x4B400000 + d0), sc, -12582912.0f * sc);
    const float f1 = fmaf(__int_as_float(0x4B400000 + d1), sc, -12582912.0f * sc);
    return __floats2bfloat162_rn(f0, f1);
}

template <int D>
__device__ __forceinline__ void store_words(uint16_t *ob, size_t plane, unsigned long long x0,
                                            unsigned long long x1, int e) {
    uint32_t w[Dig<D>::S];
    digit_words<D>(x0, x1, e, w);
#pragma unroll
    for (int s = 0; s < Dig<D>::S; s++) *reinterpret_cast<uint32_t *>(ob + s * plane) = w[s];
}

// Base-128 digits here come from the loop above: digit_words, the same values,
// costs these kernels 0.2 % of a step of 114 spin orbitals.
template <int D>
__device__ __forceinline__ void store_digits(uint16_t *ob, size_t plane, unsigned long long x0,
                                             unsigned long long x1, int e) {
    constexpr int S = Dig<D>::S;
    if constexpr (Dig<D>::WIDE) {
        uint32_t w[S];
        digit_words<D>(x0, x1, e, w);
#pragma unroll
        for (int s = 0; s < S; s++) *reinterpret_cast<uint32_t *>(ob + s * plane) = w[s];
    } else {
        int d0[S], d1[S];
        digits_of_s<S>(x0, e, d0);
        digits_of_s<S>(x1, e, d1);
        *reinterpret_cast<__nv_bfloat162 *>(ob) = digit_pair<0>(d0[0], d1[0]);
        if constexpr (S > 1)
            *reinterpret_cast<__nv_bfloat162 *>(ob + plane) = digit_pair<1>(d0[1], d1[1]);
        if constexpr (S > 2)
            *reinterpret_cast<__nv_bfloat162 *>(ob + 2 * plane) = digit_pair<2>(d0[2], d1[2]);
        if constexpr (S > 3)
            *reinterpret_cast<__nv_bfloat162 *>(ob + 3 * plane) = digit_pair<3>(d0[3], d1[3]);
        if constexpr (S > 4)
            *reinterpret_cast<__nv_bfloat162 *>(ob + 4 * plane) = digit_pair<4>(d0[4], d1[4]);
    }
}

// planes[b][s][row][k] (row stride ld); each thread packs two k.
// Persistent blocks walk the 32 x 64 tiles t = blockIdx.x, + gridDim.x, ...
// (k tile fastest, then row tile, then batch); the next tile's loads are in
// flight in registers while the current one is converted.
template <int D>
__global__ void __launch_bounds__(256)
pack_digits_kernel(const __grid_constant__ PackView v, int R, int K, int ld, int rows_fast, int ktn, int rtn,
                   int ntiles, const int *__restrict__ ex, uint16_t *__restrict__ out) {
    if (!kv_depend()) return;
    __shared__ unsigned long long val[PT_R][PT_K + 1];
    __shared__ long long off[PT_R + PT_K];
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const size_t plane = (size_t)R * ld;
    auto decode = [&](int t, int &b, int &r0, int &k0) {
        b = t / (rtn * ktn);
        const int rem = t - b * rtn * ktn;
        r0 = (rem / ktn) * PT_R;
        k0 = (rem % ktn) * PT_K;
    };
    unsigned long long pre[8];
    int t = blockIdx.x;
    if (t < ntiles) {
        int b, r0, k0;
        decode(t, b, r0, k0);
        tile_offsets(v, r0, k0, R, K, off);
        __syncthreads();
        tile_fetch(v.base(b), off, rows_fast, pre);
    }
    for (; t < ntiles; t += gridDim.x) {
        const long long tn = (long long)t + gridDim.x;
        int b, r0, k0;
        decode(t, b, r0, k0);
        __syncthreads();              // val and the offsets are free again
        if (rows_fast) {
#pragma unroll
            for (int i = 0; i < 8; i++) val[lane][w + 8 * i] = pre[i];
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                val[w + 8 * i][lane] = pre[2 * i];
                val[w + 8 * i][lane + 32] = pre[2 * i + 1];
            }
        }
        int bn = 0, rn = 0, kn = 0;
        if (tn < ntiles) {
            decode((int)tn, bn, rn, kn);
            tile_offsets(v, rn, kn, R, K, off);
        }
        __syncthreads();
        if (tn < ntiles) tile_fetch(v.base(bn), off, rows_fast, pre);
        const int k = k0 + 2 * lane;
        if (k < K) {
            for (int rr = w; rr < PT_R; rr += 8) {
                const int row = r0 + rr;
                if (row >= R) break;
                const int e = exp_of(ex[(long long)b * R + row]);
                // the second value is zero beyond K (tile fill)
                store_digits<D>(out + (size_t)b * Dig<D>::S * plane + (size_t)row * ld + k, plane,
                                val[rr][2 * lane], val[rr][2 * lane + 1], e);
            }
        }
    }
}

// Short rows (K <= 64 KT): one pass.  A block holds 32 whole rows in shared
// memory, takes each row's exponent from there and writes its digits, so the
// operand is read once and no atomics are needed.  The raw exponents it
// stores are those of the two-pass path (0x80808080 for an all-zero row).
// Blocks are persistent: they walk the row tiles t = blockIdx.x, + gridDim.x,
// ... (batch-major), and while one tile is converted from shared memory the
// global loads of the block's next tile are already in flight into
// registers.
constexpr int PR_KMAX = 256;

__host__ __device__ constexpr size_t pack_rows_smem(int kt) {
    return (size_t)PT_R * (kt * PT_K + 1) * 8 + (size_t)(kt * PT_K) * 8;
}

template <int D, int KT>
__global__ void __launch_bounds__(256, 2)
pack_rows_kernel(const __grid_constant__ PackView v, int R, int K, int ld, int rows_fast, int rtiles, int ntiles,
                 int *__restrict__ ex, uint16_t *__restrict__ out) {
    if (!kv_depend()) return;
    constexpr int NK = KT * PT_K, LDV = NK + 1, PER = NK / 8;   // values per thread
    extern __shared__ unsigned long long prs[];
    unsigned long long *val = prs;                                      // [PT_R][LDV]
    long long *koff = reinterpret_cast<long long *>(prs + PT_R * LDV);  // [NK]
    __shared__ int rexp[PT_R];
    const int tid = threadIdx.x, lane = tid % 32, w = tid / 32;
    for (int x = tid; x < NK; x += 256) koff[x] = (x < K) ? v.c.off(x) : -1;
    __syncthreads();
    // rows_fast: thread (lane, w) reads row lane at k = w + 8 i; otherwise rows
    // w + 8 i at k = lane + 32 j.  Both cover 32 x NK values, PER per thread.
    unsigned long long pre[PER];
    auto fetch = [&](int t) {
        const int b = t / rtiles, r0 = (t - b * rtiles) * PT_R;
        const double *base = v.base(b);
        if (rows_fast) {
            const long long ro = (r0 + lane < R) ? v.r.off(r0 + lane) : -1;
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const long long ko = koff[w + 8 * i];
                pre[i] = (ro >= 0 && ko >= 0)
                             ? (unsigned long long)__double_as_longlong(__ldg(base + ro + ko))
                             : 0ull;
            }
        } else {
#pragma unroll
            for (int i = 0; i < PT_R / 8; i++) {
                const int row = r0 + w + 8 * i;
                const long long ro = (row < R) ? v.r.off(row) : -1;
#pragma unroll
                for (int j = 0; j < 2 * KT; j++) {
                    const long long ko = koff[lane + 32 * j];
                    pre[i * 2 * KT + j] =
                        (ro >= 0 && ko >= 0)
                            ? (unsigned long long)__double_as_longlong(__ldg(base + ro + ko))
                            : 0ull;
                }
            }
        }
    };
    if (blockIdx.x < ntiles) fetch(blockIdx.x);
    const size_t plane = (size_t)R * ld;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        __syncthreads();                      // the previous tile's values are used up
        if (rows_fast) {
#pragma unroll
            for (int i = 0; i < PER; i++) val[lane * LDV + w + 8 * i] = pre[i];
        } else {
#pragma unroll
            for (int i = 0; i < PT_R / 8; i++)
#pragma unroll
                for (int j = 0; j < 2 * KT; j++)
                    val[(w + 8 * i) * LDV + lane + 32 * j] = pre[i * 2 * KT + j];
        }
        __syncthreads();
        if ((long long)t + gridDim.x < ntiles) fetch(t + gridDim.x);
        const int b = t / rtiles, r0 = (t - b * rtiles) * PT_R;
        // raw exponent of each row: warp w takes rows w, w + 8, ...
#pragma unroll
        for (int i = 0; i < PT_R / 8; i++) {
            const int rr = w + 8 * i;
            int e = -2000;
#pragma unroll
            for (int j = 0; j < KT * 2; j++) {
                const unsigned long long bits = val[rr * LDV + lane + 32 * j];
                if ((bits & 0x7FFFFFFFFFFFFFFFull) != 0)
                    e = max(e, (int)((bits >> 52) & 0x7FF) - 1023);
            }
            for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
            if (lane == 0) {
                const int raw = (e > -2000) ? e : (int)0x80808080u;
                rexp[rr] = raw;
                if (r0 + rr < R) ex[(long long)b * R + r0 + rr] = raw;
            }
        }
        __syncthreads();
        for (int rr = w; rr < PT_R; rr += 8) {
            const int row = r0 + rr;
            if (row >= R) break;
            const int e = exp_of(rexp[rr]);
            uint16_t *ob = out + (size_t)b * Dig<D>::S * plane + (size_t)row * ld;
#pragma unroll
            for (int j = 0; j < KT; j++) {
                const int k = 2 * lane + 64 * j;
                if (k >= K) break;
                // the second value is zero beyond K
                store_digits<D>(ob + k, plane, val[rr * LDV + k], val[rr * LDV + k + 1], e);
            }
        }
    }
}

// Longer rows (up to 8 x 512): one pass by clusters.  A cluster's CTAs hold 16
// whole rows in their shared memory, a slab of K each; row maxima meet through
// distributed shared memory, and every CTA writes the digits of its slab.  The
// operand is read once and in one launch, where the general path below reads
// it twice in two and clears the exponents in a third.  The loads are
// asynchronous copies to shared memory, so a block's whole slab is in flight
// at once, and three or more blocks an SM overlap loads and conversion (16 rows
// keep a slab of 416, K = 3249, at 53 KB; 32 rows leave two blocks and cost 15 %).
// Bound by instruction issue (40 an element, 2.9 a clock, before the maxima came
// from the high words alone, the copies' predicates from k and the digits from
// two FP32 additions): 3.3 to 3.9 TB/s of 8 + 2 S bytes an element.  The general
// path, the first form and now: three levels, 3249 x 3249 2.8, 3.3, 3.3 TB/s,
// 1089 x 1089 2.6, 3.2, 3.8; seven levels, 729 x 729 2.7, 3.5, 3.9.  Whole cases,
// general path and first form: 38 spin orbitals, solve 53.2 -> 51.2 ms; 54,
// update 11.2 -> 10.7; 66 23.1 -> 22.4; 114 132.6 -> 129.8.
constexpr int PC_MAX = 8, PC_SLAB = 512;      // CTAs of a cluster, k of a slab
constexpr int PC_R = 16;                      // rows of a cluster

__host__ __device__ constexpr size_t pack_slab_smem(int slab) {
    return (size_t)PC_R * (slab + 1) * 8 + (size_t)(slab + PC_R) * 8;
}

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int D>
__global__ void __launch_bounds__(256)
pack_cluster_kernel(const __grid_constant__ PackView v, int R, int K, int ld, int rows_fast,
                    int rtiles, int ncta, int slab, int *__restrict__ ex,
                    uint16_t *__restrict__ out) {
    if (!kv_depend()) return;
    extern __shared__ unsigned long long prs[];
    const int ldv = slab + 1;
    unsigned long long *val = prs;                                       // [PC_R][ldv]
    long long *koff = reinterpret_cast<long long *>(prs + PC_R * ldv);   // [slab]
    long long *roff = koff + slab;                                       // [PC_R]
    __shared__ int rmax[PC_R];
    const int tid = threadIdx.x, lane = tid % 32, w = tid / 32;
    const int t = blockIdx.x / ncta, rank = blockIdx.x - t * ncta;
    const int b = t / rtiles, r0 = (t - b * rtiles) * PC_R, k0 = rank * slab;
    const int kn = max(0, min(slab, K - k0));
    for (int x = tid; x < slab; x += 256) koff[x] = x < kn ? v.c.off(k0 + x) : -1;
    if (tid < PC_R) roff[tid] = r0 + tid < R ? v.r.off(r0 + tid) : -1;
    __syncthreads();
    const double *base = v.base(b);
    auto load = [&](uint32_t d, const double *g, bool in) {
        if (in)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(g) : "memory");
        else
            asm volatile("st.shared.b64 [%0], %1;" ::"r"(d), "l"(0ll) : "memory");
    };
    if (rows_fast) {
        const int r = tid % PC_R;
        const double *row = base + roff[r];
        const int lim = roff[r] >= 0 ? kn : 0;
        uint32_t d = smem_u32(val + r * ldv + tid / PC_R);
#pragma unroll 8
        for (int k = tid / PC_R; k < slab; k += 256 / PC_R, d += 8 * (256 / PC_R))
            load(d, row + koff[k], k < lim);
    } else {
        const double *row0 = base + roff[w], *row1 = base + roff[w + 8];
        const int lim0 = roff[w] >= 0 ? kn : 0, lim1 = roff[w + 8] >= 0 ? kn : 0;
        uint32_t d = smem_u32(val + w * ldv + lane);
#pragma unroll 4
        for (int k = lane; k < slab; k += 32, d += 8 * 32) {
            load(d, row0 + koff[k], k < lim0);
            load(d + 8 * 8 * ldv, row1 + koff[k], k < lim1);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // the largest high word of a row has its exponent (a row of nothing but
    // subnormals below 2^-1042 counts as zero, as its digits are)
    static_assert(PC_R == 16, "rows w and w + 8 of a warp");
    {
        const uint32_t *h0 = reinterpret_cast<const uint32_t *>(val + w * ldv) + 1;
        const uint32_t *h1 = h0 + 2 * 8 * ldv;
        uint32_t m0 = 0, m1 = 0;
        for (int k = lane; k < slab; k += 32) {
            m0 = max(m0, h0[2 * k] & 0x7FFFFFFFu);
            m1 = max(m1, h1[2 * k] & 0x7FFFFFFFu);
        }
        m0 = __reduce_max_sync(0xffffffffu, m0);
        m1 = __reduce_max_sync(0xffffffffu, m1);
        if (lane == 0) {
            rmax[w] = m0 ? (int)(m0 >> 20) - 1023 : -2000;
            rmax[w + 8] = m1 ? (int)(m1 >> 20) - 1023 : -2000;
        }
    }
    cluster_arrive();
    cluster_wait();
    int em[PC_R / 8];
#pragma unroll
    for (int i = 0; i < PC_R / 8; i++) {
        int e = -2000;
        if (lane < ncta) {
            uint32_t peer;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(peer)
                         : "r"(smem_u32(&rmax[w + 8 * i])), "r"(lane));
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(e) : "r"(peer) : "memory");
        }
        em[i] = __reduce_max_sync(0xffffffffu, e);
    }
    cluster_arrive();                         // the peers' maxima have been read
    const size_t plane = (size_t)R * ld;
#pragma unroll
    for (int i = 0; i < PC_R / 8; i++) {
        const int rr = w + 8 * i, row = r0 + rr;
        if (row >= R) break;
        // the raw exponents of the other paths (0x80808080 for an all-zero row)
        const int raw = em[i] > -2000 ? em[i] : (int)0x80808080u;
        if (rank == 0 && lane == 0) ex[(long long)b * R + row] = raw;
        const int e = exp_of(raw);
        uint16_t *ob = out + (size_t)b * Dig<D>::S * plane + (size_t)row * ld + k0;
        // the second value of the last pair is zero beyond K
        for (int k = 2 * lane; k < kn; k += 64)
            store_words<D>(ob + k, plane, val[rr * ldv + k], val[rr * ldv + k + 1], e);
    }
    cluster_wait();
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                             cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

}  // namespace

int kv_tc_map(kvft_ctx *ctx, CUtensorMap *map, void *base, int K, int ld, long long rows, int kb,
              int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return kv_fail(ctx, KVFT_EDEVICE, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)kb, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE,
                    kb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return kv_fail(ctx, KVFT_EDEVICE, "cuTensorMapEncodeTiled failed");
    return KVFT_OK;
}

namespace {

// Digit planes [nb][S][R][ld] and exponents [nb][R].  ld = K rounded up to 64
// elements, so that every row starts on a 128-byte line and a TMA box row
// (one k-block of one row) touches one line, not two.  No row or K padding is
// written: the tensor map's extent is (K, nb S R) and TMA fills out-of-range
// boxes with zeros; rows past R inside a 128-row box belong to the next plane
// and only reach output rows/columns that the epilogue discards.
// Identity of a packed operand: address, view, extents and digit count.
std::string pack_key(const PackView &v, int R, int K, int nb, int D) {
    char b[400];
    snprintf(b, sizeof b, "%p|%d,%d,%d:%lld,%lld,%lld|%d,%d,%d:%lld,%lld,%lld|%lld|%d,%d,%d,%d",
             (const void *)v.p, v.r.size[0], v.r.size[1], v.r.size[2], v.r.st[0], v.r.st[1],
             v.r.st[2], v.c.size[0], v.c.size[1], v.c.size[2], v.c.st[0], v.c.st[1], v.c.st[2],
             v.bst, R, K, nb, D);
    std::string key = b;
    for (int q = 0; q < v.nsub; q++) key += "," + std::to_string(v.sub[q]);
    return key;
}

// persistent digit pass: as many blocks as fit on the SMs at once
template <int D>
int launch_pack_digits(kvft_ctx *ctx, const PackView &v, int R, int K, int ld, int rows_fast,
                       int ktn, int rtn, long long tiles, Packed *out) {
    int per_sm = 1;
    KV_TRY(kv_blocks_per_sm(ctx, pack_digits_kernel<D>, 256, 0, &per_sm));
    const int grid = (int)std::min(tiles, (long long)per_sm * ctx->sm_count);
    kv_launch(ctx, pack_digits_kernel<D>, grid, 256, 0, v, R, K, ld, rows_fast, ktn, rtn,
              (int)tiles, out->ex, out->planes);
    return KVFT_OK;
}

template <int D>
int launch_pack_cluster(kvft_ctx *ctx, const PackView &v, int R, int K, int ld, int nb,
                        int rows_fast, Packed *out) {
    KV_TRY(kv_smem_optin(ctx, pack_cluster_kernel<D>, pack_slab_smem(PC_SLAB)));
    // slabs of at most 256, longer ones only for K > 2048; shorter ones while
    // the blocks do not fill the SMs
    const int rtiles = (R + PC_R - 1) / PC_R;
    const long long tiles = (long long)rtiles * nb;
    int ncta = std::min(PC_MAX, (K + 255) / 256);
    while (ncta < PC_MAX && tiles * ncta < 2LL * ctx->sm_count && K > 64 * ncta) ncta++;
    const int slab = ((K + ncta - 1) / ncta + 31) / 32 * 32;
    ncta = (K + slab - 1) / slab;
    if (tiles * ncta > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "pack: too many row tiles");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * ncta));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = pack_slab_smem(slab);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ncta;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    KV_CHECK(ctx, cudaLaunchKernelEx(&cfg, pack_cluster_kernel<D>, v, R, K, ld, rows_fast,
                                     rtiles, ncta, slab, out->ex, out->planes));
    return kv_launch_check(ctx, "pack_cluster");
}

template <int D, int KT>
int launch_pack_rows(kvft_ctx *ctx, const PackView &v, int R, int K, int ld, int nb,
                     int rows_fast, int rtiles, Packed *out) {
    constexpr size_t smem = pack_rows_smem(KT);
    int per_sm = 1;
    KV_TRY(kv_smem_optin(ctx, pack_rows_kernel<D, KT>, smem));
    KV_TRY(kv_blocks_per_sm(ctx, pack_rows_kernel<D, KT>, 256, smem, &per_sm));
    const long long ntiles = (long long)rtiles * nb;
    if (ntiles > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "pack: too many row tiles");
    const int grid = (int)std::min(ntiles, (long long)per_sm * ctx->sm_count);
    kv_launch(ctx, pack_rows_kernel<D, KT>, grid, 256, smem, v, R, K, ld, rows_fast, rtiles,
              (int)ntiles, out->ex, out->planes);
    return kv_launch_check(ctx, "pack_rows");
}

template <int D>
int pack_rows_s(kvft_ctx *ctx, const PackView &v, int R, int K, int ld, int nb, int rows_fast,
                int rtiles, Packed *out) {
    if (K <= PT_K) return launch_pack_rows<D, 1>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    if (K <= 2 * PT_K)
        return launch_pack_rows<D, 2>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    if (K > PR_KMAX) return launch_pack_cluster<D>(ctx, v, R, K, ld, nb, rows_fast, out);
    return launch_pack_rows<D, 4>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
}

int pack_rows(kvft_ctx *ctx, const PackView &v, int R, int K, int ld, int nb, int D,
              int rows_fast, int rtiles, Packed *out) {
    switch (D) {
    case 2: return pack_rows_s<2>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    case 3: return pack_rows_s<3>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    case 4: return pack_rows_s<4>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    case 5: return pack_rows_s<5>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    case 6: return pack_rows_s<6>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    case 7: return pack_rows_s<7>(ctx, v, R, K, ld, nb, rows_fast, rtiles, out);
    default: return kv_fail(ctx, KVFT_EINVAL, "pack: digit count out of range");
    }
}

// row exponents of v: cleared, then the maxima of k ranges by atomics
int launch_pack_exp(kvft_ctx *ctx, const PackView &v, int R, int K, int nb, int *ex) {
    const int rows_fast = (kidx_fast_stride(v.r) == 1 && kidx_fast_stride(v.c) != 1) ? 1 : 0;
    KV_CHECK(ctx, cudaMemsetAsync(ex, 0x80, (size_t)nb * R * sizeof(int), ctx->stream));
    const dim3 g((K + PT_K - 1) / PT_K, (unsigned)((R + PT_R - 1) / PT_R), nb);
    if (g.y > 65535) return kv_fail(ctx, KVFT_EINVAL, "pack: too many rows");
    if (g.z > 65535) return kv_fail(ctx, KVFT_EINVAL, "pack: batch too large");
    // long rows: each exponent block walks up to 16 k tiles, so that about
    // 32 blocks per SM remain and the atomics per row drop accordingly
    const long long tiles = (long long)g.x * g.y * g.z;
    const int ktiles = (int)std::max(1LL, std::min(16LL, tiles / (32LL * ctx->sm_count)));
    const dim3 ge((g.x + ktiles - 1) / ktiles, g.y, g.z);
    kv_launch(ctx, pack_exp_kernel, ge, 256, 0, v, R, K, rows_fast, ktiles, ex);
    return kv_launch_check(ctx, "pack_exp");
}

}  // namespace

int kv_tc_pack(kvft_ctx *ctx, const char *key, const PackView &v, int R, int K, int nb, int D,
               Packed *out) {
    const int S = dig_planes(D);
    const int ld = (K + 63) / 64 * 64;
    const size_t plane_bytes = (size_t)R * ld * 2;
    const size_t pbytes = ((size_t)nb * S * plane_bytes + 1023) / 1024 * 1024;
    const size_t bytes = pbytes + (size_t)nb * R * sizeof(int);
    out->R = R;
    out->ld = ld;
    out->K = K;
    out->nb = nb;
    if (v.nb > 65535) return kv_fail(ctx, KVFT_EINVAL, "pack: batch too large");
    void *buf = nullptr;
    std::string ckey;
    if (v.stable && ctx->pack_cache_on) {
        // an integral block packed during an earlier residual evaluation
        ckey = pack_key(v, R, K, nb, D);
        auto it = ctx->pack_cache.find(ckey);
        if (it != ctx->pack_cache.end()) {
            out->planes = (uint16_t *)it->second.first;
            out->ex = (int *)((uint8_t *)it->second.first + pbytes);
            return KVFT_OK;
        }
        // keep it only while a tenth of the device stays free
        size_t fr = 0, tot = 0;
        if (kv_mem_info(ctx, &fr, &tot) == KVFT_OK && fr > bytes + tot / 10 &&
            kv_dev_alloc(ctx, bytes, &buf) == KVFT_OK) {
            ctx->pack_cache[ckey] = {buf, bytes};
            ctx->scratch_gen++;
        } else {
            cudaGetLastError();
            buf = nullptr;
        }
    }
    if (!buf) KV_TRY(kv_scratch(ctx, key, bytes, &buf));
    out->planes = (uint16_t *)buf;
    out->ex = (int *)((uint8_t *)buf + pbytes);
    KvProfScope prof(ctx, KV_CAT_PACK, 8.0 * nb * (double)R * K + (double)nb * S * plane_bytes);
    // coalesce global reads along the contiguous index
    const int rows_fast = (kidx_fast_stride(v.r) == 1 && kidx_fast_stride(v.c) != 1) ? 1 : 0;
    const long long rtiles = (R + PT_R - 1) / PT_R;
    if (rtiles > 65535) return kv_fail(ctx, KVFT_EINVAL, "pack: too many rows");
    if (K <= PC_MAX * PC_SLAB) return pack_rows(ctx, v, R, K, ld, nb, D, rows_fast, (int)rtiles, out);
    KV_TRY(launch_pack_exp(ctx, v, R, K, nb, out->ex));
    const dim3 g((K + PT_K - 1) / PT_K, (unsigned)rtiles, nb);
    const long long tiles = (long long)g.x * g.y * g.z;
    if (tiles > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "pack: too many tiles");
    switch (D) {
#define KV_PACK_CASE(s_)                                                                   \
    case s_:                                                                               \
        KV_TRY(launch_pack_digits<s_>(ctx, v, R, K, ld, rows_fast, g.x, g.y, tiles, out)); \
        break;
        KV_PACK_CASE(2) KV_PACK_CASE(3) KV_PACK_CASE(4) KV_PACK_CASE(5) KV_PACK_CASE(6)
        KV_PACK_CASE(7)
#undef KV_PACK_CASE
    default: return kv_fail(ctx, KVFT_EINVAL, "pack: digit count out of range");
    }
    KV_TRY(kv_launch_check(ctx, "pack_digits"));
    return KVFT_OK;
}

int kv_tc_exps(kvft_ctx *ctx, const char *key, const PackView &v, int R, int K, int nb,
               Packed *out) {
    void *buf = nullptr;
    KV_TRY(kv_scratch(ctx, key, (size_t)nb * R * sizeof(int), &buf));
    out->planes = nullptr;
    out->ex = (int *)buf;
    out->R = R;
    out->ld = out->K = K;
    out->nb = nb;
    KvProfScope prof(ctx, KV_CAT_PACK, 8.0 * nb * (double)R * K);
    return launch_pack_exp(ctx, v, R, K, nb, out->ex);
}

PackView kv_tc_group_view(const double *p, const KIdx &r, const KIdx &c, long long bst, int stable,
                          int nb, int n, const long long *off, int *which) {
    PackView v{p, r, c, bst, stable, nb, 0, {}};
    for (int q = 0; q < n; q++) {
        which[q] = (int)(std::find(v.sub, v.sub + v.nsub, off[q]) - v.sub);
        if (which[q] == v.nsub) v.sub[v.nsub++] = off[q];
    }
    return v;
}

bool kv_tc_pow2(double alpha, int *exp, unsigned *sign) {
    int ex = 0;
    const bool yes = std::fabs(std::frexp(alpha, &ex)) == 0.5;
    *exp = yes ? ex - 1 : 0;
    *sign = yes && alpha < 0 ? 0x80000000u : 0u;
    return yes;
}

namespace {

// C = beta C + the copies of its K ranges, product after product and range
// after range: one thread per element (rows fastest, as the copies are), y = block
// of C, z = batch entry.
struct SumRanges {
    int beg[KV_MAXPROD + 1], prod[KV_MAXPROD];
    long long coff[KV_MAXPROD];
};

__global__ void __launch_bounds__(256)
sum_ranges_kernel(int M, int MN, int nranges, double beta, KOut C, const double *__restrict__ parts,
                  long long c_split, const __grid_constant__ SumRanges s) {
    if (!kv_depend()) return;
    const int e = blockIdx.x * 256 + threadIdx.x;
    if (e >= MN) return;
    const double *part = parts + (long long)blockIdx.z * MN + e;
    double acc = 0.0;
    for (int q = s.beg[blockIdx.y]; q < s.beg[blockIdx.y + 1]; q++) {
        const double *x = part + s.prod[q] * nranges * c_split;
        for (int r = 0; r < nranges; r++) acc += x[r * c_split];
    }
    const int n = e / M, m = e - n * M;
    double *d = C.p + (long long)blockIdx.z * C.bst + s.coff[blockIdx.y] + C.r.off(m) + C.c.off(n);
    *d = beta == 0.0 ? acc : fma(beta, *d, acc);
}

// The stride-1 index of a view: its fastest dimension of extent > 1 has
// element stride 1 (or the index has a single value).
bool unit_stride(const KIdx &x) {
    const long long f = kidx_fast_stride(x);
    return f == 1 || f == 0;
}

constexpr size_t SMEM_CAP = 225 * 1024;
// Below half of an SM's shared memory two CTAs could share an SM and the
// second one's 512-column TMEM allocation would block: always take more.
constexpr size_t SMEM_FLOOR = 120 * 1024;

// Launches the persistent kernel, one CTA per SM.
template <int TN, bool FF, int KBT, int DL, bool CV = false>
int launch_tc(kvft_ctx *ctx, const CUtensorMap &ma, const CUtensorMap &mb, TcParams &p) {
    if constexpr (!CV && TN <= 64)
        if (p.A) return launch_tc<TN, FF, KBT, DL, true>(ctx, ma, mb, p);
    auto kern = tc_gemm_kernel<TN, FF, KBT, DL, CV>;
    int NS = 2;
    while (NS < 8 && tc_smem(p.S, NS + 1, TN, KBT, CV) <= SMEM_CAP) NS++;
    if (tc_smem(p.S, NS, TN, KBT, CV) > SMEM_CAP)
        return kv_fail(ctx, KVFT_EINVAL, "tensor-core gemm: stages exceed shared memory");
    p.NS = NS;
    const size_t smem = std::max(tc_smem(p.S, NS, TN, KBT, CV), SMEM_FLOOR);
    KV_TRY(kv_smem_optin(ctx, kern, SMEM_CAP));
    const int grid = std::min(p.units, ctx->sm_count);
    KvProfScope prof(ctx, ctx->gemm_cat, ctx->gemm_work);
    kv_launch(ctx, kern, grid, NTHREADS + (CV ? 32 * NCV : 0), smem, ma, mb, p);
    return kv_launch_check(ctx, "tc_gemm");
}

// Products whose A the kernel converts itself: one tile, K beyond the packing
// in one pass (so that packing would read A twice, write and read its planes),
// A not a cached operand, its row a single index and its K contiguous, so that
// a warp reads a row's neighbouring values.  The K ranges of all products give
// every SM a unit (a residual of one tau point, 37 virtual and 21 occupied spin
// orbitals, does not: there packing, which uses all SMs, is 1.5 % faster), and
// the products are few enough that ranges run as units of their own (C
// pre-scaled, every write an addition).  Exponents and contraction of the
// F_ae, F_mi and R1 reductions, before and now: 114 spin orbitals, three tau
// points a launch, three levels 14.4 -> 12.6 ms a step, six levels 21.8 -> 16.2;
// 66 and 16, three levels 3.5 -> 3.0; 54 and 10, seven levels 1.6 -> 1.35.
bool cv_fits(kvft_ctx *ctx, int M, int N, int K, int batch, int nprod, const KMat &A) {
    return M <= CV_M && N <= 64 && batch < 2 * ctx->sm_count && A.r.size[0] == 1 &&
           A.r.size[1] == 1 && K > PC_MAX * PC_SLAB && !A.stable &&
           kidx_fast_stride(A.c) == 1 &&
           (long long)batch * nprod * ((K + KRANGE - 1) / KRANGE) >= ctx->sm_count;
}

int gemm_tc_run(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
                const KMat &B, double beta, const KOut &C, int D, const KvProds &g, bool cv) {
    const int S = dig_planes(D);
    // D >= 4: three to five levels, FP32 pairs or integers, TN = 64 (48 at D = 7, see the
    // kernel) and 32-deep k-blocks (up to five digit
    // planes per stage); D <= 3: 64-deep k-blocks, so that every TMA box row is
    // a full 128-byte line, and TN = 128 unless C has at most 64 columns (then
    // 64-wide tiles keep all eight epilogue warps busy)
    const bool ff = D >= 4;
    const int tn = D == 7 && (!cv || N <= 48) ? 48 : (ff || N <= 64) ? 64 : 128;
    const int kchunk = D == 7 ? Dig<7>::KCHUNK : Dig<6>::KCHUNK;
    const int kb = ff ? 32 : 64;
    const int nbA = A.bst ? batch : 1, nbB = B.bst ? batch : 1;
    int wa[KV_MAXPROD], wb[KV_MAXPROD];
    // B is K x N; its K-major form has rows = N (B's column index), cols = K
    const PackView va = kv_tc_group_view(A.p, A.r, A.c, A.bst, A.stable, nbA, g.n, g.oa, wa);
    const PackView vb = kv_tc_group_view(B.p, B.c, B.r, B.bst, B.stable, nbB, g.n, g.ob, wb);
    Packed pa, pb;
    if (cv) KV_TRY(kv_tc_exps(ctx, "tc_pack_a", va, M, K, va.nsub * nbA, &pa));
    else KV_TRY(kv_tc_pack(ctx, "tc_pack_a", va, M, K, va.nsub * nbA, D, &pa));
    KV_TRY(kv_tc_pack(ctx, "tc_pack_b", vb, N, K, vb.nsub * nbB, D, &pb));
    const long long rows_a = (long long)va.nsub * nbA * S * M, rows_b = (long long)vb.nsub * nbB * S * N;
    if (rows_a > 0x7FFFFFFFLL || rows_b > 0x7FFFFFFFLL)
        return kv_fail(ctx, KVFT_EINVAL, "tensor-core gemm: operand too large");
    CUtensorMap ma = {}, mb;
    if (!cv) KV_TRY(kv_tc_map(ctx, &ma, pa.planes, pa.K, pa.ld, rows_a, kb, TM));
    KV_TRY(kv_tc_map(ctx, &mb, pb.planes, pb.K, pb.ld, rows_b, kb, tn));
    const int mt = (M + TM - 1) / TM, nt = (N + tn - 1) / tn;
    const int nkb_total = (K + kb - 1) / kb;
    const long long tiles = (long long)mt * nt * batch;
    // K ranges.  Fewer output tiles than two waves of SMs and several ranges of
    // 2048: every range of every product becomes a unit of its own and adds
    // into C with FP64 atomics (C pre-scaled by beta).  At D >= 4 the ranges
    // may be shorter (the exact sums stay so): while there are fewer units than
    // SMs, down to 256 deep (below that the pipeline's start and the additions
    // cost what the other SMs would save).  Where only that cuts K, the ranges
    // go to copies of C, at most two tiles per SM, which one more launch (in
    // place of the scaling) adds in a fixed order: a sum of up to 2048 terms
    // is repeatable to the bit, as it is uncut.  D <= 3 keeps 2048, which is part
    // of its rounding.  37 x 37 outputs against K = 16317, one product, seven
    // levels: 40 us on 8 SMs; the residual of 37 virtual and 21 occupied spin
    // orbitals 1067 -> 962 us, a solve of 38 and 10 points 53.6 -> 52.8 ms.
    int nranges = (nkb_total + KRANGE / kb - 1) / (KRANGE / kb);
    bool par = nranges > 1 && tiles < 2LL * ctx->sm_count;
    const long long now = tiles * (par ? (long long)nranges * g.n : kv_group_tab(g, false).ncb);
    bool ordered = false;
    if (ff && now < ctx->sm_count) {
        ordered = nranges == 1;
        const long long want = (ctx->sm_count + tiles * g.n - 1) / (tiles * g.n);
        nranges = (int)std::max<long long>(nranges, std::min<long long>(want, K / 256));
        par = nranges > 1;
        ordered = ordered && par;
    }
    const int split_kb = (nkb_total + nranges - 1) / nranges;     // balanced ranges
    nranges = (nkb_total + split_kb - 1) / split_kb;
    const int nchunks = (split_kb + kchunk / kb - 1) / (kchunk / kb);
    const int chunk_kb = (split_kb + nchunks - 1) / nchunks;      // balanced chunks
    const KvGroupTab tab = kv_group_tab(g, par);
    const long long units = tiles * (par ? nranges : 1) * tab.ncb;
    if (units > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "tensor-core gemm: too many tiles");
    const KvGroupTab blocks = kv_group_tab(g, false);
    if (par && !ordered && beta != 1.0)
        KV_TRY(kv_scale_blocks(ctx, M, N, batch, beta, C, blocks.ncb, blocks.coff));
    TcParams p;
    p.batch = batch;
    for (int c = 0; c <= tab.ncb; c++) p.beg[c] = tab.beg[c];
    for (int c = 0; c < tab.ncb; c++) p.coff[c] = tab.coff[c];
    for (int q = 0; q < g.n; q++) {
        const int x = wa[tab.prod[q]], y = wb[tab.prod[q]];
        p.arow[q] = x * nbA * S * M, p.aex[q] = x * nbA * M;
        p.brow[q] = y * nbB * S * N, p.bex[q] = y * nbB * N;
        p.oa[q] = g.oa[tab.prod[q]];
    }
    p.A = cv ? A.p : nullptr;
    if (cv)                               // bytes it must move: A as FP64, B's planes, C
        ctx->gemm_work = g.n * (8.0 * M * (double)K * nbA + 2.0 * S * N * (double)K * nbB) +
                         8.0 * M * N * (double)batch * tab.ncb * (beta != 0.0 ? 2 : 1);
    p.ar = A.r.st[2], p.Ac = A.c, p.a_bst = A.bst, p.dv_ac = kidx_div(A.c);
    p.K = K;
    p.M = M;
    p.N = N;
    p.mt = mt;
    p.nt = nt;
    p.units = (int)units;
    p.nsplit = par ? nranges : 1;
    p.split_kb = par ? split_kb : nkb_total;
    p.chunk_kb = chunk_kb;
    p.flush_kb = std::max(1, WFLUSH / kb / chunk_kb) * chunk_kb;
    p.nkb_total = nkb_total;
    p.S = S;
    p.D = D;
    p.NS = 0;
    p.Mp = pa.R;
    p.Np = pb.R;
    p.a_batch_rows = (nbA > 1) ? S * pa.R : 0;
    p.b_batch_rows = (nbB > 1) ? S * pb.R : 0;
    p.ea = pa.ex;
    p.eb = pb.ex;
    p.ea_bst = (nbA > 1) ? pa.R : 0;
    p.eb_bst = (nbB > 1) ? pb.R : 0;
    p.alpha = alpha;
    p.beta = ordered ? 0.0 : par ? 1.0 : beta;
    p.alpha_pow2 = kv_tc_pow2(alpha, &p.alpha_exp, &p.alpha_sign);
    p.C = C;
    p.c_split = 0;
    if (ordered) {
        // copies [product][range][batch][n][m]
        const long long mn = (long long)M * N;
        void *parts = nullptr;
        KV_TRY(kv_scratch(ctx, "tc_ranges", sizeof(double) * mn * batch * nranges * g.n, &parts));
        p.C = KOut{(double *)parts, kidx1(M, 1), kidx1(N, M), mn};
        p.c_split = mn * batch;
        for (int c = 0; c < tab.ncb; c++) p.coff[c] = tab.prod[c] * nranges * p.c_split;
    }
    p.err = ctx->dflag;
    p.dv_split = fastdiv(p.nsplit);
    p.dv_perb = fastdiv(p.mt * p.nt);
    p.dv_gsz = fastdiv(GROUP_M * p.nt);
    p.dv_batch = fastdiv(batch);
    p.dv_cr2 = fastdiv(p.C.r.size[2]);
    p.dv_cr1 = fastdiv(p.C.r.size[1]);
    const auto run = [&]() -> int {
        switch (D) {
        case 2:
            return tn == 64 ? launch_tc<64, false, 64, 2>(ctx, ma, mb, p)
                            : launch_tc<128, false, 64, 2>(ctx, ma, mb, p);
        case 3:
            return tn == 64 ? launch_tc<64, false, 64, 3>(ctx, ma, mb, p)
                            : launch_tc<128, false, 64, 3>(ctx, ma, mb, p);
        case 4: return launch_tc<64, true, 32, 4>(ctx, ma, mb, p);
        case 5: return launch_tc<64, true, 32, 5>(ctx, ma, mb, p);
        case 6: return launch_tc<64, true, 32, 6>(ctx, ma, mb, p);
        default:
            return tn == 64 ? launch_tc<64, true, 32, 7, true>(ctx, ma, mb, p)
                            : launch_tc<48, true, 32, 7>(ctx, ma, mb, p);
        }
    };
    KV_TRY(run());
    if (!ordered) return KVFT_OK;
    SumRanges sr;
    for (int c = 0; c <= blocks.ncb; c++) sr.beg[c] = blocks.beg[c];
    for (int c = 0; c < blocks.ncb; c++) sr.coff[c] = blocks.coff[c];
    for (int q = 0; q < g.n; q++) sr.prod[q] = blocks.prod[q];
    kv_launch(ctx, sum_ranges_kernel,
              dim3((unsigned)(((long long)M * N + 255) / 256), blocks.ncb, batch), 256, 0, M,
              M * N, nranges, beta, C, (const double *)p.C.p, p.c_split, sr);
    return kv_launch_check(ctx, "sum_ranges");
}

}  // namespace

int kv_gemm_tc(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
               const KMat &B, double beta, const KOut &C, int digits, const KvProds &g) {
    const int D = digits;
    if (D < 2 || D > 7) return kv_fail(ctx, KVFT_EINVAL, "tensor-core digits out of range");
    if (M <= 0 || N <= 0 || batch <= 0) return KVFT_OK;
    if (K <= 0) return kv_gemm_f64(ctx, M, N, K, batch, alpha, A, B, beta, C, g);
    // C^T = B^T A^T, the same products
    const KMat At{B.p, B.c, B.r, B.bst, B.stable};
    const KMat Bt{A.p, A.c, A.r, A.bst, A.stable};
    const KOut Ct{C.p, C.c, C.r, C.bst};
    KvProds gt = g;
    std::swap(gt.oa, gt.ob);
    if (kv_thin_fits(M, N, K, batch, A, B, C))
        return kv_gemm_thin(ctx, M, N, K, batch, alpha, A, B, beta, C, D, g);
    if (kv_thin_fits(N, M, K, batch, At, Bt, Ct))
        return kv_gemm_thin(ctx, N, M, K, batch, alpha, At, Bt, beta, Ct, D, gt);
    // The transpose costs nothing but the operand roles.  The epilogue's lanes
    // are the tile rows, so the stride-1 index of C goes to the rows (each
    // store then covers 32 consecutive doubles) unless that extent is short
    // and K long (the unused TMEM lanes would cost MMA time); otherwise the
    // larger extent goes to the rows.
    // A long K against few rows (the reductions to F_ae, F_mi and R1): the side
    // that no cache holds is converted in the kernel.
    if (cv_fits(ctx, M, N, K, batch, g.n, A))
        return gemm_tc_run(ctx, M, N, K, batch, alpha, A, B, beta, C, D, g, true);
    if (cv_fits(ctx, N, M, K, batch, g.n, At))
        return gemm_tc_run(ctx, N, M, K, batch, alpha, At, Bt, beta, Ct, D, gt, true);
    bool swap = M < N;
    const bool rc = unit_stride(C.r), cc = unit_stride(C.c);
    if (rc != cc) {
        const int ext = cc ? N : M;
        if (ext >= 64 || K <= 512) swap = cc;
    }
    if (swap) return gemm_tc_run(ctx, N, M, K, batch, alpha, At, Bt, beta, Ct, D, gt, false);
    return gemm_tc_run(ctx, M, N, K, batch, alpha, A, B, beta, C, D, g, false);
}

int kv_tc_planes(int digits) { return dig_planes(std::min(digits, 7)); }

// Device status word written by bounded waits (0 = fine).
int kv_device_status(kvft_ctx *ctx) {
    int h = 0;
    KV_CHECK(ctx, cudaMemcpyAsync(&h, ctx->dflag, sizeof(int), cudaMemcpyDeviceToHost,
                                  ctx->stream));
    KV_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    if (h != 0) {
        cudaMemsetAsync(ctx->dflag, 0, sizeof(int), ctx->stream);
        return kv_fail(ctx, KVFT_ETIMEOUT,
                       "tensor-core GEMM: a bounded device wait expired (code " +
                           std::to_string(h) + ")");
    }
    return KVFT_OK;
}

// Plain row-major GEMM through the selected engine (test and measurement hook):
// C[M][N] = A[M][K] B[K][N] for `batch` consecutive matrices, device pointers.
extern "C" int kvft_gemm(kvft_ctx *ctx, int M, int N, int K, int batch, int precision,
                         int digits, const double *A, const double *B, double *C) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_gemm: not on a dry-run context");
    if (!ctx || M <= 0 || N <= 0 || K <= 0 || batch <= 0 || !A || !B || !C)
        return kv_fail(ctx, KVFT_EINVAL, "kvft_gemm: bad argument");
    cudaSetDevice(ctx->device);
    KMat a{A, kidx1(M, K), kidx1(K, 1), (long long)M * K};
    KMat b{B, kidx1(K, N), kidx1(N, 1), (long long)K * N};
    KOut c{C, kidx1(M, N), kidx1(N, 1), (long long)M * N};
    kv_gemm_prof_set(ctx, M, N, K, batch, batch, batch, 0.0, precision != KVFT_PREC_FP64);
    int st;
    if (precision == KVFT_PREC_FP64)
        st = kv_gemm_f64(ctx, M, N, K, batch, 1.0, a, b, 0.0, c, kv_one_prod());
    else
        st = kv_gemm_tc(ctx, M, N, K, batch, 1.0, a, b, 0.0, c, digits, kv_one_prod());
    if (st != KVFT_OK) return st;
    return kv_device_status(ctx);
}

// Device helpers and host entry points shared by the tensor-core contraction
// kernels (kvft_tc.cu: the general tiles; kvft_tc_thin.cu: a big tensor with a
// small matrix).
#pragma once

#include "kvft_internal.h"

#include <cuda.h>
#include <cuda_bf16.h>

namespace {

constexpr int TM = 128;

// ---- digit schemes -------------------------------------------------------------
// The digit count D = 2..7 of the interface names an accuracy.  A scheme writes
// y, |y| < 1/2, as sum_s d_s 2^-pos(s) with S digits of bits(s) bits (balanced:
// |d_s| <= 2^(bits(s) - 1)), stored as P_s = d_s 2^(C - pos(s)), exact in
// BF16; products P_s P_t of one level s + t add up in one FP32
// accumulator, the levels 2 .. NL + 1 are kept, and a sum runs over at most
// KCHUNK terms before it is read out.
//   D <= 6  seven-bit digits, S = NL = D - 1.
//   D = 7   digits of 8, 9, 9, 9 and 9 bits, five levels: 15 products; seven-bit
//           digits need 21 for six planes.
// BF16 holds balanced nine-bit digits, so the wide ones spend no product on
// bits that the type leaves empty.  What bounds the width is the rounding of
// the FP32 sums: they are exact up to 2^24, and a level's weight falls by 2^-9
// (2^-7) from one level to the next.  KCHUNK keeps exact by the digits' bounds
// what weighs enough to show beside the planes' own rounding (2^-45, seven-bit
// planes at D = 7 2^-43):
//   D = 7   128 terms of level 3 (two products of at most 2^7 2^8) reach 2^23,
//           of level 4 (2^7 2^8 twice and 2^8 2^8) 2^24; level 5 may round at
//           weight 2^-43.  With 512 terms level 3 could reach 2^25, and rows
//           of close-by values (1.9605 (1 + 1e-4 x)) came out 10^5 times less
//           accurate than with seven-bit digits; with 256 terms level 4 could,
//           up to 180 times (rows that agree in three digits).
//   D <= 6  2048 terms of level 3 (two products of at most 2^12) reach 2^24.
// So many read-outs want a short epilogue: the running sums of D = 7 are 64-bit
// integers (the levels are integers: half the instructions of an FP32 pair
// and no rounding).  8192^3: 15.6 ms with pairs, 12.6 so; 11.8 read out every
// 512 terms, 12.9 with seven-bit digits.  3249^3 4 times 4.35, 3.51; 3.35; 3.71.
// 361^3 60 times 0.237, 0.231; 0.216; 0.316.  Update of 54 spin orbitals and 10
// tau points 11.0, 10.3; 10.0; two Lambda iterations of 38 and 10 31.0, 29.6; 29.3.
// Error against seven-bit digits with exact sums (K = 33 to 4129; normal,
// constant, few-valued and wide-range operands, A A^T, rows of close-by
// values): 0.2 to 0.8 of it, in the 2-norm and for the largest element.  At D =
// 6 the digits stay as they are: results there are only good to ~1e-9, and any
// other digits would move them by that.
template <int D>
struct Dig {
    static_assert(D >= 2 && D <= 7, "digit count");
    static constexpr bool WIDE = D == 7;
    static constexpr int S = WIDE ? 5 : D - 1;
    static constexpr int NL = S;                       // levels (accumulators)
    static constexpr int KCHUNK = WIDE ? 128 : 2048;
    static constexpr int C = WIDE ? 8 : 7;
    // bits after the point down to and including digit s = 1 .. S
    __host__ __device__ static constexpr int pos(int s) { return WIDE ? 9 * s - 1 : 7 * s; }
    __host__ __device__ static constexpr int bits(int s) {
        return s == 1 ? pos(1) : pos(s) - pos(s - 1);
    }
};
inline int dig_planes(int D) { return D == 7 ? Dig<7>::S : D - 1; }
constexpr unsigned long long WAIT_NS = 2000000000ull;   // 2 s per wait

// Knuth's error-free sum: s + e == a + b exactly (round-to-nearest FP32)
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// FP64 value of x 2^k with sign flipped by `sgn` (0 or 0x80000000), built
// from the FP32 bit pattern in 32-bit halves: high word = sign | exponent
// E - 127 + 1023 + k | top 20 mantissa bits, low word = the other 3 mantissa
// bits at the top (exact; FP32 subnormals, below 2^-126 of the accumulator,
// give 0)
__device__ __forceinline__ double f32_scaled(float x, int k, unsigned sgn) {
    const uint32_t u = __float_as_uint(x);
    const int E = (int)((u >> 23) & 0xFF);
    const int e64 = E + (1023 - 127) + k;
    if (E == 0 || e64 <= 0) return 0.0;
    const uint32_t hi = ((u & 0x80000000u) ^ sgn) | ((uint32_t)e64 << 20) | ((u >> 3) & 0xFFFFFu);
    return __hiloint2double((int)hi, (int)(u << 29));
}

// FP64 value of the integer r times 2^k, rounded to nearest, with sign flipped
// by `sgn`, by integer operations (GB300's FP64 pipe would take 16 clocks a
// warp for the conversion alone).  Below 2^-1022 zero, above the FP64 range
// infinite.
__device__ __forceinline__ double i64_scaled(long long r, int k, unsigned sgn) {
    if (r == 0) return 0.0;
    const unsigned neg = (unsigned)(r >> 63);
    unsigned long long a = r < 0 ? 0ull - (unsigned long long)r : (unsigned long long)r;
    const int z = __clzll((long long)a);
    a <<= z;                                        // 2^63 <= a
    const int E = 63 - z + k + 1023;
    if (E <= 0) return 0.0;
    const unsigned s = (neg & 0x80000000u) ^ sgn;
    if (E >= 0x7FF) return __hiloint2double((int)(s | 0x7FF00000u), 0);
    // 53 bits, ties to even; the leading bit adds one to the exponent field
    // and a carry out of the rounding another
    unsigned long long m = a >> 11;
    const unsigned rest = (unsigned)a & 0x7FFu;
    m += rest > 0x400u || (rest == 0x400u && (m & 1));
    m += (unsigned long long)(E - 1) << 52;
    return __hiloint2double((int)((unsigned)(m >> 32) | s), (int)(unsigned)m);
}

// Raw row exponents are reduced with atomicMax into an array preset to
// 0x80808080 (below any binary exponent); exp_of turns a raw maximum into the
// packing exponent e_r = max + 2 (|x| 2^-e_r < 1/2), or 0 for an all-zero row.
constexpr int EXP_RAW_FLOOR = -1100;
__host__ __device__ __forceinline__ int exp_of(int raw) {
    return raw < EXP_RAW_FLOOR ? 0 : raw + 2;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait: false after WAIT_NS of wall time
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity) {
    if (mbar_try(a, parity)) return true;
    const unsigned long long t0 = gtime();
    while (true) {
        if (mbar_try(a, parity)) return true;
        if (gtime() - t0 > WAIT_NS) return false;
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}

// UMMA shared-memory descriptor of a K-major operand tile whose rows are one
// k-block of KBT BF16 values: KBT = 32 -> 64-byte swizzle (8-row groups 512 B
// apart), KBT = 64 -> 128-byte swizzle (8-row groups 1024 B apart)
template <int KBT>
__device__ __forceinline__ uint64_t desc_of(uint32_t saddr) {
    static_assert(KBT == 32 || KBT == 64, "k-block of 32 or 64");
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;                         // leading byte offset (unused)
    d |= (uint64_t)((8 * KBT * 2) >> 4) << 32;      // stride byte offset
    d |= (uint64_t)1 << 46;                         // descriptor version
    d |= (uint64_t)(KBT == 32 ? 4 : 2) << 61;       // SWIZZLE_64B / SWIZZLE_128B
    return d;
}

// kind::f16 instruction descriptor: BF16 x BF16 -> FP32, K-major A and B,
// M = 128, N = tn
__host__ __device__ constexpr uint32_t idesc_of(int tn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tn >> 3) << 17) |
           ((uint32_t)(TM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                     uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
        : "memory");
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

#define TMEM_LD16(taddr, r)                                                                   \
    asm volatile(                                                                             \
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13," \
        "%14,%15}, [%16];"                                                                    \
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),              \
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),           \
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                                  \
        : "r"(taddr))

#define TMEM_LD8(taddr, r)                                                                    \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"     \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),     \
                   "=r"(r[6]), "=r"(r[7])                                                     \
                 : "r"(taddr))

#define TMEM_LD4(taddr, r)                                                                    \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"                 \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])                             \
                 : "r"(taddr))

// 32 lanes x LW consecutive columns of TMEM
template <int LW>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t *r) {
    static_assert(LW == 16 || LW == 8 || LW == 4, "TMEM load width");
    if constexpr (LW == 16) {
        TMEM_LD16(taddr, r);
    } else if constexpr (LW == 8) {
        TMEM_LD8(taddr, r);
    } else {
        TMEM_LD4(taddr, r);
    }
}

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ int raw_exp(unsigned long long bits) {
    return (bits & 0x7FFFFFFFFFFFFFFFull) ? (int)((bits >> 52) & 0x7FF) - 1023 : -2000;
}

// Digit planes of the pair (x0, x1) of a row with packing exponent e: word s -
// 1 holds the two BF16 values P_s.  The balanced digits of the rounded |x|
// 2^(pos(S) - e) are its bit fields once half a digit has been added at every
// place but the top one, so no digit waits for another's carry; a field
// becomes a float by its place in the significand of 1.5 2^23, and the sign is
// set on the packed word.  Subnormals count as zero.  The kernels that use it
// are bound by its instructions: up to 21 bits it takes 15 a value, where
// shifts by a variable took 20 (with the packing's shorter loops 66 spin
// orbitals, three levels, 21.9 -> 21.4 ms a step, 114 128.0 -> 126.8).
template <int D>
__device__ __forceinline__ void digit_words(unsigned long long x0, unsigned long long x1, int e,
                                            uint32_t (&w)[Dig<D>::S]) {
    using G = Dig<D>;
    constexpr int S = G::S, T = G::pos(S);
    uint32_t sg = 0;
    float f[2][S];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned long long x = h ? x1 : x0;
        const uint32_t hi = (uint32_t)(x >> 32);
        sg |= h ? (hi & 0x80000000u) : (hi >> 31) << 15;
        uint32_t fld[S];
        if constexpr (T <= 21) {
            // the T bits and the rounding bit lie in the significand's high
            // word (|x| 2^-e < 1/2: the shift of the whole is at least 33).
            // |x| 2^(T - e), cut to them, is an FP32 value f < 2^(T - 1) by its
            // bits; floor(f + 1/2) is the rounded integer (f + 1/2 is exact or
            // far from one), taken from the significand of 2^23 + bias + f + 1/2
            // rounded down.  Below 1/2, and for subnormals, f = 0.
            uint32_t bias = 0;
#pragma unroll
            for (int s = 2; s <= S; s++) bias |= 1u << (T - G::pos(s) + G::bits(s) - 1);
            const uint32_t ah = hi & 0x7FFFFFFFu;
            const int least = max((1022 + e - T) * (1 << 20), 1 << 20);
            const float v = __uint_as_float(ah * 8u - ((uint32_t)(896 + e - T) << 23));
            const uint32_t Y = __float_as_uint(__fadd_rd(((int)ah >= least ? v : 0.f) + 0.5f,
                                                         8388608.0f + (float)bias));
#pragma unroll
            for (int s = 1; s <= S; s++)
                fld[s - 1] = (Y >> (T - G::pos(s))) & ((1u << (G::bits(s) + (s == 1))) - 1);
        } else {
            unsigned long long bias = 0;
#pragma unroll
            for (int s = 2; s <= S; s++) bias |= 1ull << (T - G::pos(s) + G::bits(s) - 1);
            const int be = (int)((hi >> 20) & 0x7FF);
            const int n = 1023 + 52 + e - T - be;             // at least 54 - T
            const unsigned long long mant = (x & 0xFFFFFFFFFFFFFull) | (1ull << 52);
            unsigned long long Y = n < 55 && be != 0 ? (mant + (1ull << (n - 1))) >> n : 0ull;
            Y += bias;
#pragma unroll
            for (int s = 1; s <= S; s++) {
                const uint32_t q = (uint32_t)(Y >> (T - G::pos(s)));
                fld[s - 1] = s == 1 ? q : q & ((1u << G::bits(s)) - 1);
            }
        }
#pragma unroll
        for (int s = 1; s <= S; s++) {
            const float sc = 1.0f / (float)(1ull << (G::pos(s) - G::C));   // P_s = d_s sc, exact
            const float off = s == 1 ? 12582912.0f : 12582912.0f + (float)(1 << (G::bits(s) - 1));
            f[h][s - 1] = fmaf(__uint_as_float(0x4B400000u | fld[s - 1]), sc, -off * sc);
        }
    }
#pragma unroll
    for (int s = 0; s < S; s++) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(f[0][s], f[1][s]);
        w[s] = *reinterpret_cast<const uint32_t *>(&v) ^ sg;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Digit packing (kvft_tc.cu): FP64 strided view (rows x K) -> S BF16 planes
// [b][s][R][ld] and row exponents [b][R].
// ---------------------------------------------------------------------------
struct PackView {
    const double *p;
    KIdx r, c;
    long long bst;
    int stable;         // contents fixed while the pack cache is on
    int nb;             // batch entries of one sub-block
    int nsub;           // sub-blocks of the view (the group's distinct operands) and
    long long sub[KV_MAXPROD];   // where they start
    // batch entry b of the packed form: sub-block b / nb, its entry b % nb
    __device__ __forceinline__ const double *base(int b) const {
        const int q = b / nb;
        return p + sub[q] + (long long)(b - q * nb) * bst;
    }
};

struct Packed {
    uint16_t *planes;
    int *ex;
    int R, ld, K, nb;
};


// Packs v (R rows x K, nb packed batch entries, the digits of scheme D) into
// the scratch buffer `key`, or into the cache of stable operands.
int kv_tc_pack(kvft_ctx *ctx, const char *key, const PackView &v, int R, int K, int nb, int D,
               Packed *out);
// The row exponents of v alone, into the scratch buffer `key`.
int kv_tc_exps(kvft_ctx *ctx, const char *key, const PackView &v, int R, int K, int nb,
               Packed *out);
// 2D tensor map over digit planes (K x rows, row stride ld elements); one box
// is a k-block of kb values (swizzled by its 2 kb bytes) by box_rows rows.
int kv_tc_map(kvft_ctx *ctx, CUtensorMap *map, void *base, int K, int ld, long long rows, int kb,
              int box_rows);
// The view of a group's distinct operand sub-blocks; which[q]: the one product
// q uses.
PackView kv_tc_group_view(const double *p, const KIdx &r, const KIdx &c, long long bst, int stable,
                          int nb, int n, const long long *off, int *which);
// alpha = +-2^exp: exp and the sign bit of its high word; false otherwise
// (exp = sign = 0).
bool kv_tc_pow2(double alpha, int *exp, unsigned *sign);

// The contraction of a big tensor with a small matrix (K and one free extent
// at most 64, each a single tensor index): kvft_tc_thin.cu.  kv_thin_fits says
// whether the shape is one it takes, with the big operand as A.
bool kv_thin_fits(int M, int N, int K, int batch, const KMat &A, const KMat &B, const KOut &C);
int kv_gemm_thin(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
                 const KMat &B, double beta, const KOut &C, int D, const KvProds &g);

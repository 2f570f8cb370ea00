// FP64 (DFMA) strided, batched GEMM for the CCSD contractions.
//
// C[b](m,n) = alpha * sum_k A[b](m,k) B[b](k,n) + beta * C[b](m,n), where every
// index is a composite of up to three tensor indices with their own strides
// (KIdx), so permuted views of the n^4 amplitude/integral tensors are read in
// place, for a group of products (the spin blocks of one contraction) per
// launch.
#include "kvft_internal.h"

namespace {

// GB300 issues about 2 FP64 FMAs per clock per SM: a warp's FMA occupies the
// pipe for 16 clocks, in which the SM can issue 64 other instructions and
// serve 16 shared-memory wavefronts.  So FMAs spent on padding are what costs,
// and operand reuse in registers buys little.  Three layouts:
//   rows   a big tensor times a small matrix (N columns at a time, N <= 24): a
//          thread owns one row and all N columns, its A value comes from shared
//          memory once per k and B's by broadcast; no FMA is padding but those
//          of the last, partial row block.
//   square many full 64 x 64 tiles: 256 threads with 4 x 4 outputs each, so an
//          operand value serves four FMAs and the k-blocks have two barriers.
//   flat   everything else: a BM x BN tile of any extents (chosen by the host
//          to divide M and N), its outputs flat over the threads -- o = t + 128
//          i, i < T, along C's contiguous index -- and both operands of every
//          FMA from shared memory (2 LDS against 16 pipe clocks).
// Blocks are small, so several per SM overlap one's loads with another's FMAs.
// Measured, the whole update of 19 plane waves (38 spin orbitals, ng = 10,
// 26.4 GFLOP; 21 ms at the FP64 peak): 64.7 ms with 64 x 64 tiles (19-wide
// outputs padded to 64) and one launch per product, 29.1 ms with flat tiles
// and one launch per group (27.9 with the rows layout); an 8-site ring's
// iteration (8-wide outputs) 4.5 -> 0.6 ms (0.47 with K slices and dependent
// launches).
constexpr int NT = 128, TMAX = 16, BDIM_MAX = 128;

struct F64Params {
    int M, N, K;
    int BM, BN, mt, nt;          // tile and tiles along M and N
    int batch, nsplit, klen;     // K range of one block: klen (a multiple of BK)
    int a_kfast, b_kfast;        // K contiguous in A / B
    int cm_fast;                 // outputs of a tile flat along m (else along n)
    int store;                   // 0 add by atomics (K split), 1 store, 2 add, 3 general beta
    int unit;                    // alpha = 1 (1) or -1 (2): no multiplication by it
    int c_trans;                 // rows layout: C contiguous along its columns
    double alpha, beta;
    const double *A, *B;
    KIdx Ar, Ac, Br, Bc;
    KIdxDiv dar, dac, dbr, dbc, dcr, dcc;
    FastDiv dnt, dmt, dks, dbatch, dflat;
    long long a_bst, b_bst;
    KOut C;
    int beg[KV_MAXPROD + 1];     // sources of each block of C
    long long oa[KV_MAXPROD], ob[KV_MAXPROD], oc[KV_MAXPROD];
};

// block -> (C block, batch, K split, tile), tiles along n fastest
struct F64Tile {
    int tn, tm, ks, b, cb;
    __device__ __forceinline__ F64Tile(const F64Params &p, int u) {
        int q = p.dnt.div(u);
        tn = u - q * p.nt;
        u = q, q = p.dmt.div(u);
        tm = u - q * p.mt;
        u = q, q = p.dks.div(u);
        ks = u - q * p.nsplit;
        cb = p.dbatch.div(q);
        b = q - cb * p.batch;
    }
};

__device__ __forceinline__ void f64_out(const F64Params &p, double *dst, double acc) {
    const double v = p.unit ? (p.unit == 2 ? -acc : acc) : p.alpha * acc;
    if (p.store == 1) *dst = v;
    else if (p.store == 2) *dst += v;
    else if (p.store == 0) atomicAdd(dst, v);
    else *dst = fma(p.beta, *dst, v);
}

__host__ __device__ constexpr size_t f64_smem(int BM, int BN, int BK) {
    const int work = BK * ((BM | 1) + (BN | 1));       // and one sum per thread
    return 8 * (size_t)((work > NT ? work : NT) + 2 * (BM + BN) + 2 * BK);
}

// BK: k values per shared-memory block; 32 where few outputs per thread make
// the loads' latency the chain.  SL > 1: a tile of at most NT / SL outputs,
// whose threads take K in SL interleaved slices.
template <int T, int BK, int SL>
__global__ void __launch_bounds__(NT) gemm_f64_kernel(const __grid_constant__ F64Params p) {
    if (!kv_depend()) return;
    extern __shared__ double sm[];
    const int lda = p.BM | 1, ldb = p.BN | 1;
    double *As = sm;                                   // [BK][lda]
    double *Bs = As + BK * lda;                        // [BK][ldb]
    long long *ar = (long long *)(sm + max(BK * (lda + ldb), NT));   // A row, B column, C row, C column
    long long *bc = ar + p.BM, *cr = bc + p.BN, *cc = cr + p.BM;
    long long *ak = cc + p.BN, *bk = ak + BK;          // K offsets of the current k block
    const int tid = threadIdx.x;
    const F64Tile t(p, blockIdx.x);
    const int m0 = t.tm * p.BM, n0 = t.tn * p.BN;
    const int bm = min(p.BM, p.M - m0), bn = min(p.BN, p.N - n0);
    const int kbeg = t.ks * p.klen, kend = min(p.K, kbeg + p.klen);
    for (int x = tid; x < bm; x += NT) {
        ar[x] = p.dar.off(p.Ar, m0 + x);
        cr[x] = p.dcr.off(p.C.r, m0 + x);
    }
    for (int x = tid; x < bn; x += NT) {
        bc[x] = p.dbc.off(p.Bc, n0 + x);
        cc[x] = p.dcc.off(p.C.c, n0 + x);
    }
    // this thread's outputs as shared-memory offsets m | n << 16; one past the
    // tile (not in `ok`) repeats element 0 and is not stored
    constexpr int CS = NT / SL;                        // threads of a K slice
    const int cnt = p.BM * p.BN, ot = tid % CS, ks = tid / CS, wbase = ot & ~31;
    int mn[T];
    unsigned ok = 0;
    double acc[T];
#pragma unroll
    for (int i = 0; i < T; i++) {
        const int o = ot + NT * i;
        const int q = p.dflat.div(o), r = o - q * (p.cm_fast ? p.BM : p.BN);
        const int m = p.cm_fast ? r : q, n = p.cm_fast ? q : r;
        const bool in = o < cnt && m < bm && n < bn;
        mn[i] = in ? m | n << 16 : 0;
        ok |= (unsigned)in << i;
        acc[i] = 0.0;
    }
    for (int s = p.beg[t.cb]; s < p.beg[t.cb + 1]; s++) {
        const double *A = p.A + (long long)t.b * p.a_bst + p.oa[s];
        const double *B = p.B + (long long)t.b * p.b_bst + p.ob[s];
        for (int k0 = kbeg; k0 < kend; k0 += BK) {
            const int kn = min(BK, kend - k0);
            __syncthreads();                           // the last k block is used up
            if (tid < kn) ak[tid] = p.dac.off(p.Ac, k0 + tid);
            else if (tid >= 64 && tid < 64 + kn) bk[tid - 64] = p.dbr.off(p.Br, k0 + tid - 64);
            __syncthreads();
            if (p.a_kfast) {
                const int k = tid % BK;
                if (k < kn)
                    for (int m = tid / BK; m < bm; m += NT / BK) As[k * lda + m] = A[ar[m] + ak[k]];
            } else {
                for (int x = tid; x < kn * bm; x += NT) {
                    const int k = x / bm, m = x - k * bm;
                    As[k * lda + m] = A[ar[m] + ak[k]];
                }
            }
            if (p.b_kfast) {
                const int k = tid % BK;
                if (k < kn)
                    for (int n = tid / BK; n < bn; n += NT / BK) Bs[k * ldb + n] = B[bc[n] + bk[k]];
            } else {
                for (int x = tid; x < kn * bn; x += NT) {
                    const int k = x / bn, n = x - k * bn;
                    Bs[k * ldb + n] = B[bc[n] + bk[k]];
                }
            }
            __syncthreads();
            const double *as = As + ks * lda, *bs = Bs + ks * ldb;
            for (int k = ks; k < kn; k += SL, as += SL * lda, bs += SL * ldb) {
#pragma unroll
                for (int i = 0; i < T; i++)
                    if (wbase + NT * i < cnt)
                        acc[i] = fma(as[mn[i] & 0xFFFF], bs[mn[i] >> 16], acc[i]);
            }
        }
    }
    if constexpr (SL > 1) {                            // the slices' sums, in order
        __syncthreads();
        As[tid] = acc[0];
        __syncthreads();
        if (ks > 0) return;
#pragma unroll
        for (int q = 1; q < SL; q++) acc[0] += As[ot + q * CS];
    }
    double *C = p.C.p + (long long)t.b * p.C.bst + p.oc[t.cb];
#pragma unroll
    for (int i = 0; i < T; i++)
        if (ok >> i & 1) f64_out(p, C + cr[mn[i] & 0xFFFF] + cc[mn[i] >> 16], acc[i]);
}

// the square layout: 64 x 64 tiles, thread (tx, ty) owns rows ty + 16 i and
// columns tx + 16 j
constexpr int SQ = 64, SQ_K = 16, SQ_T = 256;

__global__ void __launch_bounds__(SQ_T)
gemm_f64_square_kernel(const __grid_constant__ F64Params p) {
    if (!kv_depend()) return;
    __shared__ double As[SQ_K][SQ + 1], Bs[SQ_K][SQ + 1];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const F64Tile t(p, blockIdx.x);
    const int m0 = t.tm * SQ, n0 = t.tn * SQ;
    const int kbeg = t.ks * p.klen, kend = min(p.K, kbeg + p.klen);
    // a thread loads rows and columns ty + 16 r at k = tid % 16 where k is
    // contiguous, else row or column tid % 64 at k = tid / 64 + 4 r
    long long ao[4], bo[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int m = m0 + (p.a_kfast ? ty + 16 * r : tid % SQ);
        const int n = n0 + (p.b_kfast ? ty + 16 * r : tid % SQ);
        ao[r] = m < p.M ? p.dar.off(p.Ar, m) : -1;
        bo[r] = n < p.N ? p.dbc.off(p.Bc, n) : -1;
    }
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
    for (int s = p.beg[t.cb]; s < p.beg[t.cb + 1]; s++) {
        const double *A = p.A + (long long)t.b * p.a_bst + p.oa[s];
        const double *B = p.B + (long long)t.b * p.b_bst + p.ob[s];
        for (int k0 = kbeg; k0 < kend; k0 += SQ_K) {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int ka = p.a_kfast ? tx : tid / SQ + 4 * r;
                const int kb = p.b_kfast ? tx : tid / SQ + 4 * r;
                As[ka][p.a_kfast ? ty + 16 * r : tid % SQ] =
                    ao[r] >= 0 && k0 + ka < kend ? A[ao[r] + p.dac.off(p.Ac, k0 + ka)] : 0.0;
                Bs[kb][p.b_kfast ? ty + 16 * r : tid % SQ] =
                    bo[r] >= 0 && k0 + kb < kend ? B[bo[r] + p.dbr.off(p.Br, k0 + kb)] : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < SQ_K; k++) {
                double a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] = As[k][ty + 16 * i];
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
    double *C = p.C.p + (long long)t.b * p.C.bst + p.oc[t.cb];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty + 16 * i;
        if (m >= p.M) continue;
        const long long ro = p.dcr.off(p.C.r, m);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx + 16 * j;
            if (n < p.N) f64_out(p, C + ro + p.dcc.off(p.C.c, n), acc[i][j]);
        }
    }
}

constexpr int RK = 16;           // k values per shared-memory block of the rows layout

// doubles of the operand blocks, or of the transposed result
__host__ __device__ constexpr int rows_work(int nthr, int T) {
    return RK * (nthr | 1) + RK * T > nthr * (T | 1) ? RK * (nthr | 1) + RK * T : nthr * (T | 1);
}
__host__ __device__ constexpr size_t rows_smem(int nthr, int T) {
    return 8 * (size_t)(rows_work(nthr, T) + nthr + 2 * RK + 2 * T);
}

// the rows layout: blockDim.x rows, columns n0 .. n0 + T - 1
template <int T>
__global__ void __launch_bounds__(NT) gemm_f64_rows_kernel(const __grid_constant__ F64Params p) {
    if (!kv_depend()) return;
    extern __shared__ __align__(16) double sm[];
    const int nthr = blockDim.x, lda = nthr | 1, tid = threadIdx.x;
    double *Bs = sm;                                   // [RK][T]
    double *As = Bs + RK * T;                          // [RK][lda]
    long long *ar = (long long *)(sm + rows_work(nthr, T));   // A row offsets
    long long *ak = ar + nthr, *bk = ak + RK;          // K offsets of the current k block
    long long *bc = bk + RK, *cc = bc + T;
    const F64Tile t(p, blockIdx.x);
    const int m0 = t.tm * p.BM, n0 = t.tn * p.BN;
    const int bm = min(p.BM, p.M - m0), bn = min(p.BN, p.N - n0);
    const bool live = tid < bm;
    const long long aro = live ? p.dar.off(p.Ar, m0 + tid) : 0;
    ar[tid] = aro;
    if (tid < bn) {
        bc[tid] = p.dbc.off(p.Bc, n0 + tid);
        cc[tid] = p.dcc.off(p.C.c, n0 + tid);
    }
    double acc[T];
#pragma unroll
    for (int i = 0; i < T; i++) acc[i] = 0.0;
    for (int s = p.beg[t.cb]; s < p.beg[t.cb + 1]; s++) {
        const double *A = p.A + (long long)t.b * p.a_bst + p.oa[s];
        const double *B = p.B + (long long)t.b * p.b_bst + p.ob[s];
        for (int k0 = 0; k0 < p.K; k0 += RK) {
            const int kn = min(RK, p.K - k0);
            __syncthreads();                           // the last k block is used up
            if (tid < kn) {
                ak[tid] = p.dac.off(p.Ac, k0 + tid);
                bk[tid] = p.dbr.off(p.Br, k0 + tid);
            }
            __syncthreads();
            if (p.a_kfast) {
                const int k = tid % RK;
                if (k < kn)
                    for (int m = tid / RK; m < bm; m += nthr / RK)
                        As[k * lda + m] = A[ar[m] + ak[k]];
            } else if (live) {
                double v[RK];
#pragma unroll
                for (int k = 0; k < RK; k++) v[k] = k < kn ? A[aro + ak[k]] : 0.0;
#pragma unroll
                for (int k = 0; k < RK; k++) As[k * lda + tid] = v[k];
            }
            for (int x = tid; x < kn * T; x += nthr) {
                const int k = x / T, n = x - k * T;
                Bs[x] = n < bn ? B[bc[n] + bk[k]] : 0.0;
            }
            __syncthreads();
            if (live)
                for (int k = 0; k < kn; k++) {
                    const double a = As[k * lda + tid];
                    const double2 *bs = reinterpret_cast<const double2 *>(Bs + k * T);
#pragma unroll
                    for (int i = 0; i < T; i += 2) {
                        if (i < bn) {
                            const double2 b = bs[i / 2];
                            acc[i] = fma(a, b.x, acc[i]);
                            if (i + 1 < bn) acc[i + 1] = fma(a, b.y, acc[i + 1]);
                        }
                    }
                }
        }
    }
    double *C = p.C.p + (long long)t.b * p.C.bst + p.oc[t.cb] +
                (live ? p.dcr.off(p.C.r, m0 + tid) : 0);
    if (p.c_trans) {
        // C contiguous along its columns: the block's rows go through shared
        // memory so that neighbouring threads write neighbouring columns
        __syncthreads();
        double *Cs = sm;                               // [nthr][T | 1], in As and Bs
        long long *cr = ar;
        cr[tid] = C - p.C.p;
#pragma unroll
        for (int i = 0; i < T; i++) Cs[tid * (T | 1) + i] = acc[i];
        __syncthreads();
        for (int x = tid; x < bm * bn; x += nthr) {
            const int m = x / bn, n = x - m * bn;
            f64_out(p, p.C.p + cr[m] + cc[n], Cs[m * (T | 1) + n]);
        }
        return;
    }
    if (!live) return;
#pragma unroll
    for (int i = 0; i < T; i++)
        if (i < bn) f64_out(p, C + cc[i], acc[i]);
}

struct ScaleBlocks {
    int n;
    long long off[64];
};

// one block per (C block, batch, row chunk); threads walk (rows, columns) with
// 32-bit arithmetic
__global__ void __launch_bounds__(256)
scale_blocks_kernel(int M, int N, long long items, int batch, double beta, KOut C,
                    const __grid_constant__ ScaleBlocks g, int rows_fast) {
    if (!kv_depend()) return;
    constexpr int CH = 2048;
    const long long per = (long long)M * N, nch = (per + CH - 1) / CH;
    for (long long it = blockIdx.x; it < items; it += gridDim.x) {
        const long long q = it / nch;
        const long long e0 = (it - q * nch) * CH;
        const int b = (int)(q % batch), blk = (int)(q / batch);
        double *base = C.p + (long long)b * C.bst + g.off[blk];
        const int cnt = (int)min((long long)CH, per - e0);
        for (int x = threadIdx.x; x < cnt; x += 256) {
            const long long e = e0 + x;
            const int fast = rows_fast ? M : N;
            const int o = (int)(e / fast), i = (int)(e - (long long)o * fast);
            double *d = base + C.r.off(rows_fast ? i : o) + C.c.off(rows_fast ? o : i);
            *d = (beta == 0.0) ? 0.0 : beta * (*d);
        }
    }
}

int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Tile BM x BN of at most cap outputs (at most BDIM_MAX either way) that
// divides M x N with the least padding: the shorter extent whole when it
// fits 64, the other as long as the outputs allow, both then evened out over
// their tile counts.
void f64_tile(int M, int N, int cap, int *BM, int *BN) {
    const int s = std::min(M, N), l = std::max(M, N);
    const int side = std::max(1, std::min(std::min(64, s), cap));
    const int bs = ceil_div(s, ceil_div(s, side));
    const int room = std::max(1, std::min(BDIM_MAX, cap / bs));
    const int bl = ceil_div(l, ceil_div(l, room));
    *BM = M <= N ? bs : bl;
    *BN = M <= N ? bl : bs;
}

template <int T, int BK, int SL = 1>
int launch_f64_t(kvft_ctx *ctx, const F64Params &p, int grid) {
    const size_t smem = f64_smem(p.BM, p.BN, BK);
    kv_launch(ctx, gemm_f64_kernel<T, BK, SL>, grid, NT, smem, p);
    return kv_launch_check(ctx, "gemm_f64");
}

template <int T>
int launch_rows_t(kvft_ctx *ctx, const F64Params &p, int grid) {
    kv_launch(ctx, gemm_f64_rows_kernel<T>, grid, p.BM, rows_smem(p.BM, T), p);
    return kv_launch_check(ctx, "gemm_f64_rows");
}

}  // namespace

KvGroupTab kv_group_tab(const KvProds &g, bool split) {
    KvGroupTab t;
    std::vector<long long> off;
    std::vector<std::vector<int>> src;
    for (int q = 0; q < g.n; q++) {
        size_t c = split ? off.size() : std::find(off.begin(), off.end(), g.oc[q]) - off.begin();
        if (c == off.size()) {
            off.push_back(g.oc[q]);
            src.emplace_back();
        }
        src[c].push_back(q);
    }
    std::vector<int> ord(off.size());
    for (size_t c = 0; c < ord.size(); c++) ord[c] = (int)c;
    std::stable_sort(ord.begin(), ord.end(),
                     [&](int x, int y) { return src[x].size() > src[y].size(); });
    int q = 0;
    for (int c : ord) {
        t.beg[t.ncb] = q;
        t.coff[t.ncb++] = off[c];
        for (int x : src[c]) t.prod[q++] = x;
    }
    t.beg[t.ncb] = q;
    return t;
}

int kv_scale_blocks(kvft_ctx *ctx, int M, int N, int batch, double beta, const KOut &C, int n,
                    const long long *off) {
    if (beta == 1.0 || M <= 0 || N <= 0 || batch <= 0 || n <= 0) return KVFT_OK;
    if (ctx->dry) {
        for (int k = 0; k < n; k++) {
            KvDryOp op;
            op.kind = 3;
            op.M = M, op.N = N, op.batch = batch, op.beta = beta, op.C = C;
            op.C.p += off[k];
            ctx->dry->push_back(op);
        }
        return KVFT_OK;
    }
    const int rows_fast = kidx_fast_stride(C.r) == 1;
    for (int k0 = 0; k0 < n; k0 += 64) {
        ScaleBlocks g;
        g.n = std::min(64, n - k0);
        for (int k = 0; k < g.n; k++) g.off[k] = off[k0 + k];
        const long long items = (((long long)M * N + 2047) / 2048) * batch * g.n;
        kv_launch(ctx, scale_blocks_kernel, (unsigned)std::min(items,
                  (long long)ctx->sm_count * 16), 256, 0, M, N, items, batch, beta, C, g,
                  rows_fast);
        KV_TRY(kv_launch_check(ctx, "scale_view"));
    }
    return KVFT_OK;
}

int kv_scale_view(kvft_ctx *ctx, int M, int N, int batch, double beta, const KOut &C) {
    const long long zero = 0;
    return kv_scale_blocks(ctx, M, N, batch, beta, C, 1, &zero);
}

int kv_gemm_f64(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
                const KMat &B, double beta, const KOut &C, const KvProds &g) {
    if (M <= 0 || N <= 0 || batch <= 0) return KVFT_OK;
    KvGroupTab tab = kv_group_tab(g, false);
    if (K <= 0) return kv_scale_blocks(ctx, M, N, batch, beta, C, tab.ncb, tab.coff);
    if (N > 64 && M <= 64) {
        // C^T = B^T A^T: the big operand goes to the rows
        const KMat At{B.p, B.c, B.r, B.bst, B.stable}, Bt{A.p, A.c, A.r, A.bst, A.stable};
        KvProds gt = g;
        std::swap(gt.oa, gt.ob);
        return kv_gemm_f64(ctx, N, M, K, batch, alpha, At, Bt, beta, KOut{C.p, C.c, C.r, C.bst},
                           gt);
    }
    F64Params p;
    p.M = M, p.N = N, p.K = K, p.batch = batch;
    p.nsplit = 1, p.klen = K;
    const long long want = 2LL * ctx->sm_count, nprod = (long long)batch * tab.ncb;
    // The rows layout for a big tensor times a small matrix, with the widest
    // blocks (128, 64 or 32 rows) that leave four per SM; when even 32 rows
    // leave less than two per SM the flat layout balances better (and splits K).
    p.nt = ceil_div(N, 24);
    p.BN = ceil_div(N, p.nt);
    bool rows = N <= 64 && M >= 4 * N;
    for (p.BM = 128; rows; p.BM /= 2) {
        const long long blocks = ceil_div(M, p.BM) * (long long)p.nt * nprod;
        if (blocks >= 2 * want) break;
        if (p.BM == 32) {
            rows = blocks >= want;
            break;
        }
    }
    // The square layout where its tiles are full (at most 2 % of their FMAs on
    // padding) and enough to balance the SMs (six each): 3249^3 61.6 ms in flat
    // tiles, 59.3 here; with 625 tiles (1596^3) flat ones are as fast.  Also
    // where one tile holds C (at most 30 % padding) and a long K gives every SM
    // ranges of 256: 57 x 57, K = 57^3, two products, 2.85 ms in flat tiles,
    // 2.66 here; 40 x 40 (61 % padding) is better off flat.
    const long long sq = (long long)ceil_div(M, SQ) * ceil_div(N, SQ);
    // Sums that are never cut, and so repeatable to the bit: K up to 64, and
    // products that fill the SMs twice with 64 x 64 tiles.
    const bool cut = K > 64 && sq * batch < want;
    const long long sqk = (long long)batch * g.n * (K / 256);
    const bool square_k = cut && !rows && sq == 1 && M * N >= 0.7 * SQ * SQ && K >= 1024 &&
                          sqk >= want && nprod < 2 * want;
    const bool square = square_k || (!rows && sq * nprod >= 6LL * ctx->sm_count &&
                                     (double)sq * SQ * SQ <= 1.02 * M * (double)N);
    if (square) p.BM = p.BN = SQ, p.nt = ceil_div(N, SQ);
    p.mt = rows || square ? ceil_div(M, p.BM) : 0;
    int T = TMAX;
    long long tiles = (long long)p.mt * p.nt * batch;
    if (!rows && !square) {
        // The largest tile (16 outputs per thread) that leaves four blocks per
        // SM to balance the SMs; where neither extent is short, K ranges of 256
        // of a long K count as blocks (every product's, since they then add by
        // atomics).  Else smaller tiles, down to two outputs per thread.
        // Shrinking first reads a long operand once per tile: 57 x 57 outputs,
        // K = 57^3, two products, 5.7 ms in tiles of 57 x 4, 2.85 so.
        const bool longk = cut && K >= 1024 && std::min(M, N) > 32;
        for (;; T /= 2) {
            f64_tile(M, N, NT * T, &p.BM, &p.BN);
            p.mt = ceil_div(M, p.BM);
            p.nt = ceil_div(N, p.BN);
            tiles = (long long)p.mt * p.nt * batch;
            if (T == 2 || tiles * tab.ncb >= 2 * want ||
                (longk && tiles * g.n * (K / 256) >= 2 * want))
                break;
        }
        while (T > 2 && p.BM * p.BN <= NT * T / 2) T /= 2;
        const int bk = T <= 4 ? 32 : 16;
        if (longk && tiles * tab.ncb < 2 * want)
            p.nsplit = (int)std::min<long long>(ceil_div(4 * want, tiles * g.n), K / 256);
        else if (cut && tiles * tab.ncb < want)
            p.nsplit = (int)std::min<long long>(ceil_div(want, tiles * tab.ncb), ceil_div(K, 32));
        p.klen = ceil_div(ceil_div(K, p.nsplit), bk) * bk;
        p.nsplit = ceil_div(K, p.klen);
    }
    if (square_k) {
        p.nsplit = (int)std::min<long long>(ceil_div(want, (long long)batch * g.n), K / 256);
        p.klen = ceil_div(ceil_div(K, p.nsplit), SQ_K) * SQ_K;
        p.nsplit = ceil_div(K, p.klen);
    }
    p.store = beta == 0.0 ? 1 : beta == 1.0 ? 2 : 3;
    if (p.nsplit > 1) {
        KV_TRY(kv_scale_blocks(ctx, M, N, batch, beta, C, tab.ncb, tab.coff));
        tab = kv_group_tab(g, true);
        p.store = 0;
    }
    const long long grid = tiles * p.nsplit * tab.ncb;
    if (grid > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "gemm: too many tiles");
    p.a_kfast = kidx_fast_stride(A.c) == 1 && kidx_fast_stride(A.r) != 1;
    p.b_kfast = kidx_fast_stride(B.r) == 1;
    p.cm_fast = kidx_fast_stride(C.r) == 1 && kidx_fast_stride(C.c) != 1;
    p.c_trans = kidx_fast_stride(C.c) == 1 && kidx_fast_stride(C.r) != 1;
    p.unit = alpha == 1.0 ? 1 : alpha == -1.0 ? 2 : 0;
    p.alpha = alpha, p.beta = beta;
    p.A = A.p, p.B = B.p, p.C = C;
    p.Ar = A.r, p.Ac = A.c, p.Br = B.r, p.Bc = B.c;
    p.dar = kidx_div(A.r), p.dac = kidx_div(A.c), p.dbr = kidx_div(B.r), p.dbc = kidx_div(B.c);
    p.dcr = kidx_div(C.r), p.dcc = kidx_div(C.c);
    p.dnt = fastdiv(p.nt), p.dmt = fastdiv(p.mt), p.dks = fastdiv(p.nsplit);
    p.dbatch = fastdiv(batch);
    p.dflat = fastdiv(p.cm_fast ? p.BM : p.BN);
    p.a_bst = A.bst, p.b_bst = B.bst;
    for (int c = 0; c < tab.ncb; c++) p.oc[c] = tab.coff[c];
    for (int c = 0; c <= tab.ncb; c++) p.beg[c] = tab.beg[c];
    for (int q = 0; q < g.n; q++) {
        p.oa[q] = g.oa[tab.prod[q]];
        p.ob[q] = g.ob[tab.prod[q]];
    }
    KvProfScope prof(ctx, ctx->gemm_cat, ctx->gemm_work);
    if (rows) {
        if (p.BN <= 8) return launch_rows_t<8>(ctx, p, (int)grid);
        if (p.BN <= 16) return launch_rows_t<16>(ctx, p, (int)grid);
        return launch_rows_t<24>(ctx, p, (int)grid);
    }
    if (square) {
        kv_launch(ctx, gemm_f64_square_kernel, (unsigned)grid, SQ_T, 0, p);
        return kv_launch_check(ctx, "gemm_f64_square");
    }
    switch (T) {
    case 16: return launch_f64_t<16, 16>(ctx, p, (int)grid);
    case 8: return launch_f64_t<8, 16>(ctx, p, (int)grid);
    case 4: return launch_f64_t<4, 32>(ctx, p, (int)grid);
    default:
        // At most 64 outputs a tile leave half or more of a block's warps
        // without one, always the same warps and so the same FP64 pipes of the
        // SM; they take slices of K instead (60 products of 8 x 8 outputs, K =
        // 512: 20 -> 12.5 us; an 8-site ring's iteration 503 -> 471 us).
        if (p.BM * p.BN <= 32) return launch_f64_t<2, 32, 4>(ctx, p, (int)grid);
        if (p.BM * p.BN <= 64) return launch_f64_t<2, 32, 2>(ctx, p, (int)grid);
        return launch_f64_t<2, 32>(ctx, p, (int)grid);
    }
}

namespace {

// Moves K component p of both operands' K indices to the fastest position,
// keeping the order of the others (the contraction is the same sum).
void k_to_fast(KIdx &a, KIdx &b, int p) {
    KIdx na = a, nb = b;
    int q = 0;
    for (int d = 0; d < 3; d++)
        if (d != p) {
            na.size[q] = a.size[d];
            na.st[q] = a.st[d];
            nb.size[q] = b.size[d];
            nb.st[q] = b.st[d];
            q++;
        }
    na.size[2] = a.size[p];
    na.st[2] = a.st[p];
    nb.size[2] = b.size[p];
    nb.st[2] = b.st[p];
    a = na;
    b = nb;
}

// The order of the contraction index's components is free.  Operands are read
// in tiles coalesced along their row index or along K, whichever is contiguous
// in memory; when an operand's rows are not, the K component that is
// contiguous in it (if any) is made the fastest, for the larger operand first.
void order_k(int M, int N, int batch, KMat &A, KMat &B) {
    const long long sa = (long long)M * (A.bst ? batch : 1);
    const long long sb = (long long)N * (B.bst ? batch : 1);
    for (int pass = 0; pass < 2; pass++) {
        const bool a_turn = (pass == 0) == (sa >= sb);
        const KIdx &rows = a_turn ? A.r : B.c;      // rows of the packed form
        const KIdx &k = a_turn ? A.c : B.r;
        if (kidx_fast_stride(rows) == 1) continue;
        if (kidx_fast_stride(k) == 1) return;        // already contiguous along K
        for (int d = 0; d < 3; d++)
            if (k.size[d] > 1 && k.st[d] == 1) {
                k_to_fast(A.c, B.r, d);
                return;
            }
    }
}

}  // namespace

void kv_gemm_prof_set(kvft_ctx *ctx, int M, int N, int K, int batch, int nbA, int nbB,
                      double beta, bool tc) {
    // n^6-class: every GEMM dimension is a pair of orbital indices or more;
    // its work is counted in flops, the other contractions' in the bytes the
    // kernel must move (operands as read: BF16 digit planes on the tensor
    // cores, FP64 otherwise; C written, or read and written when added to)
    const long long mn = std::min(std::min(M, N), K), mx = std::max(std::max(M, N), K);
    ctx->gemm_cat = (mn * mn > mx) ? KV_CAT_GEMM6 : KV_CAT_GEMM;
    if (ctx->gemm_cat == KV_CAT_GEMM6) {
        ctx->gemm_work = 2.0 * M * N * (double)K * batch;
    } else {
        const double el = tc ? 2.0 * kv_tc_planes(ctx->digits) : 8.0;
        ctx->gemm_work = el * K * ((double)M * nbA + (double)N * nbB) +
                         8.0 * M * (double)N * batch * (beta != 0.0 ? 2 : 1);
    }
}

int kv_gemm_group(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha,
                  const KMat &A_in, const KMat &B_in, double beta, const KOut &C,
                  const KvProds &g) {
    if (g.n <= 0) return KVFT_OK;
    if (ctx->dry) {
        // one record per product, a later product of the same block adding
        for (int q = 0; q < g.n; q++) {
            KvDryOp op;
            op.kind = 0;
            op.M = M, op.N = N, op.K = K, op.batch = batch;
            op.alpha = alpha;
            op.beta = std::find(g.oc, g.oc + q, g.oc[q]) == g.oc + q ? beta : 1.0;
            op.A = A_in, op.B = B_in, op.C = C;
            op.A.p += g.oa[q], op.B.p += g.ob[q], op.C.p += g.oc[q];
            ctx->dry->push_back(op);
        }
        return KVFT_OK;
    }
    KMat A = A_in, B = B_in;
    order_k(M, N, batch, A, B);
    // Tensor cores for everything but short sums and tiny products, which stay
    // on the FP64 pipe.  Skinny shapes (a few columns against a long K) go to
    // the tensor cores too: even with most of a 128-wide tile idle they beat
    // GB300's FP64 pipe by an order of magnitude.
    const bool tc = ctx->precision != KVFT_PREC_FP64 && K >= 16 &&
                    2.0 * M * N * (double)K * batch >= 2.0e6;
    kv_gemm_prof_set(ctx, M, N, K, batch * g.n, A.bst ? batch * g.n : g.n,
                     B.bst ? batch * g.n : g.n, beta, tc);
    if (ctx->prof) {
        ctx->prof->shape[0] = M, ctx->prof->shape[1] = N;
        ctx->prof->shape[2] = K, ctx->prof->shape[3] = batch * g.n;
    }
    if (!tc) return kv_gemm_f64(ctx, M, N, K, batch, alpha, A, B, beta, C, g);
    return kv_gemm_tc(ctx, M, N, K, batch, alpha, A, B, beta, C, ctx->digits, g);
}

int kv_gemm(kvft_ctx *ctx, int M, int N, int K, int batch, double alpha, const KMat &A,
            const KMat &B, double beta, const KOut &C) {
    return kv_gemm_group(ctx, M, N, K, batch, alpha, A, B, beta, C, kv_one_prod());
}

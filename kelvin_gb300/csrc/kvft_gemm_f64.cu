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
// serve 16 shared-memory wavefronts.  So FMAs spent on padding are the only
// cost that counts, and operand reuse in registers buys nothing.  The tile
// is BM x BN for any extents (chosen by the host to divide M and N, whatever
// the orbital count), its outputs are laid out flat over the threads -- o =
// t + 128 i, i < T, along C's contiguous index, so stores coalesce -- and
// every FMA takes its two operands from shared memory (2 LDS against 16 pipe
// clocks).  Blocks are small (128 threads, under 30 KB), so several per SM
// overlap one's loads with another's FMAs.
// Measured, the whole update of 19 plane waves (38 spin orbitals, ng = 10,
// 26.4 GFLOP; 21 ms at the FP64 peak): 64.7 ms with 64 x 64 tiles (19-wide
// outputs padded to 64) and one launch per product, 29.1 ms with these tiles
// and one launch per group; an 8-site ring's iteration (8-wide outputs)
// 4.5 -> 0.6 ms.
constexpr int NT = 128, BK = 16, TMAX = 16, BDIM_MAX = 128;

struct F64Params {
    int M, N, K;
    int BM, BN, mt, nt;          // tile and tiles along M and N
    int batch, nsplit, klen;     // K range of one block: klen (a multiple of BK)
    int a_kfast, b_kfast;        // K contiguous in A / B
    int cm_fast;                 // outputs of a tile flat along m (else along n)
    int atomic;                  // add into C by atomics (K split over blocks)
    double alpha, beta;
    const double *A, *B;
    KIdx Ar, Ac, Br, Bc;
    long long a_bst, b_bst;
    KOut C;
    int beg[KV_MAXPROD + 1];     // sources of each block of C
    long long oa[KV_MAXPROD], ob[KV_MAXPROD], oc[KV_MAXPROD];
};

__host__ __device__ constexpr size_t f64_smem(int BM, int BN) {
    return 8 * (size_t)(BK * ((BM | 1) + (BN | 1)) + 2 * (BM + BN) + 2 * BK);
}

template <int T>
__global__ void __launch_bounds__(NT) gemm_f64_kernel(const __grid_constant__ F64Params p) {
    extern __shared__ double sm[];
    const int lda = p.BM | 1, ldb = p.BN | 1;
    double *As = sm;                                   // [BK][lda]
    double *Bs = As + BK * lda;                        // [BK][ldb]
    long long *ar = (long long *)(Bs + BK * ldb);      // A row, B column, C row, C column
    long long *bc = ar + p.BM, *cr = bc + p.BN, *cc = cr + p.BM;
    long long *ak = cc + p.BN, *bk = ak + BK;          // K offsets of the current k block
    const int tid = threadIdx.x;
    // block -> (C block, batch, K split, tile), tiles along n fastest
    int u = blockIdx.x;
    const int tn = u % p.nt;
    u /= p.nt;
    const int tm = u % p.mt;
    u /= p.mt;
    const int ks = u % p.nsplit;
    u /= p.nsplit;
    const int b = u % p.batch, cb = u / p.batch;
    const int m0 = tm * p.BM, n0 = tn * p.BN;
    const int bm = min(p.BM, p.M - m0), bn = min(p.BN, p.N - n0);
    const int kbeg = ks * p.klen, kend = min(p.K, kbeg + p.klen);
    for (int x = tid; x < bm; x += NT) {
        ar[x] = p.Ar.off(m0 + x);
        cr[x] = p.C.r.off(m0 + x);
    }
    for (int x = tid; x < bn; x += NT) {
        bc[x] = p.Bc.off(n0 + x);
        cc[x] = p.C.c.off(n0 + x);
    }
    // this thread's outputs; one past the tile repeats the last output and is
    // not stored, and costs FMAs only in a warp that has others
    const int cnt = bm * bn, wbase = tid & ~31;
    short im[T], in[T];
    double acc[T];
#pragma unroll
    for (int i = 0; i < T; i++) {
        const int o = min(tid + NT * i, cnt - 1);
        const int q = p.cm_fast ? o / bm : o / bn;
        const int r = o - q * (p.cm_fast ? bm : bn);
        im[i] = (short)(p.cm_fast ? r : q);
        in[i] = (short)(p.cm_fast ? q : r);
        acc[i] = 0.0;
    }
    for (int s = p.beg[cb]; s < p.beg[cb + 1]; s++) {
        const double *A = p.A + (long long)b * p.a_bst + p.oa[s];
        const double *B = p.B + (long long)b * p.b_bst + p.ob[s];
        for (int k0 = kbeg; k0 < kend; k0 += BK) {
            const int kn = min(BK, kend - k0);
            __syncthreads();                           // the last k block is used up
            if (tid < kn) ak[tid] = p.Ac.off(k0 + tid);
            else if (tid >= 32 && tid < 32 + kn) bk[tid - 32] = p.Br.off(k0 + tid - 32);
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
            const double *as = As, *bs = Bs;
            for (int k = 0; k < kn; k++, as += lda, bs += ldb) {
#pragma unroll
                for (int i = 0; i < T; i++)
                    if (wbase + NT * i < cnt) acc[i] = fma(as[im[i]], bs[in[i]], acc[i]);
            }
        }
    }
    double *C = p.C.p + (long long)b * p.C.bst + p.oc[cb];
#pragma unroll
    for (int i = 0; i < T; i++) {
        if (tid + NT * i >= cnt) break;
        double *dst = C + cr[im[i]] + cc[in[i]];
        const double v = p.alpha * acc[i];
        if (p.atomic) atomicAdd(dst, v);
        else *dst = (p.beta != 0.0) ? v + p.beta * (*dst) : v;
    }
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

template <int T>
int launch_f64_t(kvft_ctx *ctx, const F64Params &p, int grid) {
    const size_t smem = f64_smem(p.BM, p.BN);
    gemm_f64_kernel<T><<<grid, NT, smem, ctx->stream>>>(p);
    return kv_launch_check(ctx, "gemm_f64");
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
        scale_blocks_kernel<<<(unsigned)std::min(items, (long long)ctx->sm_count * 16), 256, 0,
                              ctx->stream>>>(M, N, items, batch, beta, C, g, rows_fast);
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
    F64Params p;
    p.M = M, p.N = N, p.K = K, p.batch = batch;
    // The largest tile (16 outputs per thread) that leaves four blocks per
    // SM to balance the SMs, down to two outputs per thread; then K is split
    // into chunks of at least 64 while fewer than two blocks per SM remain.
    int T = TMAX;
    long long tiles = 0;
    for (;; T /= 2) {
        f64_tile(M, N, NT * T, &p.BM, &p.BN);
        p.mt = ceil_div(M, p.BM);
        p.nt = ceil_div(N, p.BN);
        tiles = (long long)p.mt * p.nt * batch;
        if (T == 2 || tiles * tab.ncb >= 4LL * ctx->sm_count) break;
    }
    const long long want = 2LL * ctx->sm_count;
    p.nsplit = 1;
    if (tiles * tab.ncb < want && K > 64)
        p.nsplit = (int)std::min<long long>(ceil_div(want, tiles * tab.ncb), ceil_div(K, 64));
    p.klen = ceil_div(ceil_div(K, p.nsplit), BK) * BK;
    p.nsplit = ceil_div(K, p.klen);
    p.atomic = p.nsplit > 1;
    if (p.atomic) {
        KV_TRY(kv_scale_blocks(ctx, M, N, batch, beta, C, tab.ncb, tab.coff));
        tab = kv_group_tab(g, true);
    }
    const long long grid = tiles * p.nsplit * tab.ncb;
    if (grid > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "gemm: too many tiles");
    p.a_kfast = kidx_fast_stride(A.c) == 1;
    p.b_kfast = kidx_fast_stride(B.r) == 1;
    p.cm_fast = kidx_fast_stride(C.r) == 1 && kidx_fast_stride(C.c) != 1;
    p.alpha = alpha, p.beta = beta;
    p.A = A.p, p.B = B.p, p.C = C;
    p.Ar = A.r, p.Ac = A.c, p.Br = B.r, p.Bc = B.c;
    p.a_bst = A.bst, p.b_bst = B.bst;
    for (int c = 0; c < tab.ncb; c++) p.oc[c] = tab.coff[c];
    for (int c = 0; c <= tab.ncb; c++) p.beg[c] = tab.beg[c];
    for (int q = 0; q < g.n; q++) {
        p.oa[q] = g.oa[tab.prod[q]];
        p.ob[q] = g.ob[tab.prod[q]];
    }
    KvProfScope prof(ctx, ctx->gemm_cat, ctx->gemm_work);
    switch (T) {
    case 16: return launch_f64_t<16>(ctx, p, (int)grid);
    case 8: return launch_f64_t<8>(ctx, p, (int)grid);
    case 4: return launch_f64_t<4>(ctx, p, (int)grid);
    default: return launch_f64_t<2>(ctx, p, (int)grid);
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
        const double el = tc ? 2.0 * std::min(ctx->digits - 1, 6) : 8.0;
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

// FT-CC grand potential (kelvin/ft_cc_energy.py:7-32):
//   Omega = (1/beta) [ sum_ai t1n[a,i] f[i,a] + sum_abij t2n[a,b,i,j] eri[i,j,a,b] ]
//   t1n = sum_y g_y T1_y,  t2n = sum_y g_y (T2_y/4 + [Qterm] T1_y[a,i] T1_y[b,j]/2)
// One pass over T2 (HBM-bound apart from GB300's slow FP64 FMAs); eri is read
// through a shared-memory transpose so both streams stay coalesced.  Partial
// sums are reduced in a fixed order, so the result is deterministic.
#include "kvft_internal.h"

namespace {

constexpr int TILE = 32;
constexpr int EN_T = 256;

// Block sum of acc (fixed order) into partial[blockIdx.x]; the last block to
// arrive adds the partials in index order and writes (sum) inv_beta to *res, so
// one launch gives a deterministic total.  *count is zero before the launch
// and zero again after it.
__device__ __forceinline__ void finish_sum(double acc, double *red, double *partial,
                                           unsigned *count, double inv_beta, double *res) {
    __shared__ bool last;
    const int t = threadIdx.x;
    red[t] = acc;
    __syncthreads();
    for (int s = EN_T / 2; s > 0; s >>= 1) {
        if (t < s) red[t] += red[t + s];
        __syncthreads();
    }
    if (t == 0) {
        partial[blockIdx.x] = red[0];
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0;
    for (int k = t; k < (int)gridDim.x; k += EN_T) a += __ldcg(partial + k);
    red[t] = a;
    __syncthreads();
    for (int s = EN_T / 2; s > 0; s >>= 1) {
        if (t < s) red[t] += red[t + s];
        __syncthreads();
    }
    if (t == 0) {
        *res = red[0] * inv_beta;
        *count = 0;
    }
}

// This thread's share of sum_y g_y sum_ai T1_y[a,i] f[i,a]
__device__ __forceinline__ double energy1(int ng, int nv, int no, const double *T1,
                                          const double *f, const double *g) {
    double acc = 0.0;
    for (int k = blockIdx.x * EN_T + threadIdx.x; k < nv * no; k += gridDim.x * EN_T) {
        const int a = k / no, i = k - a * no;
        double s = 0.0;
        for (int y = 0; y < ng; y++) s = fma(g[y], T1[(long long)y * nv * no + k], s);
        acc = fma(s, f[i * nv + a], acc);
    }
    return acc;
}

// Blocks walk 32 x 32 tiles of (a,b) x (i,j); thread (tx, ty) takes i,j = ij0 +
// tx and the four (a,b) rows ty + 8k.  Per element and tau point one FP64 FMA,
// s1 += g_y T2_y, and on half of the elements a second: M[ai,bj] = sum_y (g_y
// T1_y[a,i]) T1_y[b,j] is symmetric in its two pairs, so only the rows a <= b
// form it, and those with a < b take it against eri[ij,ab] + eri[ji,ba] (66
// spin orbitals, 16 points: 1.43 -> 1.16 ms; the FP64 pipe's floor is 1.0, the
// memory's 0.38).  The first factors come from a shared table over the few
// (a, i) of the tile, filled for a chunk of tau points at a time.
constexpr int WTAB = 1024;                  // doubles of the (y, a, i) table

__global__ void __launch_bounds__(EN_T, 3)
energy2_kernel(int ng, int nv, int no, const double *__restrict__ T1,
               const double *__restrict__ T2, const double *__restrict__ f,
               const double *__restrict__ eri, const double *__restrict__ g, int qterm, int sh,
               int gx, int tiles, double *partial, unsigned *count, double inv_beta,
               double *res) {
    if (!kv_depend()) return;
    __shared__ double E[TILE][TILE + 1];     // [ij][ab]
    __shared__ double red[EN_T];
    __shared__ double gs[WTAB / 4];          // g_y of the chunk
    __shared__ double wt[WTAB];              // [y][a - a_lo][i - i_lo]: g_y T1_y[a,i]
    __shared__ int tile_live;
    const long long V2 = (long long)nv * nv, O2 = (long long)no * no;
    const int t = threadIdx.x, tx = t % TILE, ty = t / TILE;   // ty in [0, 8)
    double acc = energy1(ng, nv, no, T1, f, g);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long ab0 = (long long)(tile / gx) * TILE, ij0 = (long long)(tile % gx) * TILE;
        __syncthreads();                     // the last tile's tables are used up
        if (sh > 0) {
            // spin blocks: a tile whose (a,b) spin sums and (i,j) spin sums never
            // meet holds only zero amplitudes and adds nothing
            if (t < 32) {
                const long long ab = ab0 + t, ij = ij0 + t;
                unsigned sab = 0, sij = 0;
                if (ab < V2) sab = 1u << ((int)(ab / nv >= sh) + (int)(ab % nv >= sh));
                if (ij < O2) sij = 1u << ((int)(ij / no >= sh) + (int)(ij % no >= sh));
                sab = __reduce_or_sync(0xffffffffu, sab);
                sij = __reduce_or_sync(0xffffffffu, sij);
                if (t == 0) tile_live = (sab & sij) != 0;
            }
            __syncthreads();
            if (!tile_live) continue;
        }
        for (int r = ty; r < TILE; r += 8) {
            const long long ij = ij0 + r, ab = ab0 + tx;
            E[r][tx] = (ij < O2 && ab < V2) ? eri[ij * V2 + ab] : 0.0;
        }
        const long long ab_hi = min(ab0 + TILE, V2) - 1, ij_hi = min(ij0 + TILE, O2) - 1;
        const int a_lo = (int)(ab0 / nv), na = (int)(ab_hi / nv) - a_lo + 1;
        const int i_lo = (int)(ij0 / no), ni = (int)(ij_hi / no) - i_lo + 1;
        const int yc = qterm ? max(1, min(WTAB / 4, WTAB / (na * ni))) : WTAB / 4;
        const long long ij = ij0 + tx;
        const bool live = ij < O2;
        const int i = live ? (int)(ij / no) : 0, j = live ? (int)(ij - (long long)i * no) : 0;
        // row k of this thread: ab0 + ty + 8 k, the last row again past the end
        const int row0 = ty, rows = (int)(ab_hi - ab0);
        auto row = [&](int k) { return (long long)min(row0 + 8 * k, rows); };
        double s1[4] = {0.0, 0.0, 0.0, 0.0}, s2[4] = {0.0, 0.0, 0.0, 0.0};
        const long long sy = (long long)nv * no;
        for (int y0 = 0; y0 < ng; y0 += yc) {
            const int ny = min(yc, ng - y0);
            __syncthreads();
            for (int x = t; x < ny; x += EN_T) gs[x] = g[y0 + x];
            if (qterm)
                for (int x = t; x < ny * na * ni; x += EN_T) {
                    const int yy = x / (na * ni), r = x % (na * ni);
                    const int a = a_lo + r / ni, ii = i_lo + r % ni;
                    wt[x] = g[y0 + yy] * T1[(y0 + yy) * sy + (long long)a * no + ii];
                }
            __syncthreads();
            if (!live) continue;
            const double *t2 = T2 + (long long)y0 * V2 * O2 + ab0 * O2 + ij;
            // four tau points of loads in flight
            int yy = 0;
            for (; yy + 4 <= ny; yy += 4) {
                double v[4][4];
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int k = 0; k < 4; k++) v[q][k] = t2[q * V2 * O2 + row(k) * O2];
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int k = 0; k < 4; k++) s1[k] = fma(gs[yy + q], v[q][k], s1[k]);
                t2 += 4 * V2 * O2;
            }
            for (; yy < ny; yy++) {
#pragma unroll
                for (int k = 0; k < 4; k++) s1[k] = fma(gs[yy], t2[row(k) * O2], s1[k]);
                t2 += V2 * O2;
            }
            if (qterm) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int ab = (int)(ab0 + row(k)), a = ab / nv, b = ab - a * nv;
                    if (a > b) continue;                       // warp-uniform
                    const double *u = T1 + (long long)y0 * sy + (long long)b * no + j;
                    const double *w = wt + (a - a_lo) * ni + (i - i_lo);
#pragma unroll 8
                    for (int z = 0; z < ny; z++) s2[k] = fma(w[z * na * ni], u[z * sy], s2[k]);
                }
            }
        }
        if (live)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int r = ty + 8 * k;
                if (ab0 + r >= V2) continue;
                const double e = E[tx][r];
                acc = fma(0.25 * s1[k], e, acc);
                const int ab = (int)(ab0 + r), a = ab / nv, b = ab - a * nv;
                if (!qterm || a > b) continue;
                const double e2 = a < b ? eri[((long long)j * no + i) * V2 + (long long)b * nv + a]
                                        : 0.0;
                acc = fma(0.5 * s2[k], e + e2, acc);
            }
    }
    finish_sum(acc, red, partial, count, inv_beta, res);
}

// Spin blocks (nv = no = 2h): only the spin-conserving (a, b, i, j) carry
// amplitudes and integrals.  Item (a, i, q) is one h x h block of (b, j): with
// s_a = s_i the blocks s_b = s_j = q (q = 0, 1), otherwise the one block
// s_b = s_i, s_j = s_a (q = 0; q = 1 is empty).  The block's integrals
// eri[i][j][a][b] are read along b into shared memory and its amplitudes
// T2_y[a][b][i][j] along j, so both streams are coalesced and no element
// outside the conserving blocks is read.  The T1 T1 term vanishes unless s_b
// = s_j (T1 is spin-diagonal), i.e. on the s_a = s_i items.
constexpr int ESP_HMAX = 96;                 // h x (h + 1) doubles of shared memory

__global__ void __launch_bounds__(EN_T)
energy2_spin_kernel(int ng, int n, int h, const double *__restrict__ T1,
                    const double *__restrict__ T2, const double *__restrict__ f,
                    const double *__restrict__ eri, const double *__restrict__ g, int qterm,
                    long long items, double *partial, unsigned *count, double inv_beta,
                    double *res) {
    if (!kv_depend()) return;
    extern __shared__ double E[];            // [h][h + 1]: E[j1][b1]
    __shared__ double red[EN_T];
    __shared__ double gs[64], w[64];         // g_y and g_y T1_y[a][i]
    const int t = threadIdx.x, hh = h * h, ld = h + 1;
    const long long n2 = (long long)n * n, P = n2 * n2;
    double acc = energy1(ng, n, n, T1, f, g);
    for (long long it = blockIdx.x; it < items; it += gridDim.x) {
        const int q = (int)(it & 1);
        const long long ai = it >> 1;
        const int a = (int)(ai / n), i = (int)(ai - (long long)a * n);
        const int sa = a >= h, si = i >= h;
        if (sa != si && q) continue;         // block-uniform
        const int sb = sa == si ? q : si, sj = sa == si ? q : sa;
        const bool tt = qterm && sa == si;
        __syncthreads();                     // E, gs, w of the last item are used up
        for (int x = t; x < ng; x += EN_T) {
            gs[x] = g[x];
            w[x] = tt ? g[x] * T1[(long long)x * n2 + (long long)a * n + i] : 0.0;
        }
        for (int x = t; x < hh; x += EN_T) {
            const int j1 = x / h, b1 = x - j1 * h;
            E[j1 * ld + b1] = eri[(((long long)i * n + sj * h + j1) * n + a) * n + sb * h + b1];
        }
        __syncthreads();
        const long long base = ((long long)a * n + sb * h) * n2 + (long long)i * n + sj * h;
        for (int x = t; x < hh; x += EN_T) {
            const int b1 = x / h, j1 = x - b1 * h;
            const double *t2 = T2 + base + (long long)b1 * n2 + j1;
            double s1 = 0.0, s2 = 0.0;
#pragma unroll 4
            for (int y = 0; y < ng; y++) s1 = fma(gs[y], t2[(long long)y * P], s1);
            if (tt) {
                const double *u = T1 + (long long)(sb * h + b1) * n + sj * h + j1;
#pragma unroll 4
                for (int y = 0; y < ng; y++) s2 = fma(w[y], u[(long long)y * n2], s2);
            }
            acc = fma(fma(0.25, s1, 0.5 * s2), E[j1 * ld + b1], acc);
        }
    }
    finish_sum(acc, red, partial, count, inv_beta, res);
}

// Blocks of the dense form: two per SM resident, eight waves of them at most
int energy_grid(int sm_count, long long tiles) {
    return (int)std::max(1LL, std::min(tiles, (long long)sm_count * 16));
}

}  // namespace

// Writes Omega to dres[0] (device).  Uses context scratch.
int kv_energy(kvft_ctx *ctx, int ng, int nv, int no, const double *T1, const double *T2,
              const double *f, const double *eri, const double *g, double beta, int qterm,
              double *dres, int spin_half) {
    const long long V2 = (long long)nv * nv, O2 = (long long)no * no;
    const long long gx = (O2 + TILE - 1) / TILE, gy = (V2 + TILE - 1) / TILE;
    const int sh = (nv == no && nv == 2 * spin_half) ? spin_half : 0;
    const bool spin = sh > 0 && sh <= ESP_HMAX && ng <= 64;
    // spin items (a, i, q), or the 32 x 32 tiles of the dense kernel
    const long long work = spin ? 2LL * nv * nv : gx * gy;
    if (work > 0x7FFFFFFFLL) return kv_fail(ctx, KVFT_EINVAL, "energy: too many tiles");
    const int grid = spin ? (int)std::min<long long>(work, (long long)ctx->sm_count * 8)
                          : energy_grid(ctx->sm_count, work);
    void *part = nullptr;
    KV_TRY(kv_scratch(ctx, "energy_partial", sizeof(double) * grid, &part));
    double *pp = (double *)part;
    unsigned *count = (unsigned *)ctx->dflag + KV_FLAG_ENERGY;
    // algorithmic bytes: T2 (all tau points) + eri + T1; with spin blocks the
    // spin-conserving elements of T2 and eri
    KvProfScope prof(ctx, KV_CAT_ENERGY,
                     8.0 * (((double)ng * V2 * O2 + (double)V2 * O2) * kv_spin_frac(nv, no, sh) +
                            (double)ng * nv * no));
    if (spin) {
        const size_t smem = sizeof(double) * (size_t)sh * (sh + 1);
        KV_TRY(kv_smem_optin(ctx, energy2_spin_kernel, sizeof(double) * ESP_HMAX * (ESP_HMAX + 1)));
        kv_launch(ctx, energy2_spin_kernel, grid, EN_T, smem, ng, nv, sh, T1, T2, f, eri, g, qterm,
                  work, pp, count, 1.0 / beta, dres);
        return kv_launch_check(ctx, "energy2_spin");
    }
    kv_launch(ctx, energy2_kernel, grid, EN_T, 0, ng, nv, no, T1, T2, f, eri, g, qterm, sh, (int)gx,
              (int)work, pp, count, 1.0 / beta, dres);
    return kv_launch_check(ctx, "energy2");
}

extern "C" int kvft_ft_cc_energy(kvft_ctx *ctx, int ng, int nv, int no, const double *T1,
                                 const double *T2, const double *f, const double *eri,
                                 const double *g, double beta, int qterm,
                                 double *omega_host) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_ft_cc_energy: not on a dry-run context");
    if (!ctx || ng < 1 || nv <= 0 || no <= 0 || !T1 || !T2 || !f || !eri || !g || !omega_host ||
        beta == 0.0)
        return kv_fail(ctx, KVFT_EINVAL, "ft_cc_energy: bad argument");
    cudaSetDevice(ctx->device);
    void *res = nullptr;
    KV_TRY(kv_scratch(ctx, "energy_result", sizeof(double), &res));
    KV_TRY(kv_energy(ctx, ng, nv, no, T1, T2, f, eri, g, beta, qterm, (double *)res));
    KV_CHECK(ctx, cudaMemcpyAsync(omega_host, res, sizeof(double), cudaMemcpyDeviceToHost,
                                  ctx->stream));
    KV_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return KVFT_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free energy reduction.
//
// Some callers cannot let a library call cudaMalloc: a host process that has
// handed (nearly) all device memory to its own pool, a serving loop whose
// latency budget has no room for the device-wide synchronisation cudaMalloc
// and cudaFree can imply, or a plugin host that forbids allocations outside
// its allocator.  kvft_ft_cc_energy_noalloc computes the same grand
// potential as kvft_ft_cc_energy without any allocation: the per-tile
// partial sums live in the file-scope array below, which every GPU that loads
// libkvft holds (256 KiB) until the process exits.  Its device address is
// looked up with cudaGetSymbolAddress once per device, on that device's first
// call, so that first call should come before any stream capture.  All calls
// on a device share the array; every call overwrites the partial sums it
// reads and clears the arrival count before its launch, so nothing is left to
// the caller between calls.  Two calls that overlap on the GPU (different
// streams, no ordering) race on both.
// ---------------------------------------------------------------------------
#include <mutex>

namespace {
constexpr int NOALLOC_MAX_TILES = 32767;   // 32 x 32 tiles of (a,b) x (i,j)
// partial sums of the blocks, and the arrival count in the last word
__device__ __align__(256) double g_energy_scratch[NOALLOC_MAX_TILES + 1];
std::mutex g_energy_scratch_mu;
double *g_energy_scratch_ptr[64] = {};     // device address of the array, per device
}  // namespace

extern "C" int kvft_ft_cc_energy_noalloc(void *stream, int ng, int nv, int no,
                                         const double *T1, const double *T2,
                                         const double *f, const double *eri,
                                         const double *g, double beta, int qterm,
                                         double *omega_dev) {
    if (ng < 1 || nv <= 0 || no <= 0 || !T1 || !T2 || !f || !eri || !g || !omega_dev ||
        beta == 0.0)
        return KVFT_EINVAL;
    const long long V2 = (long long)nv * nv, O2 = (long long)no * no;
    const long long gx = (O2 + TILE - 1) / TILE, gy = (V2 + TILE - 1) / TILE;
    if (gx * gy > NOALLOC_MAX_TILES) return KVFT_EINVAL;   // beyond the static scratch
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return KVFT_EDEVICE;
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_energy_scratch_mu);
        if (!g_energy_scratch_ptr[dev]) {
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_energy_scratch) != cudaSuccess || !p)
                return KVFT_EDEVICE;
            g_energy_scratch_ptr[dev] = (double *)p;
        }
        scratch = g_energy_scratch_ptr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return KVFT_EDEVICE;
    // the launch's own status (cudaLaunchKernel reports that launch), so that
    // an earlier unrelated error left on the thread is not returned as this
    // call's
    int sh = 0, igx = (int)gx, tiles = (int)(gx * gy);
    unsigned *count = (unsigned *)(scratch + NOALLOC_MAX_TILES);
    double inv_beta = 1.0 / beta;
    void *a2[] = {&ng, &nv, &no, (void *)&T1, (void *)&T2, (void *)&f, (void *)&eri, (void *)&g,
                  &qterm, &sh, &igx, &tiles, &scratch, &count, &inv_beta, &omega_dev};
    // the count starts from zero whatever an overlapping (racing) call left
    if (cudaMemsetAsync(count, 0, sizeof(unsigned), st) != cudaSuccess ||
        cudaLaunchKernel((const void *)energy2_kernel, dim3((unsigned)energy_grid(sms, tiles)),
                         dim3(EN_T), a2, 0, st) != cudaSuccess)
        return KVFT_EDEVICE;
    return KVFT_OK;
}

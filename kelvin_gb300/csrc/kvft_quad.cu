// Exp-weighted cumulative tau integrals (kelvin/quadrature.py:292-317,
// 348-369) and the fused "integrate + damp + norms" pass of the solver.
//
// For every amplitude element p with denominator d:
//     T_y = sum_x G[y,x] w(y,x) tbar_x,
//     w(y,x) = exp((ti[x]-ti[y]) d) for x < y (all x if `full`), else 1.
// GB300 issues about two FP64 FMAs per clock per SM, so exp evaluations are
// the cost to cut, not HBM bytes:
//   * w(y,x) is built as a running product of step factors
//     r_k = exp((ti[k]-ti[k+1]) d), one exp per grid step -- and a single exp
//     when the grid is uniform (Kelvin's default 'lin' rule);
//   * when G has the structure of Kelvin's Simpson/midpoint/left rules
//     (G[y,x] == G[y-s,x] for x < y-s, zero above the diagonal), rows are
//     chained: T_y = w(y,y-s) (T_{y-s} - G[y-s,y-s] tbar_{y-s})
//                    + sum_{x=y-s}^{y} G[y,x] w(y,x) tbar_x,
//     which is O(ng) per element instead of O(ng^2).
// The product of <= ng factors, each within 1.25 units in the last place,
// differs from a direct exp by at most ~2 ng ulp (relative), far inside the
// 1e-10 parity tolerance.
#include "kvft_internal.h"

#include <cmath>

namespace {

constexpr int QT = 128;      // threads per block
constexpr int MAXNG = 64;

struct QuadParams {
    int ng;
    long long P;             // elements per tau slice
    int rank;                // 1: [nv][no], 2: [nv][nv][no][no]
    int nv, no;
    int step;                // recurrence step (0: general path)
    int uniform;             // all ti[k+1]-ti[k] equal
    int full;
    int same;                // first chained row from which gd, g1 and cs are constant
    int symmetric;           // ti[x] + ti[ng-1-x] the same for every x
    int mirror;              // ti[x] - tc and ti[ng-1-x] - tc differ in sign alone
    double alpha;            // damping (fused update only)
    int spin_half;           // fused update over the spin-conserving elements only (0: all)
};

// d of element p = l NR + r (rank 1: l = a, r = i; rank 2: l = a nv + b, r = i
// no + j)
__device__ __forceinline__ double denom(const QuadParams &q, long long p, int l, int r,
                                        const double *D, const double *ev, const double *eo) {
    if (D) return D[p];
    if (q.rank == 1) return ev[l] - eo[r];
    const int a = l / q.nv, i = r / q.no;
    return ev[a] + ev[l - a * q.nv] - eo[i] - eo[r - i * q.no];
}

// e^x by table lookup (P. T. P. Tang, ACM TOMS 15, 144 (1989)): x = n ln2/64 +
// r, |r| <= ln2/128, e^x = 2^(n / 64) (1 + (e^r - 1)) with the 64 values of
// 2^(j/64) in shared memory and a Taylor polynomial -- the FP64 pipe is what
// these kernels wait for.
//   exp_tab   fifth order: ten FP64 operations, where the library function
//             takes about 17, and three of them more for e^-x (exp_tab2), where
//             a reciprocal takes ten; 1.25 units in the last place.
//   exp_acc   sixth order, and the table's rounding added: twelve operations,
//             0.51 units, as the library function.  For the one step factor of
//             a uniform grid, which the rows raise to powers of up to ng: the
//             integral of 66 spin orbitals and 16 points has an error of
//             7.8e-16 with it (8.0e-16 with the library function), 1.0e-15
//             with exp_tab, for 2.71 -> 2.78 ms.  Factors of their own
//             for every step or node do not add up so (17 logarithmic points
//             4.4e-16 with exp_tab, 5.0e-16 with the library function; 16
//             Gauss-Legendre points 3.5e-16, 3.9e-16), and there exp_acc would
//             cost 2 to 7 %.
// |x| >= 700 and NaN go to the library function.
constexpr int ETAB = 64;
// 2^(j/64): rounded to FP64, and the difference from it
__device__ const double EXP2_TAB[ETAB][2] = {
    {1.0, 0.0}, {1.0108892860517005, -1.523477860e-17},
    {1.0218971486541166, 5.109225029e-17}, {1.0330248790212284, 7.600838874e-18},
    {1.0442737824274138, 8.551889706e-17}, {1.0556451783605572, 1.759325739e-18},
    {1.0671404006768237, -7.899853967e-17}, {1.0787607977571199, -6.656660436e-17},
    {1.0905077326652577, -3.046782080e-17}, {1.102382583307841, 5.266036872e-17},
    {1.1143867425958924, 1.041027846e-16}, {1.1265216186082418, 5.165856759e-17},
    {1.1387886347566916, 8.912812676e-17}, {1.1511892299529827, 3.250710219e-17},
    {1.1637248587775775, 3.829204837e-17}, {1.1763969916502812, 5.554203254e-17},
    {1.189207115002721, 3.982015231e-17}, {1.202156731452703, 6.644981499e-17},
    {1.215247359980469, -7.712630693e-17}, {1.22848053610687, -1.898781631e-17},
    {1.241857812073484, 4.658027592e-17}, {1.255380757024691, -6.711389821e-18},
    {1.2690509571917332, 2.667932131e-18}, {1.2828700160787783, 1.713594918e-17},
    {1.2968395546510096, 2.538250279e-17}, {1.3109612115247644, -7.181536136e-17},
    {1.3252366431597413, -2.858731210e-17}, {1.339667524053303, 8.927282595e-17},
    {1.3542555469368927, 7.700948380e-17}, {1.3690024229745905, 9.593797919e-17},
    {1.383909881963832, -6.770511659e-17}, {1.3989796725383112, -9.614213209e-17},
    {1.4142135623730951, -9.667293313e-17}, {1.42961333839197, -1.203164249e-17},
    {1.4451808069770467, -3.023758135e-17}, {1.460917794180647, -5.600377186e-17},
    {1.4768261459394993, -3.483994557e-17}, {1.4929077282912648, 1.419292015e-17},
    {1.5091644275934228, -1.016455328e-16}, {1.5255981507445384, -1.102494171e-16},
    {1.5422108254079407, 7.949834810e-17}, {1.559004400237837, 3.781207053e-17},
    {1.5759808451078865, -1.013691647e-17}, {1.593142151342267, -1.009440654e-16},
    {1.6104903319492543, 2.470719257e-17}, {1.6280274218573478, -6.712955085e-17},
    {1.645755478153965, -1.012567991e-16}, {1.6636765803267364, 5.890992697e-17},
    {1.681792830507429, 8.199010021e-17}, {1.7001063537185235, -8.023719370e-18},
    {1.718619298122478, -1.851380418e-17}, {1.7373338352737062, 3.164389299e-17},
    {1.7562521603732995, 2.960140695e-17}, {1.7753764925265212, 6.429731797e-17},
    {1.7947090750031072, 1.822745843e-17}, {1.8142521755003989, -9.969531539e-17},
    {1.8340080864093424, 3.283107224e-17}, {1.8539791250833855, 9.761887491e-17},
    {1.8741676341103, -6.122763413e-17}, {1.8945759815869656, 3.403403535e-17},
    {1.9152065613971474, -1.061994606e-16}, {1.9360617934922943, 1.033238596e-16},
    {1.9571441241754002, 8.960767791e-17}, {1.978456026387951, 4.038875311e-17},
};
// shared-memory copy: the rounded values, then the rests
__device__ __forceinline__ void exp_table(double *T) {       // caller synchronises
    for (int j = threadIdx.x; j < 2 * ETAB; j += blockDim.x) T[j] = EXP2_TAB[j % ETAB][j / ETAB];
}
template <bool ACC = false>
__device__ __forceinline__ double exp_scaled(const double *T, int n, double p) {
    const double t = T[n & (ETAB - 1)];
    const double y = ACC ? t + fma(t, p, T[ETAB + (n & (ETAB - 1))]) : fma(t, p, t);
    return __hiloint2double(__double2hiint(y) + (n >> 6) * (1 << 20), __double2loint(y));
}
__device__ __forceinline__ bool exp_reduce(double x, int &n, double &r) {
    if ((__double2hiint(x) & 0x7FFFFFFF) >= 0x4085E000) return false;       // |x| >= 700, NaN
    const double t = fma(x, 92.332482616893656877, 6755399441055744.0);     // 64 / ln 2
    n = __double2loint(t);
    const double nd = t - 6755399441055744.0;
    r = fma(nd, -0.010830424696223417, x);               // ln2/64, 36 bits, and the rest
    r = fma(nd, -2.5728046223276688e-14, r);
    return true;
}
__device__ __forceinline__ double exp_tab(double x, const double *T) {
    int n;
    double r;
    if (!exp_reduce(x, n, r)) return exp(x);
    const double q = fma(fma(fma(r, 1.0 / 120.0, 1.0 / 24.0), r, 1.0 / 6.0), r, 0.5);
    return exp_scaled(T, n, fma(q * r, r, r));
}
__device__ __forceinline__ double exp_acc(double x, const double *T) {
    int n;
    double r;
    if (!exp_reduce(x, n, r)) return exp(x);
    const double q = fma(fma(fma(fma(r, 1.0 / 720.0, 1.0 / 120.0), r, 1.0 / 24.0), r, 1.0 / 6.0), r, 0.5);
    return exp_scaled<true>(T, n, fma(q * r, r, r));
}
// e^x and e^-x: the polynomial's even and odd parts
__device__ __forceinline__ void exp_tab2(double x, const double *T, double &ep, double &em) {
    int n;
    double r;
    if (!exp_reduce(x, n, r)) {
        ep = exp(x);
        em = exp(-x);
        return;
    }
    const double r2 = r * r;
    const double ev = r2 * fma(r2, 1.0 / 24.0, 0.5);
    const double od = fma(r * r2, fma(r2, 1.0 / 120.0, 1.0 / 6.0), r);
    ep = exp_scaled(T, n, ev + od);
    em = exp_scaled(T, -n, ev - od);
}

// f(p, l, r) for this thread's elements: every one, or with spin blocks the
// spin-conserving ones (the others are zero and stay zero)
template <class F>
__device__ __forceinline__ void quad_visit(const QuadParams &q, F f) {
    if (q.spin_half > 0) {
        const KvSpinUnits su(q.spin_half);
        const long long n2 = (long long)q.no * q.no, units = su.count();
        for (long long u = blockIdx.x * (long long)(QT / 32) + threadIdx.x / 32; u < units;
             u += (long long)gridDim.x * (QT / 32)) {
            int l, r;
            if (su.at(u, threadIdx.x % 32, l, r)) f(l * n2 + r, l, r);
        }
        return;
    }
    const int NR = q.rank == 2 ? q.no * q.no : q.no;
    for (long long p = blockIdx.x * (long long)QT + threadIdx.x; p < q.P;
         p += (long long)gridDim.x * QT) {
        const int l = (int)(p / NR);
        f(p, l, (int)(p - (long long)l * NR));
    }
}

// Shared memory: ti[ng], G[ng*ng], the chained-row coefficients cs[ng]
// (G[y,y-s] - G[y-s,y-s]), g1[ng] (G[y,y-1]) and gd[ng] (G[y,y]), then the
// per-thread columns r[ng][QT] (non-uniform grids) and tb[ng][QT] (general
// path).
// |x| as a float (mantissa truncated), from the FP64 bit pattern with
// integer operations: GB300's FP64 pipe, not its integer or FP32 pipes, is
// the scarce unit of this kernel.  Below 2^-126 the result is 0; above the
// float range it is infinity (NaN stays NaN).
__device__ __forceinline__ float abs_to_f32(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7FF) - 1023 + 127;
    if (e <= 0) return 0.f;
    if (e >= 255) {
        const bool nan = (hi & 0x7FF00000u) == 0x7FF00000u && (((hi & 0xFFFFFu) | lo) != 0);
        return __int_as_float(nan ? 0x7FC00000 : 0x7F800000);
    }
    return __int_as_float((e << 23) | (int)((hi & 0xFFFFFu) << 3) | (int)(lo >> 29));
}

// MODE 0: out = T.  MODE 1 (fused solver update): Told = alpha Told + (1-alpha) T,
// with block partial sums of |T - Told|^2 and |Told_new|^2.  Those two norms
// only steer convergence: each element's sum over tau points is taken in
// FP32 (relative error ~1e-7) and added to FP64 block sums.  UNI: uniform
// grid, one step factor for every step.
template <int MODE, bool UNI>
__global__ void __launch_bounds__(QT)
quad_kernel(QuadParams q, const double *__restrict__ tbar, const double *__restrict__ ti_g,
            const double *__restrict__ G_g, const double *__restrict__ D,
            const double *__restrict__ ev, const double *__restrict__ eo,
            double *out, double *__restrict__ partial) {
    if (!kv_depend()) return;
    extern __shared__ double sm[];
    const int ng = q.ng;
    double *ti = sm;
    double *G = ti + ng;
    double *cs = G + ng * ng, *g1 = cs + ng, *gd = g1 + ng;
    double *et = gd + ng;                                  // 2^(j/64)
    double *rk = et + 2 * ETAB;                              // [ng][QT]
    double *tb = rk + (q.uniform ? 0 : ng * QT);           // [ng][QT]
    for (int k = threadIdx.x; k < ng; k += QT) ti[k] = ti_g[k];
    for (int k = threadIdx.x; k < ng * ng; k += QT) G[k] = G_g[k];
    for (int y = threadIdx.x; y < ng; y += QT) {
        const int sy = q.step > 0 ? q.step : 1;
        cs[y] = (y >= sy) ? G_g[y * ng + y - sy] - G_g[(y - sy) * ng + y - sy] : 0.0;
        g1[y] = (y >= 1) ? G_g[y * ng + y - 1] : 0.0;
        gd[y] = G_g[y * ng + y];
    }
    exp_table(et);
    __syncthreads();
    const double oma = 1.0 - q.alpha;

    double s_diff = 0.0, s_norm = 0.0;
    const int t = threadIdx.x;
    auto element = [&](long long p, int l, int r) {
        const double d = denom(q, p, l, r, D, ev, eo);
        // step factors r_k = exp((ti[k]-ti[k+1]) d)
        double r0 = 1.0;
        if (UNI) {
            r0 = (ng > 1) ? exp_acc((ti[0] - ti[1]) * d, et) : 1.0;
        } else {
            for (int k = 0; k + 1 < ng; k++) rk[k * QT + t] = exp_tab((ti[k] - ti[k + 1]) * d, et);
        }
        const double r02 = r0 * r0;
        float f_diff = 0.f, f_norm = 0.f;
#define RK(k) (UNI ? r0 : rk[(k) * QT + t])
        if (q.step > 0) {
            // chained rows; keep the last `step` outputs and inputs in registers
            double Tm1 = 0.0, Tm2 = 0.0, tbm1 = 0.0, tbm2 = 0.0;
            const double *tp = tbar + p;
            double *op = out + p;
            auto emit = [&](double *o, double told, double Ty, double tby) {
                if (MODE == 0) {
                    *o = Ty;
                } else {
                    // damped update Told + (1 - alpha)(T - Told) and the norms
                    const double df = Ty - told;
                    const double nt = fma(oma, df, told);
                    const float fd = abs_to_f32(df), fn = abs_to_f32(nt);
                    f_diff = fmaf(fd, fd, f_diff);
                    f_norm = fmaf(fn, fn, f_norm);
                    *o = nt;
                }
                Tm2 = Tm1; Tm1 = Ty;
                tbm2 = tbm1; tbm1 = tby;
            };
            const int same = UNI ? q.same : ng;
            for (int y = 0; y < same; y++, tp += q.P, op += q.P) {
                const double tby = *tp;
                double Ty;
                if (y < q.step) {
                    // direct: x in [0, y]
                    Ty = G[y * ng + y] * tby;
                    double w = 1.0;
                    for (int x = y - 1; x >= 0; x--) {
                        w *= RK(x);
                        const double v = (x == y - 1) ? tbm1 : tbm2;
                        Ty = fma(G[y * ng + x] * w, v, Ty);
                    }
                } else if (q.step == 1) {
                    // T_y = w (T_{y-1} - G[y-1,y-1] tb_{y-1}) + G[y,y-1] w tb_{y-1}
                    //       + G[y,y] tb_y
                    Ty = fma(gd[y], tby, RK(y - 1) * fma(cs[y], tbm1, Tm1));
                } else {  // step 2: r_{y-1} (r_{y-2} (T + cs tb)_{y-2} + g1 tb_{y-1}) + gd tb_y
                    const double z = fma(RK(y - 2), fma(cs[y], tbm2, Tm2), g1[y] * tbm1);
                    Ty = fma(RK(y - 1), z, gd[y] * tby);
                }
                emit(op, MODE == 1 ? *op : 0.0, Ty, tby);
            }
            if (UNI && same < ng) {
                // rows that share their coefficients (Simpson's rule on a
                // uniform grid): the products with the step factors are formed
                // once, four FP64 operations per row instead of five; the
                // loads of four rows are issued together
                const double cd = gd[same], c1 = g1[same] * r0, c2 = cs[same] * r02;
                for (int y = same; y < ng; y += 4) {
                    double tv[4], ov[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        tv[k] = y + k < ng ? tp[k * q.P] : 0.0;
                        ov[k] = MODE == 1 && y + k < ng ? op[k * q.P] : 0.0;
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (y + k >= ng) break;
                        const double Ty = fma(cd, tv[k], fma(c1, tbm1, fma(c2, tbm2, r02 * Tm2)));
                        emit(op + k * q.P, ov[k], Ty, tv[k]);
                    }
                    tp += 4 * q.P;
                    op += 4 * q.P;
                }
            }
        } else {
            for (int x = 0; x < ng; x++) tb[x * QT + t] = tbar[(long long)x * q.P + p];
            for (int y = 0; y < ng; y++) {
                double Ty = 0.0;
                // x <= y: running product downward from x = y
                double w = 1.0;
                for (int x = y; x >= 0; x--) {
                    if (x < y) w *= RK(x);
                    const double gyx = G[y * ng + x];
                    if (gyx != 0.0) Ty = fma(gyx * w, tb[x * QT + t], Ty);
                }
                // x > y: factor 1 (the reference's rule; dense grids with
                // the exponential for every pair run quad_dense_kernel)
                for (int x = y + 1; x < ng; x++) {
                    const double gyx = G[y * ng + x];
                    if (gyx != 0.0) Ty = fma(gyx, tb[x * QT + t], Ty);
                }
                if (MODE == 0) {
                    out[(long long)y * q.P + p] = Ty;
                } else {
                    double *o = out + (long long)y * q.P + p;
                    const double told = *o;
                    const double df = Ty - told;
                    const double nt = fma(oma, df, told);
                    const float fd = abs_to_f32(df), fn = abs_to_f32(nt);
                    f_diff = fmaf(fd, fd, f_diff);
                    f_norm = fmaf(fn, fn, f_norm);
                    *o = nt;
                }
            }
        }
#undef RK
        if (MODE == 1) {
            s_diff += (double)f_diff;
            s_norm += (double)f_norm;
        }
    };
    quad_visit(q, element);
    if (MODE == 1) {
        // block reduction of the two sums (fixed order: deterministic)
        __shared__ double red[2][QT];
        red[0][t] = s_diff;
        red[1][t] = s_norm;
        __syncthreads();
        for (int s = QT / 2; s > 0; s >>= 1) {
            if (t < s) {
                red[0][t] += red[0][t + s];
                red[1][t] += red[1][t + s];
            }
            __syncthreads();
        }
        if (t == 0) {
            partial[2 * blockIdx.x] = red[0][0];
            partial[2 * blockIdx.x + 1] = red[1][0];
        }
    }
}

// ---------------------------------------------------------------------------
// Dense G (Gauss-Legendre grids; the backward Lambda integral):
//     T_y = sum_x G[y,x] exp((ti[x]-ti[y]) d) tbar_x   for every x.
// Factorised about the grid's centre tc, exp((ti[x]-ti[y]) d) = E_x / E_y with
// E_x = exp((ti[x]-tc) d), so T_y = (1/E_y) sum_x G[y,x] u_x, u_x = E_x tbar_x.
// GB300 has ~64x more FP32 than FP64 throughput, so:
//   * no exponentials per element: d = e_a + e_b - e_i - e_j, and E_x, 1/E_y
//     are products of a pair table of the virtual indices and one of the
//     occupied indices (quad_tables_kernel, exps of the orbital energies);
//   * the ng^2 sum runs in compensated FP32: u (scaled by a power of two to
//     order one) and G split into FP32 high and low parts; the high products
//     are summed with error-free two-sums and their rounding errors, the
//     cross terms and the sum's errors go to a second FP32 accumulator
//     (relative error ~1e-14 of sum |G u|, far inside the parity bounds).
// An element whose factors leave the safe range (non-finite u, or a bound on
// |T_y| near the FP64 limit), and every element when D is given explicitly,
// takes the FP64 path: table exponentials, E_{ng-1-x} = 1/E_x on a grid
// symmetric about tc, and FP64 FMAs.
// ---------------------------------------------------------------------------
struct DenseTabs {
    const double *v, *vi, *o, *oi;   // [ng][NL] / [ng][NR]: E and 1/E factors
    long long NL, NR;                // p = l NR + r
};

// tables: v[x][l] = exp((ti[x]-tc)(e_a (+ e_b))), vi = its inverse,
// o[x][r] = exp(-(ti[x]-tc)(e_i (+ e_j))), oi = its inverse; l = a (rank 1)
// or a nv + b (rank 2), r = i or i no + j
__global__ void quad_tables_kernel(int ng, int rank, int nv, int no, double tc,
                                   const double *__restrict__ ti, const double *__restrict__ ev,
                                   const double *__restrict__ eo, long long NL, long long NR,
                                   double *__restrict__ tab) {
    if (!kv_depend()) return;
    const long long per = NL + NR;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < ng * per;
         k += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(k / per);
        const long long c = k - x * per;
        const double dt = ti[x] - tc;
        double e;
        if (c < NL)
            e = (rank == 2) ? ev[c / nv] + ev[c % nv] : ev[c];
        else
            e = (rank == 2) ? -(eo[(c - NL) / no] + eo[(c - NL) % no]) : -eo[c - NL];
        const double f = exp(dt * e), fi = exp(-dt * e);
        if (c < NL) {
            tab[x * NL + c] = f;
            tab[ng * NL + x * NL + c] = fi;
        } else {
            tab[2 * ng * NL + x * NR + (c - NL)] = f;
            tab[2 * ng * NL + ng * NR + x * NR + (c - NL)] = fi;
        }
    }
}

// s + e == a + b exactly (FP32 round to nearest)
__device__ __forceinline__ void two_sum_f(float a, float b, float &s, float &e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Biased exponent field of x (0: zero or subnormal, 0x7FF: inf or NaN).
__device__ __forceinline__ int dexp(double x) {
    return (__double2hiint(x) >> 20) & 0x7FF;
}

// x 2^-k as an FP32 pair hi + lo, from the bit pattern with integer
// operations (hi: the sign, exponent and top 23 mantissa bits; lo: the
// remaining 29 bits, rounded to 24), |x 2^-k - hi - lo| <= 2^-47 |x 2^-k|.
// For |x 2^-k| < 2: parts below 2^-126 are dropped (absolute error below
// 2^-126 of the scale 1).
__device__ __forceinline__ float2 dsplit_scaled(double x, int k) {
    const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
    const int e = (int)((hw >> 20) & 0x7FF) - 1023 - k;      // unbiased exponent of x 2^-k
    if (((hw >> 20) & 0x7FF) == 0 || e < -126) return make_float2(0.f, 0.f);
    const unsigned sg = hw & 0x80000000u;
    const float hi = __uint_as_float(sg | ((unsigned)(e + 127) << 23) | ((hw & 0xFFFFFu) << 3) |
                                     (lw >> 29));
    const unsigned rem = lw & 0x1FFFFFFFu;                   // 29 low mantissa bits
    float lo = 0.f;
    if (rem != 0 && e - 52 >= -126)
        lo = __uint_as_float(sg | __float_as_uint(__uint2float_rn(rem) *
                                                  __uint_as_float((unsigned)(e - 52 + 127) << 23)));
    return make_float2(hi, lo);
}

// (double) f 2^k for a finite float f, by integer operations on the bit
// pattern: 0 stays 0, a result below 2^-1022 is 0 (an absolute error far
// below anything the integral resolves), one above the FP64 range infinite.
__device__ __forceinline__ double f32_to_f64_scaled(float f, int k) {
    const unsigned u = __float_as_uint(f);
    const int E = (int)((u >> 23) & 0xFF);
    const int eb = E - 127 + 1023 + k;                       // biased FP64 exponent
    if (E == 0 || eb <= 0) return 0.0;                       // zero, float subnormals, underflow
    const unsigned sg = u & 0x80000000u;
    if (eb >= 0x7FF) return __hiloint2double((int)(sg | 0x7FF00000u), 0);
    const unsigned hw = sg | ((unsigned)eb << 20) | ((u >> 3) & 0xFFFFFu);
    return __hiloint2double((int)hw, (int)(u << 29));
}

template <int MODE>
__global__ void __launch_bounds__(QT)
quad_dense_kernel(QuadParams q, DenseTabs tb_, const double *__restrict__ tbar,
                  const double *__restrict__ ti_g, const double *__restrict__ G_g,
                  const double *__restrict__ D, const double *__restrict__ ev,
                  const double *__restrict__ eo, double *out, double *__restrict__ partial) {
    if (!kv_depend()) return;
    extern __shared__ double sm[];
    const int ng = q.ng;
    double *ti = sm;
    double *G = ti + ng;                                   // [ng][ng] FP64
    float *Gh = reinterpret_cast<float *>(G + ng * ng);    // [ng][ng] FP32 high part
    float *Gl = Gh + ng * ng;                              //          low part
    double *et = G + ng * ng + ng * ng;                    // 2^(j/64)
    double *c0 = et + 2 * ETAB;                              // [ng][QT]: u (FP64 or FP32 pair)
    double *c1 = c0 + ng * QT;                             // [ng][QT]: E (FP64 path)
    for (int k = threadIdx.x; k < ng; k += QT) ti[k] = ti_g[k];
    for (int k = threadIdx.x; k < ng * ng; k += QT) {
        const double g = G_g[k];
        G[k] = g;
        const float h = (float)g;
        Gh[k] = h;
        Gl[k] = (float)(g - (double)h);
    }
    exp_table(et);
    __syncthreads();
    const double oma = 1.0 - q.alpha;
    const double tc = 0.5 * (ti[0] + ti[ng - 1]);
    double s_diff = 0.0, s_norm = 0.0;
    const int t = threadIdx.x;
    float2 *uf = reinterpret_cast<float2 *>(c0);

    auto emit = [&](long long p, int y, double Ty, float &f_diff, float &f_norm) {
        if (MODE == 0) {
            out[(long long)y * q.P + p] = Ty;
        } else {
            double *o = out + (long long)y * q.P + p;
            const double told = *o;
            const double df = Ty - told;
            const double nt = fma(oma, df, told);
            const float fd = abs_to_f32(df), fn = abs_to_f32(nt);
            f_diff = fmaf(fd, fd, f_diff);
            f_norm = fmaf(fn, fn, f_norm);
            *o = nt;
        }
    };

    auto element = [&](long long p, int l, int r) {
        float f_diff = 0.f, f_norm = 0.f;
        bool table = tb_.v != nullptr;
        if (table) {
            // u_x = E_x tbar_x and the largest binary exponent among them.
            // Range tests and the scale are integer operations on exponent
            // fields: the FP64 pipe, GB300's scarce unit here, only takes the
            // products
            int umax_e = 0, eimax_e = 0;
            for (int x = 0; x < ng; x++) {
                const double E = __ldg(tb_.v + x * tb_.NL + l) * __ldg(tb_.o + x * tb_.NR + r);
                const double u = E * tbar[(long long)x * q.P + p];
                c0[x * QT + t] = u;
                umax_e = max(umax_e, dexp(u));        // inf / NaN: 0x7FF, refused below
                if (q.mirror) {                       // 1 / E_{ng-1-x} = E_x
                    c1[(ng - 1 - x) * QT + t] = E;
                    eimax_e = max(eimax_e, dexp(E));
                }
            }
            for (int y = 0; y < ng && !q.mirror; y++) {
                const double Ei = __ldg(tb_.vi + y * tb_.NL + l) * __ldg(tb_.oi + y * tb_.NR + r);
                c1[y * QT + t] = Ei;
                eimax_e = max(eimax_e, dexp(Ei));
            }
            // |u|, 1/E < 2^996 (< 1e300), and |T_y| <= ng max|G| max|u| max(1/E)
            // < 2^(umax_e + eimax_e - 2044 + 8) kept below 2^956 (~1e288):
            // well inside FP64
            if (umax_e > 1023 + 995 || eimax_e > 1023 + 995 ||
                umax_e + eimax_e - 2044 + 8 > 956)
                table = false;
            if (table) {
                if (umax_e == 0) {          // all u zero (or below 2^-1022)
                    for (int y = 0; y < ng; y++) emit(p, y, 0.0, f_diff, f_norm);
                } else {
                    const int k = umax_e - 1023;     // |u 2^-k| < 2
                    for (int x = 0; x < ng; x++) uf[x * QT + t] = dsplit_scaled(c0[x * QT + t], k);
                    for (int y = 0; y < ng; y++) {
                        float s = 0.f, c = 0.f;
                        const float *gh = Gh + y * ng, *gl = Gl + y * ng;
                        for (int x = 0; x < ng; x++) {
                            const float2 u = uf[x * QT + t];
                            const float pr = gh[x] * u.x;
                            const float pe = fmaf(gh[x], u.x, -pr);      // exact
                            float s2, e2;
                            two_sum_f(s, pr, s2, e2);
                            s = s2;
                            c += e2 + pe;
                            c = fmaf(gh[x], u.y, c);
                            c = fmaf(gl[x], u.x, c);
                        }
                        const double acc = f32_to_f64_scaled(s, k) + f32_to_f64_scaled(c, k);
                        emit(p, y, acc * c1[y * QT + t], f_diff, f_norm);
                    }
                }
            }
        }
        if (!table) {
            // FP64 path
            const double d = denom(q, p, l, r, D, ev, eo);
            const int nx = q.symmetric ? (ng + 1) / 2 : ng;
            for (int x = 0; x < nx; x++) {
                double E, Ei;
                exp_tab2((ti[x] - tc) * d, et, E, Ei);
                c1[x * QT + t] = q.symmetric ? E : Ei;
                c0[x * QT + t] = E * tbar[(long long)x * q.P + p];
                const int xm = ng - 1 - x;
                if (q.symmetric && xm != x) {
                    c1[xm * QT + t] = Ei;
                    c0[xm * QT + t] = Ei * tbar[(long long)xm * q.P + p];
                }
            }
            for (int y = 0; y < ng; y++) {
                double acc = 0.0;
                for (int x = 0; x < ng; x++) acc = fma(G[y * ng + x], c0[x * QT + t], acc);
                const double Ty = acc * c1[(q.symmetric ? ng - 1 - y : y) * QT + t];
                emit(p, y, Ty, f_diff, f_norm);
            }
        }
        if (MODE == 1) {
            s_diff += (double)f_diff;
            s_norm += (double)f_norm;
        }
    };
    quad_visit(q, element);
    if (MODE == 1) {
        __shared__ double red[2][QT];
        red[0][t] = s_diff;
        red[1][t] = s_norm;
        __syncthreads();
        for (int st = QT / 2; st > 0; st >>= 1) {
            if (t < st) {
                red[0][t] += red[0][t + st];
                red[1][t] += red[1][t + st];
            }
            __syncthreads();
        }
        if (t == 0) {
            partial[2 * blockIdx.x] = red[0][0];
            partial[2 * blockIdx.x + 1] = red[1][0];
        }
    }
}

// one grid point: out = sum_x G[ig,x] w(ig,x) tbar_x (quadrature.py:348-369)
__global__ void quad_single_kernel(QuadParams q, int ig, const double *__restrict__ tbar,
                                   const double *__restrict__ ti,
                                   const double *__restrict__ G,
                                   const double *__restrict__ D,
                                   const double *__restrict__ ev,
                                   const double *__restrict__ eo,
                                   double *__restrict__ out) {
    if (!kv_depend()) return;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < q.P;
         p += (long long)gridDim.x * blockDim.x) {
        const int NR = q.rank == 2 ? q.no * q.no : q.no;
        const int l = (int)(p / NR);
        const double d = denom(q, p, l, (int)(p - (long long)l * NR), D, ev, eo);
        double acc = 0.0;
        for (int x = 0; x < q.ng; x++) {
            const double g = G[ig * q.ng + x];
            if (g == 0.0) continue;
            const double dt = (x < ig) ? (ti[x] - ti[ig]) : 0.0;
            acc = fma(g * exp(dt * d), tbar[(long long)x * q.P + p], acc);
        }
        out[p] = acc;
    }
}

__global__ void reduce_pairs_kernel(const double *__restrict__ partial, int n,
                                    double *__restrict__ res) {
    if (!kv_depend()) return;
    __shared__ double red[2][256];
    double a = 0.0, b = 0.0;
    for (int k = threadIdx.x; k < n; k += 256) {
        a += partial[2 * k];
        b += partial[2 * k + 1];
    }
    red[0][threadIdx.x] = a;
    red[1][threadIdx.x] = b;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        res[0] = red[0][0];
        res[1] = red[1][0];
    }
}

// Host-side analysis of the grid: recurrence step, uniform spacing, and (step
// 2) the first row from which the chained rows' coefficients are the same.
void analyse_grid(int ng, const double *ti, const double *G, int full, int *step,
                  int *uniform, int *same) {
    *same = ng;
    *uniform = 1;
    for (int k = 1; k + 1 < ng; k++) {
        double d0 = ti[1] - ti[0], dk = ti[k + 1] - ti[k];
        if (std::fabs(dk - d0) > 1e-14 * std::max(std::fabs(d0), 1e-300)) *uniform = 0;
    }
    *step = 0;
    if (full) return;
    for (int y = 0; y < ng; y++)
        for (int x = y + 1; x < ng; x++)
            if (G[y * ng + x] != 0.0) return;   // not lower-triangular
    for (int s = 1; s <= 2; s++) {
        bool ok = true;
        for (int y = s; y < ng && ok; y++)
            for (int x = 0; x < y - s && ok; x++)
                if (G[y * ng + x] != G[(y - s) * ng + x]) ok = false;
        if (!ok) continue;
        *step = s;
        if (s == 2) {
            auto row = [&](int y, int k) {
                return k == 0 ? G[y * ng + y] : k == 1 ? G[y * ng + y - 1]
                              : G[y * ng + y - 2] - G[(y - 2) * ng + y - 2];
            };
            int y = ng - 1;
            while (y > 2 && row(y - 1, 0) == row(ng - 1, 0) && row(y - 1, 1) == row(ng - 1, 1) &&
                   row(y - 1, 2) == row(ng - 1, 2))
                y--;
            *same = std::max(2, y);
        }
        return;
    }
}

// ti, G, cs, g1, gd, the exponential's table; then the per-thread columns: step factors (general
// lower-triangular path on a non-uniform grid), inputs (general and dense
// paths), and the dense path's scale factors
size_t quad_smem(int ng, int uniform, int step, int full) {
    return sizeof(double) * (4 * ng + ng * ng + 2 * ETAB + ((uniform || full) ? 0 : ng * QT) +
                             (step > 0 ? 0 : ng * QT) + (full ? ng * QT : 0));
}

// ti[x] + ti[ng-1-x] equal for every x (to rounding)
int grid_symmetric(int ng, const double *ti) {
    const double c = ti[0] + ti[ng - 1];
    const double tol = 1e-13 * std::max(std::fabs(ti[ng - 1] - ti[0]), 1e-300);
    for (int x = 0; x < ng; x++)
        if (std::fabs(ti[x] + ti[ng - 1 - x] - c) > tol) return 0;
    return 1;
}

// ti[x] - tc = -(ti[ng-1-x] - tc) to the bit, as the tables form them: then the
// entries for x are the inverse ones for ng-1-x to the bit, too.  (A grid off
// by a last place in its nodes would put that times beta |d| into the factors.)
int grid_mirrored(int ng, const double *ti) {
    const double tc = 0.5 * (ti[0] + ti[ng - 1]);
    for (int x = 0; x < ng; x++)
        if (ti[x] - tc != -(ti[ng - 1 - x] - tc)) return 0;
    return 1;
}

}  // namespace

namespace {

size_t dense_smem(int ng) {
    return sizeof(double) * ((size_t)ng + 2 * (size_t)ng * ng + 2 * ETAB + 2 * (size_t)ng * QT);
}

// The dense-G integral: pair tables of the orbital energies (when given),
// then quad_dense_kernel; mode 1 also damps and reduces the two norms.
int quad_dense_launch(kvft_ctx *ctx, int mode, QuadParams &q, const double *tbar,
                      const double *ti, const double *hti, const double *G, const double *D,
                      const double *ev, const double *eo, double *out, double *res) {
    const int ng = q.ng;
    DenseTabs tabs{nullptr, nullptr, nullptr, nullptr, 1, 1};
    if (!D && ev && eo) {
        const long long NL = q.rank == 2 ? (long long)q.nv * q.nv : q.nv;
        const long long NR = q.rank == 2 ? (long long)q.no * q.no : q.no;
        if (NL * NR == q.P) {
            void *tp = nullptr;
            KV_TRY(kv_scratch(ctx, "quad_tables", sizeof(double) * 2 * ng * (NL + NR), &tp));
            double *tab = (double *)tp;
            const double tc = 0.5 * (hti[0] + hti[ng - 1]);
            const long long work = ng * (NL + NR);
            const int gb = (int)std::max(1LL, std::min((work + 255) / 256, 4096LL));
            kv_launch(ctx, quad_tables_kernel, gb, 256, 0, ng, q.rank, q.nv, q.no, tc, ti, ev, eo,
                      NL, NR, tab);
            KV_TRY(kv_launch_check(ctx, "quad_tables"));
            tabs = DenseTabs{tab, tab + ng * NL, tab + 2 * ng * NL, tab + 2 * ng * NL + ng * NR,
                             NL, NR};
        }
    }
    const size_t smem = dense_smem(ng);
    KV_TRY(kv_smem_optin(ctx, mode == 0 ? quad_dense_kernel<0> : quad_dense_kernel<1>,
                         dense_smem(MAXNG)));
    int per_sm = 1;
    KV_CHECK(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                      &per_sm, mode == 0 ? (const void *)quad_dense_kernel<0>
                                         : (const void *)quad_dense_kernel<1>,
                      QT, smem));
    const long long blocks = (q.P + QT - 1) / QT;
    const int grid = (int)std::max(1LL, std::min(blocks, (long long)std::max(per_sm, 1) *
                                                             ctx->sm_count));
    KvProfScope prof(ctx, KV_CAT_QUAD, 8.0 * ng * (double)q.P * (mode == 0 ? 2 : 3) *
                                           kv_spin_frac(q.nv, q.no, q.spin_half));
    if (mode == 0) {
        kv_launch(ctx, quad_dense_kernel<0>, grid, QT, smem, q, tabs, tbar, ti, G, D, ev, eo, out,
                  nullptr);
        return kv_launch_check(ctx, "quad_dense_kernel");
    }
    void *part = nullptr;
    KV_TRY(kv_scratch(ctx, "quad_partial", sizeof(double) * 2 * grid, &part));
    kv_launch(ctx, quad_dense_kernel<1>, grid, QT, smem, q, tabs, tbar, ti, G, D, ev, eo, out,
              (double *)part);
    KV_TRY(kv_launch_check(ctx, "quad_dense_update_kernel"));
    kv_launch(ctx, reduce_pairs_kernel, 1, 256, 0, (const double *)part, grid, res);
    return kv_launch_check(ctx, "reduce_pairs");
}

}  // namespace

// Shared launcher.  ti/G are DEVICE pointers; hti/hG are host copies used for
// the grid analysis.  MODE 1 requires `partial` (2 doubles per block) and
// `res` (2 doubles) device buffers.
int kv_quad_launch(kvft_ctx *ctx, int mode, int ng, long long P, int rank, int nv,
                   int no, const double *tbar, const double *ti, const double *hti,
                   const double *G, const double *hG, const double *D,
                   const double *ev, const double *eo, int full, double alpha,
                   double *out, double *res, int spin_half) {
    if (ng < 1 || ng > MAXNG) return kv_fail(ctx, KVFT_EINVAL, "ng must be in [1, 64]");
    if (P == 0) return KVFT_OK;
    if (ctx->dry) {
        if (mode != 0 || D) return kv_fail(ctx, KVFT_EINVAL, "dry run: tau integral mode");
        KvDryOp op;
        op.kind = 2;
        op.ng = ng, op.P = P, op.rank = rank, op.full = full, op.nv = nv, op.no = no;
        op.src = tbar, op.dst = out, op.ti = ti, op.G = G, op.ev = ev, op.eo = eo;
        ctx->dry->push_back(op);
        return KVFT_OK;
    }
    QuadParams q;
    q.ng = ng;
    q.P = P;
    q.rank = rank;
    q.nv = nv;
    q.no = no;
    q.full = full;
    q.alpha = alpha;
    // spin blocks: only the spin-conserving elements are integrated (the
    // solver's passes, which read no other; callers pass 0 otherwise)
    q.spin_half = (rank == 2 && nv == no && nv == 2 * spin_half) ? spin_half : 0;
    analyse_grid(ng, hti, hG, full, &q.step, &q.uniform, &q.same);
    q.symmetric = grid_symmetric(ng, hti);
    q.mirror = grid_mirrored(ng, hti);
    if (full) return quad_dense_launch(ctx, mode, q, tbar, ti, hti, G, D, ev, eo, out, res);
    size_t smem = quad_smem(ng, q.uniform, q.step, q.full);
    long long blocks = (P + QT - 1) / QT;
    long long cap = (long long)ctx->sm_count * 16;
    int grid = (int)std::min(blocks, cap);
    KV_TRY(kv_smem_optin(ctx, mode == 0 ? (q.uniform ? quad_kernel<0, true> : quad_kernel<0, false>)
                                        : (q.uniform ? quad_kernel<1, true> : quad_kernel<1, false>),
                         quad_smem(MAXNG, 0, 0, 1)));
    // algorithmic bytes: tbar in, T out (mode 0); tbar + T_old in, T_old out
    // (mode 1); with spin blocks, of the spin-conserving elements
    KvProfScope prof(ctx, KV_CAT_QUAD, 8.0 * ng * (double)P * (mode == 0 ? 2 : 3) *
                                           kv_spin_frac(nv, no, q.spin_half));
    if (mode == 0) {
        if (q.uniform)
            kv_launch(ctx, quad_kernel<0, true>, grid, QT, smem, q, tbar, ti, G, D, ev, eo, out,
                      nullptr);
        else
            kv_launch(ctx, quad_kernel<0, false>, grid, QT, smem, q, tbar, ti, G, D, ev, eo, out,
                      nullptr);
        return kv_launch_check(ctx, "quad_kernel");
    }
    void *part = nullptr;
    KV_TRY(kv_scratch(ctx, "quad_partial", sizeof(double) * 2 * grid, &part));
    if (q.uniform)
        kv_launch(ctx, quad_kernel<1, true>, grid, QT, smem, q, tbar, ti, G, D, ev, eo, out,
                  (double *)part);
    else
        kv_launch(ctx, quad_kernel<1, false>, grid, QT, smem, q, tbar, ti, G, D, ev, eo, out,
                  (double *)part);
    KV_TRY(kv_launch_check(ctx, "quad_update_kernel"));
    kv_launch(ctx, reduce_pairs_kernel, 1, 256, 0, (const double *)part, grid, res);
    return kv_launch_check(ctx, "reduce_pairs");
}

namespace {

int int_tbar_entry(kvft_ctx *ctx, int rank, int ng, int nv, int no, const double *tbar,
                   const double *ti, const double *D, const double *G, int full,
                   double *out) {
    if (!ctx || ng < 1 || ng > MAXNG || nv <= 0 || no <= 0 || !tbar || !ti || !D || !G || !out)
        return kv_fail(ctx, KVFT_EINVAL, "int_tbar: bad argument (ng must be 1..64)");
    if (tbar == out) return kv_fail(ctx, KVFT_EINVAL, "int_tbar: output must not alias input");
    cudaSetDevice(ctx->device);
    std::vector<double> hti(ng), hG((size_t)ng * ng);
    KV_CHECK(ctx, cudaMemcpyAsync(hti.data(), ti, sizeof(double) * ng, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    KV_CHECK(ctx, cudaMemcpyAsync(hG.data(), G, sizeof(double) * ng * ng,
                                  cudaMemcpyDeviceToHost, ctx->stream));
    KV_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    long long P = (long long)nv * no * (rank == 2 ? (long long)nv * no : 1LL);
    return kv_quad_launch(ctx, 0, ng, P, rank, nv, no, tbar, ti, hti.data(), G, hG.data(), D,
                          nullptr, nullptr, full, 0.0, out, nullptr, 0);
}

int int_tbar_single_entry(kvft_ctx *ctx, int rank, int ng, int ig, int nv, int no,
                          const double *tbar, const double *ti, const double *D,
                          const double *G, double *out) {
    if (!ctx || ng < 1 || ig < 0 || ig >= ng || nv <= 0 || no <= 0 || !tbar || !ti || !D ||
        !G || !out)
        return kv_fail(ctx, KVFT_EINVAL, "int_tbar_single: bad argument");
    cudaSetDevice(ctx->device);
    QuadParams q{};
    q.ng = ng;
    q.P = (long long)nv * no * (rank == 2 ? (long long)nv * no : 1LL);
    long long blocks = (q.P + 255) / 256;
    int grid = (int)std::min(blocks, (long long)ctx->sm_count * 8);
    kv_launch(ctx, quad_single_kernel, grid, 256, 0, q, ig, tbar, ti, G, D, nullptr, nullptr, out);
    return kv_launch_check(ctx, "quad_single");
}

}  // namespace

// one grid point ig of the tau integral for the solver (D or eps form)
int kv_quad_single(kvft_ctx *ctx, int ng, int ig, long long P, int rank, int nv, int no,
                   const double *tbar, const double *ti, const double *G, const double *D,
                   const double *ev, const double *eo, double *out) {
    QuadParams q{};
    q.ng = ng;
    q.P = P;
    q.rank = rank;
    q.nv = nv;
    q.no = no;
    const int grid = (int)std::min((P + 255) / 256, (long long)ctx->sm_count * 8);
    KvProfScope prof(ctx, KV_CAT_QUAD, 8.0 * (double)P * (ng + 1));
    kv_launch(ctx, quad_single_kernel, grid, 256, 0, q, ig, tbar, ti, G, D, ev, eo, out);
    return kv_launch_check(ctx, "quad_single");
}

int kv_int_tbar(kvft_ctx *ctx, int ng, size_t P, const double *tbar, const double *ti,
                const double *D, const double *eps_v, const double *eps_o, int nv, int no,
                int rank, const double *G, int full, double *out) {
    std::vector<double> hti(ng), hG((size_t)ng * ng);
    KV_CHECK(ctx, cudaMemcpyAsync(hti.data(), ti, sizeof(double) * ng, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    KV_CHECK(ctx, cudaMemcpyAsync(hG.data(), G, sizeof(double) * ng * ng,
                                  cudaMemcpyDeviceToHost, ctx->stream));
    KV_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
    return kv_quad_launch(ctx, 0, ng, (long long)P, rank, nv, no, tbar, ti, hti.data(), G,
                          hG.data(), D, eps_v, eps_o, full, 0.0, out, nullptr, 0);
}

extern "C" {

int kvft_int_tbar1(kvft_ctx *ctx, int ng, int nv, int no, const double *t1bar,
                   const double *ti, const double *D1, const double *G, int full,
                   double *t1out) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_int_tbar1: not on a dry-run context");
    return int_tbar_entry(ctx, 1, ng, nv, no, t1bar, ti, D1, G, full, t1out);
}

int kvft_int_tbar2(kvft_ctx *ctx, int ng, int nv, int no, const double *t2bar,
                   const double *ti, const double *D2, const double *G, int full,
                   double *t2out) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_int_tbar2: not on a dry-run context");
    return int_tbar_entry(ctx, 2, ng, nv, no, t2bar, ti, D2, G, full, t2out);
}

int kvft_int_tbar1_single(kvft_ctx *ctx, int ng, int ig, int nv, int no,
                          const double *t1bar, const double *ti, const double *D1,
                          const double *G, double *t1out) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_int_tbar1_single: not on a dry-run context");
    return int_tbar_single_entry(ctx, 1, ng, ig, nv, no, t1bar, ti, D1, G, t1out);
}

int kvft_int_tbar2_single(kvft_ctx *ctx, int ng, int ig, int nv, int no,
                          const double *t2bar, const double *ti, const double *D2,
                          const double *G, double *t2out) {
    if (ctx && ctx->dry) return kv_fail(ctx, KVFT_EINVAL, "kvft_int_tbar2_single: not on a dry-run context");
    return int_tbar_single_entry(ctx, 2, ng, ig, nv, no, t2bar, ti, D2, G, t2out);
}

}  // extern "C"

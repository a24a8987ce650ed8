// gl.cu -- Gauss-Legendre quadrature, the P_l(mu) table, the shifted Legendre
// basis and the asymptotic geometric factor, all FP64 on the GPU.
#include "common.cuh"
#include "divsmall.cuh"
#include "legendre.cuh"

namespace modal {

// ---------------------------------------------------------------------------
// Gauss-Legendre nodes/weights (replaces asy, gl_integration.c:46-168; same
// ascending symmetric layout).  One thread per positive root theta (x = cos theta), from Olver's
// uniform expansion in the zeros of J_0 (DLMF 18.16(v)): psi = j_{0,k} / (n + 1/2),
//     theta = psi + (psi cot psi - 1) / (8 psi (n + 1/2)^2),
// within 1e-11 of the root (relative) for n >= 751.  P_n(cos theta) by the three-term recurrence
// in differences D_l = P_l - P_{l-1} with y = 1 - x = 2 sin^2(theta/2):
//     D_{l+1} = (l D_l - (2l+1) y P_l) / (l+1),  P_{l+1} = P_l + D_{l+1},
// which stays accurate next to x = 1, where the small endpoint weights carry a large share of the
// Gamma integrand.  With f(theta) = P_n(cos theta), df = -n Q / sin theta, Q = P_{n-1} - x P_n, and
// Legendre's equation d2f = -cot df - n(n+1) f (and its derivative for d3f), a step d = -f/df that is
// small enough is completed to third order and the derivative carried to the root,
//     w = 2 / df(theta + d)^2,
// so that one recurrence per root does for n >= 31 (two for smaller n; 30 at most).
// The bound is that recurrence: a quarter of an SM takes one FP64 warp instruction per 64 cycles, so
// it counts instructions of one warp.  The warp that recurs has six per step; a second one, on
// another quarter, prepares l, 1/(l+1) and (2l+1) y a chunk ahead (nine in one warp: n = 1501
// 448 us, now 324 us, the same bits; n = 3001 by a Newton iteration of about 20
// recurrences with a full division per step: 47.4 ms).
// ---------------------------------------------------------------------------
constexpr int GL_CH = 32;  // steps per chunk of the recurrence

// P_n and Q at cos(theta) for the 32 threads of warp 0, th on both warps (uniform control flow; 64 threads).
__device__ __forceinline__ void leg_diff(int n, double th, double &Pn, double &Q)
{
    __shared__ double rec[2][GL_CH], num[2][GL_CH + 1], tt[2][GL_CH][32];
    const int lane = threadIdx.x & 31;
    const bool ahead = threadIdx.x >= 32;
    const double s = sin(0.5 * th), y = 2.0 * s * s;
    double P = 1.0, D = 0.0;
    auto prepare = [&](int c0) {
        const int b = (c0 / GL_CH) & 1;
        const double l1 = (double)(c0 + lane + 1);
        rec[b][lane] = 1.0 / l1;
        num[b][lane + 1] = l1;
        if (lane == 0) num[b][0] = l1 - 1.0;
        __syncwarp();
#pragma unroll 4
        for (int i = 0; i < GL_CH; i++) tt[b][i][lane] = (num[b][i] + num[b][i + 1]) * y;
    };
    __syncthreads();
    if (ahead) prepare(0);
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += GL_CH) {
        if (ahead) {
            if (c0 + GL_CH < n) prepare(c0 + GL_CH);
        } else {
            const int b = (c0 / GL_CH) & 1;
            const int m = min(GL_CH, n - c0);
#pragma unroll 8
            for (int i = 0; i < m; i++) {
                D = div_small(fma(num[b][i], D, -(tt[b][i][lane] * P)), num[b][i + 1], rec[b][i]);
                P += D;
            }
        }
        __syncthreads();
    }
    Pn = P;
    Q = -D + y * P;
}

// Olver's approximation of the k-th root (k = 1 next to theta = 0).
__device__ __forceinline__ double gl_guess(int n, int k)
{
    // the first zeros of J_0, then McMahon's expansion
    const double j0[8] = {2.4048255576957728, 5.5200781102863106, 8.6537279129110122, 11.791534439014281,
                          14.930917708487785, 18.071063967910922, 21.211636629879259, 24.352471530749303};
    const double b = (k - 0.25) * 3.14159265358979323846, e = 1.0 / (8.0 * b), e2 = e * e;
    const double j = k <= 8 ? j0[k - 1] : b + e * (1.0 - e2 * (124.0 / 3.0 - e2 * (120928.0 / 15.0)));
    const double v = n + 0.5, ps = j / v;
    return ps + (ps * cos(ps) / sin(ps) - 1.0) / (8.0 * ps * v * v);
}

__global__ void __launch_bounds__(GL_THREADS) k_gl_nodes(int n, double *mu, double *w)
{
    const int half = n / 2;
    __shared__ double s_th[32];
    const int lane = threadIdx.x & 31;
    const bool first = threadIdx.x < 32;        // warp 0 holds the roots, warp 1 works ahead for it
    const int k = blockIdx.x * 32 + lane + 1;  // root index 1..half (+ middle)
    const bool root = first && k <= half, mid = first && k == half + 1 && (n & 1);
    double th = root ? gl_guess(n, k) : 1.5707963267948966192313216916397514, wk = 0.0;
    bool open = root || mid;
    for (int it = 0; it < 30; it++) {
        double f, Q;
        if (first) s_th[lane] = th;
        __syncthreads();
        leg_diff(n, s_th[lane], f, Q);
        if (open && mid) {
            wk = 2.0 / ((double)n * n * Q * Q);
            open = false;
        } else if (open) {
            const double st = sin(th), f1 = -n * Q / st, d = -f / f1;
            if ((fabs(d) <= 1e-6 * th && n * fabs(d) <= 1e-5) || it == 29) {
                const double nn = (double)n * (n + 1.0), cot = cos(th) / st, f2 = -cot * f1 - nn * f,
                             f3 = f1 / (st * st) - cot * f2 - nn * f1;
                const double dd = d - f2 / (2.0 * f1) * d * d, g = f1 + dd * (f2 + 0.5 * dd * f3);
                th += dd;
                wk = 2.0 / (g * g);
                open = false;
            } else {
                th += d;
            }
        }
        if (!__syncthreads_or(open)) break;
    }
    if (root) {
        const double x = cos(th);
        mu[n - k] = x;
        mu[k - 1] = -x;
        w[n - k] = wk;
        w[k - 1] = wk;
    } else if (mid) {
        mu[half] = 0.0;
        w[half] = wk;
    }
}

modal_status gl_nodes_dev(modal_ctx *ctx, int n, double *d_mu, double *d_w)
{
    const int threads = 32;  // roots per block: one recurring warp per SM
    const int roots = n / 2 + 1;
    k_gl_nodes<<<ceil_div(roots, threads), GL_THREADS, 0, ctx->stream>>>(n, d_mu, d_w);
    return launched(ctx, "gl_nodes");
}

// ---------------------------------------------------------------------------
// P_l table: pl[l][k] = (2l+1)^{2/3} P_l(mu_k), l = 0..lmax (gl_Pl of
// orthogonalisation_late.c:47-54, stored l-major so each step of the
// recurrence is one coalesced row).  P_l as gsl_sf_legendre_Pl: upward
// recurrence p_l = (x(2l-1)p_{l-1} - (l-1)p_{l-2})/l from P_0 = 1, P_1 = x,
// P_2 returned in closed form, exact values at x = +-1.  One thread per node;
// the (2l+1)^{2/3} factors come from a per-l table.
// ---------------------------------------------------------------------------
// pw[l] = (2l+1)^{2/3}
__global__ void k_pl_factors(int lmax, double *pw)
{
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l <= lmax) pw[l] = pow(2.0 * l + 1.0, 2.0 / 3.0);
}

// One thread per node, so that the n_mu independent recurrences spread over as
// many warps as possible: the recurrence is serial in l, so the length of the FP64
// dependency chain, not the bytes written, sets the time.  The arithmetic is
// gsl_sf_legendre_Pl's upward recurrence, (x (2l-1) P_{l-1} - (l-1) P_{l-2}) / l, the division by
// Markstein's correction (div_small: the same bits).  A quarter of an SM takes one FP64 warp
// instruction per 64 cycles, so the time is a warp's instruction count: warp 0 recurs (five per
// step), warp 1 forms x (2l-1) a chunk of PL_CH steps ahead, warp 2 scales and stores the chunk
// before.  1802 nodes to l = 1201: 244 us, all eight in one warp 363 us, with a full division 576 us; the same
// bits throughout.
constexpr int PL_CH = 16;
__global__ void __launch_bounds__(PL_THREADS) k_legendre_table(int nmu, int lmax, const double *__restrict__ mu,
                                                               const double *__restrict__ pw, double *__restrict__ pl)
{
    // [lmax+1][3]: l, 1/l, (2l+1)^{2/3}: loads, where conversions would take turns on the FP64
    // pipe and a global load of the factor would stall the chain
    extern __shared__ double tab[];
    __shared__ double st[2][PL_CH][32], sp[2][PL_CH][32];
    for (int l = threadIdx.x; l <= lmax; l += blockDim.x) {
        tab[3 * l] = (double)l;
        tab[3 * l + 1] = l > 0 ? 1.0 / (double)l : 0.0;
        tab[3 * l + 2] = pw[l];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * 32 + lane;
    const double x = k < nmu ? mu[k] : 0.0;
    const bool edge = x == 1.0 || x == -1.0;  // exact values there
    double *o = pl + k;
    double pm2 = 1.0, pm1 = x, c1 = 1.0;
    auto ahead = [&](int c) {  // x (2l - 1) of chunk c
        for (int i = 0; i < PL_CH; i++) {
            const int l = 3 + c * PL_CH + i;
            if (l <= lmax) st[c & 1][i][lane] = x * (double)(2 * l - 1);
        }
    };
    if (warp == 0) {
        if (k < nmu) {
            o[0] = tab[2];
            if (lmax >= 1) o[nmu] = tab[5] * x;
        }
        if (lmax >= 2) {
            // P_2 in closed form, as GSL; the recurrence goes on from its own value
            const double pr = div_small(fma(x * 3.0, pm1, -(c1 * pm2)), 2.0, tab[7]);
            pm2 = pm1;
            pm1 = pr;
            c1 = 2.0;
            if (k < nmu) o[2 * (size_t)nmu] = tab[8] * (0.5 * (3.0 * x * x - 1.0));
        }
    } else if (warp == 1)
        ahead(0);
    __syncthreads();
    const int nc = lmax >= 3 ? (lmax - 3) / PL_CH + 1 : 0;  // chunks of l = 3 .. lmax
    for (int c = 0; c <= nc; c++) {
        const int l0 = 3 + c * PL_CH;
        if (warp == 0) {
            if (c < nc) {
                const int m = min(PL_CH, lmax - l0 + 1);
                auto step = [&](int i) {
                    const double cl = tab[3 * (l0 + i)];
                    const double pr = div_small(fma(st[c & 1][i][lane], pm1, -(c1 * pm2)), cl, tab[3 * (l0 + i) + 1]);
                    pm2 = pm1;
                    pm1 = pr;
                    c1 = cl;
                    sp[c & 1][i][lane] = pr;
                };
                if (m == PL_CH) {
#pragma unroll
                    for (int i = 0; i < PL_CH; i++) step(i);
                } else
                    for (int i = 0; i < m; i++) step(i);
            }
        } else if (warp == 1) {
            if (c + 1 < nc) ahead(c + 1);
        } else if (c > 0 && k < nmu) {
            const int b0 = l0 - PL_CH, m = min(PL_CH, lmax - b0 + 1);
#pragma unroll 4
            for (int i = 0; i < m; i++) {
                const int l = b0 + i;
                const double pr = sp[(c - 1) & 1][i][lane];
                o[(size_t)l * nmu] = tab[3 * l + 2] * (edge ? (x > 0.0 || !(l & 1) ? 1.0 : -1.0) : pr);
            }
        }
        __syncthreads();
    }
}

modal_status legendre_table_dev(modal_ctx *ctx, int nmu, int lmax, const double *d_mu, double *d_pl)
{
    MODAL_TRY(ensure(ctx->scratch2, sizeof(double) * (lmax + 1)));
    double *pw = ctx->scratch2.as<double>();
    k_pl_factors<<<ceil_div(lmax + 1, 256), 256, 0, ctx->stream>>>(lmax, pw);
    MODAL_TRY(launched(ctx, "pl_factors"));
    const size_t smem = sizeof(double) * 3 * (size_t)(lmax + 1);
    if (smem > PL_SMEM_MAX) { set_error("legendre table: lmax = %d too large", lmax); return MODAL_ERR_ARG; }
    // the limit, not this call's size: the allocation-free entry point launches the kernel with its own size
    MODAL_CUDA(cudaFuncSetAttribute(k_legendre_table, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM_MAX));
    k_legendre_table<<<ceil_div(nmu, 32), PL_THREADS, smem, ctx->stream>>>(nmu, lmax, d_mu, pw, d_pl);
    return launched(ctx, "legendre_table");
}

// ---------------------------------------------------------------------------
// Shifted Legendre basis (basis_functions.c:88-107): one thread per value.
// ---------------------------------------------------------------------------
__global__ void k_basis_legendre(int size, int pmax, double min, double max, const double *__restrict__ values,
                                 double *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= size) return;
    double *a = out + (size_t)i * (pmax + 1);
    double x = (values[i] - min) / (max - min);
    a[0] = 1e0;
    if (pmax > 0) a[1] = 2e0 * x - 1e0;
    double a1 = 2e0 * x - 1e0, am2 = 1e0, am1 = a1;
    for (int j = 2; j <= pmax; j++) {
        double v = ((2e0 * j - 1e0) * a1 * am1 - (j - 1e0) * am2) / (1e0 * j);
        a[j] = v;
        am2 = am1;
        am1 = v;
    }
}

// ---------------------------------------------------------------------------
// Asymptotic geometric factor (calculate_geometric.c:59-92).
// ---------------------------------------------------------------------------
__global__ void k_geometric(long npts, const int *__restrict__ pts, double *__restrict__ out)
{
    long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npts) return;
    int l1 = pts[3 * n], l2 = pts[3 * n + 1], l3 = pts[3 * n + 2];
    double r = 0.0;
    if (((l1 + l2 + l3) % 2) == 0 && l1 + l2 >= l3 && l2 + l3 >= l1 && l3 + l1 >= l2) {
        double s1 = l1 + l2 + l3 + 1.0, s3 = l1 + l2 + l3 + 1.0 / 3.0, s6 = l1 + l2 + l3 + 1.0 / 6.0;
        double s13 = l2 + l3 - l1 + 1.0 / 3.0, s23 = l3 + l1 - l2 + 1.0 / 3.0, s33 = l1 + l2 - l3 + 1.0 / 3.0;
        double s16 = l2 + l3 - l1 + 1.0 / 6.0, s26 = l3 + l1 - l2 + 1.0 / 6.0, s36 = l1 + l2 - l3 + 1.0 / 6.0;
        const double ipi = 0.318309886183790671537767526745028724;
        double fact = ipi * ipi / 2.0;
        double p1 = fact * ((2.0 * l1 + 1.0) * (2.0 * l2 + 1.0) * (2.0 * l3 + 1.0)) / s1;
        double p2 = s3 / (s13 * s23 * s33);
        double p3 = sqrt(s16 * s26 * s36 / s6);
        r = p1 * p2 * p3;
    }
    out[n] = r;
}

// out[c][r] = in[r][c] for an R x C row-major FP64 matrix.
__global__ void k_transpose(const double *__restrict__ in, double *__restrict__ out, int R, int C)
{
    __shared__ double t[32][33];
    int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        int r = r0 + y, c = c0 + threadIdx.x;
        if (r < R && c < C) t[y][threadIdx.x] = in[(size_t)r * C + c];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        int c = c0 + y, r = r0 + threadIdx.x;
        if (r < R && c < C) out[(size_t)c * R + r] = t[threadIdx.x][y];
    }
}

modal_status transpose_dev(modal_ctx *ctx, const double *in, double *out, int R, int C)
{
    dim3 grid(ceil_div(C, 32), ceil_div(R, 32)), block(32, 8);
    k_transpose<<<grid, block, 0, ctx->stream>>>(in, out, R, C);
    return launched(ctx, "transpose");
}

modal_status basis_legendre_dev(modal_ctx *ctx, int size, int pmax, double min, double max, const double *d_values,
                                double *d_out)
{
    k_basis_legendre<<<ceil_div(size, 128), 128, 0, ctx->stream>>>(size, pmax, min, max, d_values, d_out);
    return launched(ctx, "basis_legendre");
}

modal_status geometric_dev(modal_ctx *ctx, long npts, const int *d_pts, double *d_out)
{
    k_geometric<<<ceil_div(npts, 256), 256, 0, ctx->stream>>>(npts, d_pts, d_out);
    return launched(ctx, "geometric");
}

}  // namespace modal

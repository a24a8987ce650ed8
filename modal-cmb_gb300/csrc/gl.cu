// gl.cu -- Gauss-Legendre quadrature, the P_l(mu) table, the shifted Legendre
// basis and the asymptotic geometric factor, all FP64 on the GPU.
#include "common.cuh"

namespace modal {

// n / c for a small positive integer c and r = 1 / c rounded: Markstein's correction of n r (P. W.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Develop. 34 (1990)).  Three dependent operations instead of a division's dozen, and the same
// bits: the residual is exact, and a quotient by c < 2^13 is never within 2^-14 ulp of a midpoint.
__device__ __forceinline__ double div_small(double n, double c, double r)
{
    const double q = n * r;
    return fma(fma(-q, c, n), r, q);
}

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
// The bound is that recurrence: n steps of six dependent FP64 operations, one warp per SM.
// n = 3001: 47.4 -> 1.06 ms per call (the Newton iteration before this ran until a step fell below
// 1e-17, about 20 recurrences, with a full division per step); weights as accurate as before (4e-14).
// ---------------------------------------------------------------------------
constexpr int GL_CH = 256;  // reciprocals staged per chunk of the recurrence

// P_n and Q at cos(theta) for every thread of the block (uniform control flow).
__device__ __forceinline__ void leg_diff(int n, double th, double &Pn, double &Q)
{
    __shared__ double rec[GL_CH];
    const double s = sin(0.5 * th), y = 2.0 * s * s;
    double P = 1.0, D = 0.0, l = 0.0;
    for (int c0 = 0; c0 < n; c0 += GL_CH) {
        __syncthreads();
        for (int i = threadIdx.x; i < GL_CH; i += blockDim.x) rec[i] = 1.0 / (double)(c0 + i + 1);
        __syncthreads();
        const int m = min(GL_CH, n - c0);
#pragma unroll 4
        for (int i = 0; i < m; i++) {
            const double t = (2.0 * l + 1.0) * y, l1 = l + 1.0;
            D = div_small(fma(l, D, -(t * P)), l1, rec[i]);
            P += D;
            l = l1;
        }
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

__global__ void k_gl_nodes(int n, double *mu, double *w)
{
    const int half = n / 2;
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;  // root index 1..half (+ middle)
    const bool root = k <= half, mid = k == half + 1 && (n & 1);
    double th = root ? gl_guess(n, k) : 1.5707963267948966192313216916397514, wk = 0.0;
    bool open = root || mid;
    for (int it = 0; it < 30; it++) {
        double f, Q;
        leg_diff(n, th, f, Q);
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
    const int threads = 32;  // one warp per SM: the roots' recurrences share an SM's FP64 pipe otherwise
    const int roots = n / 2 + 1;
    k_gl_nodes<<<ceil_div(roots, threads), threads, 0, ctx->stream>>>(n, d_mu, d_w);
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
// Markstein's correction (div_small: the same bits), which leaves four dependent operations per
// step instead of about fifteen.
// 1802 nodes to l = 1201: 576 -> 345 us, bit-identical.
constexpr int PL_WPB = 1;  // warps per block (measured: 1 and 4 give the same time; the chains do not contend)
__global__ void __launch_bounds__(32 * PL_WPB) k_legendre_table(int nmu, int lmax, const double *__restrict__ mu,
                                                                const double *__restrict__ pw, double *__restrict__ pl)
{
    // [lmax+1][3]: 2l - 1, 1/l, (2l+1)^{2/3}: loads, where conversions would take turns on the FP64
    // pipe and a global load of the factor would stall the chain
    extern __shared__ double tab[];
    for (int l = threadIdx.x; l <= lmax; l += blockDim.x) {
        tab[3 * l] = (double)(2 * l - 1);
        tab[3 * l + 1] = l > 0 ? 1.0 / (double)l : 0.0;
        tab[3 * l + 2] = pw[l];
    }
    __syncthreads();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nmu) return;
    const double x = mu[k];
    const bool edge = x == 1.0 || x == -1.0;  // exact values there
    double *o = pl + k;
    o[0] = tab[2];
    if (lmax >= 1) o[nmu] = tab[5] * x;
    double pm2 = 1.0, pm1 = x, c1 = 1.0;
    if (lmax >= 2) {
        // P_2 in closed form, as GSL; the recurrence goes on from its own value
        const double pr = div_small(fma(x * tab[6], pm1, -(c1 * pm2)), 2.0, tab[7]);
        pm2 = pm1;
        pm1 = pr;
        c1 = 2.0;
        o[2 * (size_t)nmu] = tab[8] * (0.5 * (3.0 * x * x - 1.0));
    }
#pragma unroll 4
    for (int l = 3; l <= lmax; l++) {
        const double c = c1 + 1.0;
        const double pr = div_small(fma(x * tab[3 * l], pm1, -(c1 * pm2)), c, tab[3 * l + 1]);
        pm2 = pm1;
        pm1 = pr;
        c1 = c;
        o[(size_t)l * nmu] = tab[3 * l + 2] * (edge ? (x > 0.0 || !(l & 1) ? 1.0 : -1.0) : pr);
    }
}

modal_status legendre_table_dev(modal_ctx *ctx, int nmu, int lmax, const double *d_mu, double *d_pl)
{
    MODAL_TRY(ensure(ctx->scratch2, sizeof(double) * (lmax + 1)));
    double *pw = ctx->scratch2.as<double>();
    k_pl_factors<<<ceil_div(lmax + 1, 256), 256, 0, ctx->stream>>>(lmax, pw);
    MODAL_TRY(launched(ctx, "pl_factors"));
    const size_t smem = sizeof(double) * 3 * (size_t)(lmax + 1);
    if (smem > 200 * 1024) { set_error("legendre table: lmax = %d too large", lmax); return MODAL_ERR_ARG; }
    // the limit, not this call's size: the allocation-free entry point launches the kernel with its own size
    MODAL_CUDA(cudaFuncSetAttribute(k_legendre_table, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    k_legendre_table<<<ceil_div(nmu, 32 * PL_WPB), 32 * PL_WPB, smem, ctx->stream>>>(nmu, lmax, d_mu, pw, d_pl);
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

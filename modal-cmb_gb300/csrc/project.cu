// project.cu -- projection of bispectrum shapes onto the modes.
//
// Reference (calculate_mode_3D, calculate_mode_3D.c:217-264, over the walk of
// get_ijk_next_XXX, tetrapyd_tools.c:104-142):
//   beta_r = sum_{i<=j<=k<=lmax, k<=i+j, i+j+k even}
//            permsix(i,j,k) h~^2(i,j,k) prod (2l+1)^{-1/3} S(i,j,k) w_i w_j w_k
//            * plijk_TTT(r,i,j,k)
// with plijk_TTT the 1/6 sum of the six q-products (orthogonalisation_late.c:620-644).
//
// Sum factorisation: with f(i,j,k) the scalar weight above,
//   B[a][b][c] = sum_i q_a(i) sum_j q_b(j) sum_k f(i,j,k) q_c(k)
//   beta_r     = (1/6) sum over the six orderings s of B[p_s1][p_s2][p_s3]
// for mode r = (p1,p2,p3).  That is O(points * P) instead of O(points * N).
// One CTA per shape and slab l1 = i; the tetrapyd rows j are processed JC at a time:
//   phase 1: f(i,j,k) for the JC rows into shared memory (shape evaluated here)
//   phase 2: H[j][c] = sum_k f(i,j,k) q_c(k)
//   phase 3: F_i[b][c] += sum_j q_b(j) H[j][c]          (registers)
// F_i goes to a [S][L][P*P] buffer; a second pass forms B and beta.
#include <algorithm>
#include <vector>
#include "common.cuh"

namespace modal {

// s_n(i,j,k) / (wq_i wq_j wq_k) of calculate_sijk_TTT (calculate_gamma_3d.c:813-860):
// the trapezium integral (integrate, :783-811) over x of x^2 (1/6) sum over the six
// orderings of q~(i,a) q~(j,b) q~(k,c), with the reference's rule that drops any of
// the first 10 samples above 1e-18 applied to the weighted sample.  The weights
// wq come back through the projection's point weight.
__device__ double d_radial(const RadialArgs &ra, int n, int i, int j, int k)
{
    const int a1 = ra.prim[3 * n], a2 = ra.prim[3 * n + 1], a3 = ra.prim[3 * n + 2], L1 = ra.L1;
    const double wp = ra.wq[i] * ra.wq[j] * ra.wq[k];
    double r = 0.0, yprev = 0.0;
    for (int x = 0; x < ra.xsize; x++) {
        const double *qx = ra.qt + (size_t)x * ra.Pp * L1;
        const double *q1 = qx + (size_t)a1 * L1, *q2 = qx + (size_t)a2 * L1, *q3 = qx + (size_t)a3 * L1;
        const double p1 = q1[i], p2 = q2[i], p3 = q3[i], p4 = q1[j], p5 = q2[j], p6 = q3[j], p7 = q1[k], p8 = q2[k],
                     p9 = q3[k];
        const double sum = p1 * p5 * p9 + p2 * p6 * p7 + p3 * p4 * p8 + p3 * p5 * p7 + p2 * p4 * p9 + p1 * p6 * p8;
        double y = ra.x[x] * ra.x[x] * sum * (1.0 / 6.0);
        if (x < 10 && fabs(wp * y) > 1e-18) y = 0.0;
        if (x > 0) r += (ra.x[x] - ra.x[x - 1]) * (yprev + y) * 0.5;
        yprev = y;
    }
    return r;
}

// Trapezium weight of sample x: the sum over x of w_x y_x equals the reference's
// sum over intervals of (x_x - x_{x-1}) (y_{x-1} + y_x) / 2.
__device__ __forceinline__ double trap_w(const RadialArgs &ra, int x)
{
    const double lo = x >= 1 ? ra.x[x] - ra.x[x - 1] : 0.0, hi = x + 1 < ra.xsize ? ra.x[x + 1] - ra.x[x] : 0.0;
    return 0.5 * (lo + hi);
}

constexpr int RAD_X0 = 10;  // samples below this index follow the per-point zeroing rule

// The same radial shape, sum-factorised over the row.  The integrand of sample x
// is linear in q~(k, x): with the row factors
//   U[c][x] = x^2 / 6 (sum over the orderings with q~_{a_c} at k of the
//             q~(i, x) q~(j, x) products),
// y_x = sum_c U[c][x] q~_{a_c}(k, x).  The reference drops y_x for x < 10 when
// |wq_i wq_j wq_k y_x| > 1e-18; where the factorised y_x lies within 1e-10
// (relative) of that threshold, the decision is taken on y_x summed as the
// reference sums it.  tw: [X] trapezium weights; U: [3][X] for this row.
__device__ double d_radial_rows(const RadialArgs &ra, int n, int i, int j, int k, const double *U, const double *tw)
{
    const int a1 = ra.prim[3 * n], a2 = ra.prim[3 * n + 1], a3 = ra.prim[3 * n + 2], L1 = ra.L1, X = ra.xsize;
    const double wp = ra.wq[i] * ra.wq[j] * ra.wq[k];
    double r = 0.0;
    for (int x = 0; x < X; x++) {
        const double *qx = ra.qt + (size_t)x * ra.Pp * L1;
        double y = U[x] * qx[(size_t)a1 * L1 + k];
        y = fma(U[X + x], qx[(size_t)a2 * L1 + k], y);
        y = fma(U[2 * X + x], qx[(size_t)a3 * L1 + k], y);
        if (x < RAD_X0) {
            const double t = fabs(wp * y);
            bool drop = t > 1e-18;
            if (t > 1e-18 * (1.0 - 1e-10) && t < 1e-18 * (1.0 + 1e-10)) {
                const double *q1 = qx + (size_t)a1 * L1, *q2 = qx + (size_t)a2 * L1, *q3 = qx + (size_t)a3 * L1;
                const double p1 = q1[i], p2 = q2[i], p3 = q3[i], p4 = q1[j], p5 = q2[j], p6 = q3[j], p7 = q1[k],
                             p8 = q2[k], p9 = q3[k];
                const double sum =
                    p1 * p5 * p9 + p2 * p6 * p7 + p3 * p4 * p8 + p3 * p5 * p7 + p2 * p4 * p9 + p1 * p6 * p8;
                drop = fabs(wp * (ra.x[x] * ra.x[x] * sum * (1.0 / 6.0))) > 1e-18;
            }
            if (drop) continue;
        }
        r = fma(tw[x], y, r);
    }
    return r;
}

__device__ __forceinline__ double d_shape(const DShape &s, const double *__restrict__ tab, int stride, int i, int j, int k,
                                          const RadialArgs &ra)
{
    if (s.kind == SHAPE_RADIAL) return d_radial(ra, s.nterms, i, j, k);
    if (s.kind == MODAL_SHAPE_SEPARABLE) {
        double acc = 0.0;
        for (int t = 0; t < s.nterms; t++) {
            const double *f = tab + s.tab_off + (long)t * 3 * stride;
            const double *g = f + stride, *h = g + stride;
            double v = f[i] * g[j] * h[k] + f[i] * g[k] * h[j] + f[j] * g[i] * h[k] + f[j] * g[k] * h[i] +
                       f[k] * g[i] * h[j] + f[k] * g[j] * h[i];
            acc += v / 6.0;
        }
        return acc;
    }
    double L = (double)(i + j + k);
    double x1 = i / L - s.c1, x2 = j / L - s.c2, x3 = k / L - s.c3;
    return exp(-(x1 * x1 + x2 * x2 + x3 * x3) / (2.0 * s.sigma * s.sigma));
}

// A separable shape on a fixed row (i, j), FP64: with the row coefficients
//   c[t] = (f_t(i) g_t(j) + f_t(j) g_t(i), f_t(i) h_t(j) + f_t(j) h_t(i), g_t(i) h_t(j) + g_t(j) h_t(i)) / 6
// the value at k is sum_t (c0 h_t(k) + c1 g_t(k) + c2 f_t(k)): three loads
// and three FMAs per term instead of the six-ordering sum.
constexpr int PJ_TCOEF64 = 8;  // terms per shape with row coefficients (more: d_shape)

__device__ __forceinline__ double d_sep_rows(const DShape &s, const double *__restrict__ tab, int stride, int k,
                                             const double *c)
{
    double acc = 0.0;
    for (int t = 0; t < s.nterms; t++) {
        const double *f = tab + s.tab_off + (long)t * 3 * stride;
        acc = fma(c[3 * t], f[2 * stride + k], acc);
        acc = fma(c[3 * t + 1], f[stride + k], acc);
        acc = fma(c[3 * t + 2], f[k], acc);
    }
    return acc;
}

// 1D factors of the point weight permsix h~^2 prod (2l+1)^{-1/3} w_l:
//   h~^2(l1,l2,l3) = gL(L) g(L - 2 l1) g(L - 2 l2) g(L - 2 l3) prod (2l+1), L = l1 + l2 + l3 (always even),
//   g(x) = sqrt(x + 1/6) / (x + 1/3), gL(L) = (L + 1/3) / (2 pi^2 (L + 1) sqrt(L + 1/6))
// (calculate_geometric.c:59-92 regrouped), w_l = (2l+1)^{1/6} / sqrt(C_l + N_l/b_l^2), w_0 = w_1 = 0
// (calculate_mode_3D.c:53-62, get_weight :283-290).
// v[l] = (2l+1)^{2/3} w_l for l <= lmax, then g[h] = g(2h) and gl[h] = gL(2h) for h < vl_nh.
__host__ __device__ inline int vl_nh(int lmax) { return 3 * lmax / 2 + 1; }
inline size_t vl_count(int lmax) { return (size_t)(lmax + 1) + 2 * (size_t)vl_nh(lmax); }
__global__ void k_vl(int lmax, const double *__restrict__ cl, double *__restrict__ v)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x, nh = vl_nh(lmax);
    if (h <= lmax) v[h] = (h < 2) ? 0.0 : cbrt(2.0 * h + 1.0) * sqrt(2.0 * h + 1.0) / sqrt(cl[h]);
    if (h >= nh) return;
    const double x = 2.0 * h;
    v[lmax + 1 + h] = sqrt(x + 1.0 / 6.0) / (x + 1.0 / 3.0);
    v[lmax + 1 + nh + h] = (x + 1.0 / 3.0) / ((x + 1.0) * sqrt(x + 1.0 / 6.0)) * 0.050660591821168885722;
}

constexpr int JC = 8;

__host__ __device__ inline long long tet_tri_sum(long long u)
{
    // sum_{v=0}^{u} (floor(v/2) + 1): (a+1)^2 for u = 2a, (a+1)(a+2) for u = 2a+1
    if (u < 0) return 0;
    const long long a = u / 2;
    return (u & 1) ? (a + 1) * (a + 2) : (a + 1) * (a + 1);
}

// Points of rows i..j-1 of slab i (rows hold k = j + (i & 1) + 2m <= min(i + j, lmax)).
__host__ __device__ inline long long tet_row_offset(int i, int j, int lmax)
{
    const int ip = i & 1;
    const long long n1 = (i - ip) / 2 + 1;  // points of a row with i + j <= lmax
    const int J1 = lmax - i;                // last such row
    long long off = 0;
    const int e1 = (j - 1 < J1) ? j - 1 : J1;
    if (e1 >= i) off += (long long)(e1 - i + 1) * n1;
    const int s2 = (i > J1 + 1) ? i : J1 + 1;  // rows ending at k = lmax
    if (j - 1 >= s2) off += tet_tri_sum((long long)lmax - ip - s2) - tet_tri_sum((long long)lmax - ip - (j - 1) - 1);
    return off;
}

// base[s] = points of slabs lmin..lmin+s-1 (s = 0..L); one block.
__global__ void k_slab_base(int lmin, int lmax, long long *__restrict__ base)
{
    __shared__ long long part[256];
    const int L = lmax - lmin + 1, per = (L + 255) / 256, t = threadIdx.x;
    const int a = min(L, t * per), b = min(L, a + per);
    long long sum = 0;
    for (int s = a; s < b; s++) sum += tet_row_offset(lmin + s, lmax + 1, lmax);
    part[t] = sum;
    __syncthreads();
    for (int d = 1; d < 256; d <<= 1) {  // inclusive scan
        const long long v = (t >= d) ? part[t - d] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    long long run = part[t] - sum;  // exclusive
    for (int s = a; s < b; s++) {
        base[s] = run;
        run += tet_row_offset(lmin + s, lmax + 1, lmax);
    }
    if (t == 255) base[L] = part[255];
}

// Point weights in slab and row order, from their 1D factors: five FP64 multiplications per
// point (0.36 ms of the FP64 pipe at l <= 1000) over rows of up to l/2 points, a warp each: 0.65 ms;
// the closed form's quotients and square root took 6.3 ms.  Relative error of a weight (rms, units of
// 2^-53): 2.9, the closed form 3.9.
__global__ void __launch_bounds__(256) k_weight_table_fp64(int lmin, int lmax, const double *__restrict__ vl,
                                                           const long long *__restrict__ base, double *__restrict__ Wd)
{
    const int i = lmin + blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = i + blockIdx.y * 8 + warp;
    if (j > lmax) return;
    const int ip = i & 1, kend = min(i + j, lmax), k0 = j + ip;
    if (kend < k0) return;
    const int n = (kend - k0) / 2 + 1;
    double *row = Wd + base[blockIdx.x] + tet_row_offset(i, j, lmax);
    const double *vk = vl + k0;
    const double *gl = vl + lmax + 1 + vl_nh(lmax) + (i + j + k0) / 2;
    const double *g1 = vl + lmax + 1 + (j + k0 - i) / 2, *g2 = vl + lmax + 1 + (i + k0 - j) / 2,
                 *g3 = vl + lmax + 1 + (i + j - k0) / 2;
    const double v1 = vl[i] * vl[j], v3 = 3.0 * v1, v6 = 6.0 * v1;  // with permsix
    for (int m = lane; m < n; m += 32) {
        const bool jk = m == 0 && ip == 0;
        const double v = i == j ? (jk ? v1 : v3) : (jk ? v3 : v6);
        row[m] = (gl[m] * g1[m]) * (g2[m] * g3[-m]) * (v * vk[2 * m]);
    }
}

// One CTA per shape and slab (a shape's slabs in decreasing size).  Bound by the FP64 pipe, one
// warp instruction per 16 cycles of an SM: per point 3 per term and one for the weighted shape
// value, P for the contraction over k, P^2 per row for the one over j; the sums over k run in
// four chains (an FP64 operation takes 65 cycles), and a row's points are one warp's.  At
// l <= 1000, P = 20, four shapes of two terms: 10.3 ms (9.4 ms of FP64 instructions); one CTA per
// slab that takes the shapes in turn, one chain per sum: 13.1 ms.
template <int FPT>
__global__ void __launch_bounds__(256) k_project_slab_fp64(int lmin, int lmax, int P, int KMAX,
                                                            const int *__restrict__ slab_order,
                                                            const double *__restrict__ q,
                                                            const DShape *__restrict__ shapes,
                                                            const double *__restrict__ tab,
                                                            const double *__restrict__ Wd,
                                                            const long long *__restrict__ sbase,
                                                            double *__restrict__ Fbuf, const RadialArgs ra)
{
    extern __shared__ double sm[];
    double *f = sm;               // [JC][KMAX]
    double *H = sm + JC * KMAX;   // [JC][P]
    double *Cf = H + JC * P;      // separable shapes: [JC][PJ_TCOEF64][3] row coefficients (d_sep_rows)
    double *V = Cf + JC * PJ_TCOEF64 * 3;  // radial shapes: [JC][3][X] row factors, then [X] trapezium weights
    const int XR = ra.xsize;
    double *TW = V + (size_t)JC * 3 * XR;
    const int s = blockIdx.x, slab = slab_order[blockIdx.y];
    const int i = lmin + slab;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int PP = P * P, L = lmax - lmin + 1, stride = lmax + 1;
    const int par = i & 1;
    const DShape sh = shapes[s];
    double Facc[FPT];
#pragma unroll
    for (int t = 0; t < FPT; t++) Facc[t] = 0.0;
    const bool radial = sh.kind == SHAPE_RADIAL;
    const bool rowc = sh.kind == MODAL_SHAPE_SEPARABLE && sh.nterms <= PJ_TCOEF64;
    for (int j0 = i; j0 <= lmax; j0 += JC) {
        if (rowc) {
            for (int e = tid; e < JC * sh.nterms; e += 256) {
                const int jj = e / sh.nterms, t = e - jj * sh.nterms, j = min(j0 + jj, lmax);
                const double *f = tab + sh.tab_off + (long)t * 3 * stride, *g = f + stride, *h = g + stride;
                double *c = Cf + ((size_t)jj * PJ_TCOEF64 + t) * 3;
                c[0] = (f[i] * g[j] + f[j] * g[i]) * (1.0 / 6.0);  // with h(k)
                c[1] = (f[i] * h[j] + f[j] * h[i]) * (1.0 / 6.0);  // with g(k)
                c[2] = (g[i] * h[j] + g[j] * h[i]) * (1.0 / 6.0);  // with f(k)
            }
            __syncthreads();
        }
        if (radial) {
            const int a1 = ra.prim[3 * sh.nterms], a2 = ra.prim[3 * sh.nterms + 1], a3 = ra.prim[3 * sh.nterms + 2];
            for (int e = tid; e < JC * XR; e += 256) {
                const int jj = e / XR, x = e - jj * XR, j = min(j0 + jj, lmax);
                const double *qx = ra.qt + (size_t)x * ra.Pp * ra.L1;
                const double p1 = qx[(size_t)a1 * ra.L1 + i], p2 = qx[(size_t)a2 * ra.L1 + i],
                             p3 = qx[(size_t)a3 * ra.L1 + i], p4 = qx[(size_t)a1 * ra.L1 + j],
                             p5 = qx[(size_t)a2 * ra.L1 + j], p6 = qx[(size_t)a3 * ra.L1 + j];
                const double g = ra.x[x] * ra.x[x] * (1.0 / 6.0);
                double *u = V + (size_t)jj * 3 * XR;
                u[x] = g * (p2 * p6 + p3 * p5);           // with q~_{a1}(k)
                u[XR + x] = g * (p3 * p4 + p1 * p6);      // with q~_{a2}(k)
                u[2 * XR + x] = g * (p1 * p5 + p2 * p4);  // with q~_{a3}(k)
            }
            for (int x = tid; x < XR; x += 256) TW[x] = trap_w(ra, x);
            __syncthreads();
        }
        {   // a warp per row
            const int jj = warp, j = j0 + jj, k0 = j + par;
            const int nk = j <= lmax && min(i + j, lmax) >= k0 ? (min(i + j, lmax) - k0) / 2 + 1 : 0;
            if (nk > 0) {
                const double *w = Wd + sbase[slab] + tet_row_offset(i, j, lmax);
                for (int kk = lane; kk < nk; kk += 32) {
                    const int k = k0 + 2 * kk;
                    f[jj * KMAX + kk] = w[kk] * (radial ? d_radial_rows(ra, sh.nterms, i, j, k, V + (size_t)jj * 3 * XR, TW)
                                                 : rowc ? d_sep_rows(sh, tab, stride, k, Cf + (size_t)jj * PJ_TCOEF64 * 3)
                                                        : d_shape(sh, tab, stride, i, j, k, ra));
                }
            }
        }
        __syncthreads();
        for (int e = tid; e < JC * P; e += 256) {
            const int jj = e / P, c = e - jj * P, j = j0 + jj;
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            if (j <= lmax) {
                const int kf = j + par, k1 = min(i + j, lmax), nk = (k1 >= kf) ? (k1 - kf) / 2 + 1 : 0;
                const double *fr = f + jj * KMAX;
                const double *qc = q + (size_t)(kf - lmin) * P + c;
                int kk = 0;
                for (; kk + 4 <= nk; kk += 4)
#pragma unroll
                    for (int u = 0; u < 4; u++) acc[u] = fma(fr[kk + u], qc[(size_t)2 * (kk + u) * P], acc[u]);
#pragma unroll
                for (int u = 0; u < 3; u++)
                    if (kk + u < nk) acc[u] = fma(fr[kk + u], qc[(size_t)2 * (kk + u) * P], acc[u]);
            }
            H[e] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < FPT; t++) {
            const int e = tid + 256 * t;
            if (e < PP) {
                const int b = e / P, c = e - b * P, nj = min(JC, lmax - j0 + 1);
                const double *qb = q + (size_t)(j0 - lmin) * P + b;
                double a = 0.0;
                if (nj == JC) {
#pragma unroll
                    for (int jj = 0; jj < JC; jj++) a = fma(qb[(size_t)jj * P], H[jj * P + c], a);
                } else
                    for (int jj = 0; jj < nj; jj++) a = fma(qb[(size_t)jj * P], H[jj * P + c], a);
                Facc[t] += a;
            }
        }
        // H is written again only after the next rows' points; Cf, V and f before that are not read here
    }
#pragma unroll
    for (int t = 0; t < FPT; t++) {
        const int e = tid + 256 * t;
        if (e < PP) Fbuf[((size_t)s * L + slab) * PP + e] = Facc[t];
    }
}

// B[seg][s][a][bc] = sum over the segment's slabs of q[slab][a] Fbuf[s][slab][bc].  A thread's loop
// is bound by latency, so the slabs are split until the GPU is full (grid.y segments, added by
// k_project_beta), eight loads in flight and four chains.  l <= 1000, P = 20, four shapes: 0.07 ms; one
// segment 0.25 ms.
__global__ void k_project_B(int L, int P, int S, const double *__restrict__ q, const double *__restrict__ Fbuf,
                            double *__restrict__ B)
{
    const int PP = P * P, per = (L + gridDim.y - 1) / gridDim.y, l0 = blockIdx.y * per, l1 = min(L, l0 + per);
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x, n = (size_t)S * P * PP;
    if (e >= n) return;
    int s = (int)(e / ((size_t)P * PP));
    int rem = (int)(e - (size_t)s * P * PP);
    int a = rem / PP, bc = rem - a * PP;
    const double *F = Fbuf + (size_t)s * L * PP + bc;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int l = l0;
    for (; l + 8 <= l1; l += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = F[(size_t)(l + u) * PP];
#pragma unroll
        for (int u = 0; u < 8; u++) acc[u & 3] = fma(q[(size_t)(l + u) * P + a], x[u], acc[u & 3]);
    }
    for (; l < l1; l++) acc[0] = fma(q[(size_t)l * P + a], F[(size_t)l * PP], acc[0]);
    B[blockIdx.y * n + e] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// beta[s][r] = (1/6) sum of B over the six orderings of mode r's triple
__global__ void k_project_beta(int N, int P, int S, int nseg, const int *__restrict__ triples, const double *__restrict__ B,
                               double *__restrict__ beta)
{
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)S * N) return;
    int s = (int)(e / N), r = (int)(e % N);
    int p1 = triples[3 * r], p2 = triples[3 * r + 1], p3 = triples[3 * r + 2];
    const size_t n = (size_t)S * P * P * P;
    const double *b = B + (size_t)s * P * P * P;
    double v = 0.0;
    for (int z = 0; z < nseg; z++, b += n) {
#define BB(x, y, z) b[((size_t)(x) * P + (y)) * P + (z)]
        v += BB(p1, p2, p3) + BB(p2, p3, p1) + BB(p3, p1, p2) + BB(p3, p2, p1) + BB(p2, p1, p3) + BB(p1, p3, p2);
#undef BB
    }
    beta[e] = v / 6e0;
}


// ---------------------------------------------------------------- host side
//
// A projection is planned (shapes validated, every device buffer sized, the
// slab schedule uploaded), its inputs are staged (shape tables and
// descriptors copied to the device), and its device work is recorded on the
// context stream.  The record step allocates nothing and makes no host
// round trip, so modal_project_batch can capture it into a CUDA graph.

modal_status proj_plan(modal_ctx *ctx, int S, const modal_shape *shapes, modal_prec prec, ProjPlan &pl, bool careful)
{
    const int lmin = ctx->lmin, lmax = ctx->lmax, L = ctx->L, P = ctx->P, N = ctx->N, PP = P * P;
    pl = ProjPlan();
    pl.S = S;
    pl.prec = prec;
    pl.careful = careful;
    pl.desc.resize(S);
    long tab_total = 0;
    for (int s = 0; s < S; s++) {
        const modal_shape &m = shapes[s];
        DShape &d = pl.desc[s];
        d.kind = m.kind;
        d.nterms = m.nterms;
        d.tab_off = tab_total;
        d.c1 = m.c[0]; d.c2 = m.c[1]; d.c3 = m.c[2];
        d.sigma = m.sigma;
        if (m.kind == MODAL_SHAPE_SEPARABLE) {
            if (m.nterms < 1 || !m.tab) { set_error("shape %d: separable needs nterms >= 1 and a table", s); return MODAL_ERR_ARG; }
            tab_total += (long)m.nterms * 3 * (lmax + 1);
        } else if (m.kind == MODAL_SHAPE_BUMP) {
            if (!(m.sigma > 0.0)) { set_error("shape %d: bump sigma must be > 0", s); return MODAL_ERR_ARG; }
            d.nterms = 0;
        } else {
            set_error("shape %d: unknown kind %d", s, m.kind);
            return MODAL_ERR_ARG;
        }
    }
    pl.tab_total = tab_total;
    {   // FP32 layout (pf_tab): per term and factor 16 H8 entries, H8 = groups of 8 lattice points per parity
        const long H8 = (lmax / 2 + 1 + 7) / 8 + 4;
        long off = 0;
        for (int s = 0; s < S; s++)
            if (pl.desc[s].kind == MODAL_SHAPE_SEPARABLE) {
                pl.desc[s].tab_off_f = off;
                off += 3L * 16 * H8 * pl.desc[s].nterms;
            }
        pl.tabf_total = off;
    }
    MODAL_TRY(ensure(ctx->shape_tab, sizeof(double) * (size_t)(tab_total > 0 ? tab_total : 1)));
    MODAL_TRY(ensure(ctx->shape_desc, sizeof(DShape) * (size_t)S));
    MODAL_TRY(ensure(ctx->vl, sizeof(double) * vl_count(lmax)));
    MODAL_TRY(ensure(ctx->beta, sizeof(double) * (size_t)S * N));
    if (prec == MODAL_PREC_SPLIT) {
        MODAL_TRY(pf_plan(ctx, pl));
    } else {
        // slab schedule of (lmin, lmax): heaviest slabs first
        if (ctx->slab_lmin != lmin || ctx->slab_lmax != lmax) {
            std::vector<int> order(L);
            std::vector<long long> cnt(L);
            for (int q = 0; q < L; q++) { order[q] = q; cnt[q] = tet_row_offset(lmin + q, lmax + 1, lmax); }
            std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cnt[a] > cnt[b]; });
            ctx->slab_lmin = ctx->slab_lmax = -1;
            MODAL_TRY(ensure(ctx->slab_order, sizeof(int) * (size_t)L));
            MODAL_CUDA(cudaMemcpyAsync(ctx->slab_order.ptr, order.data(), sizeof(int) * L, cudaMemcpyHostToDevice, ctx->stream));
            ctx->slab_lmin = lmin;
            ctx->slab_lmax = lmax;
        }
        const int KMAX = (lmax - lmin) / 2 + 2;
        pl.smem = sizeof(double) * ((size_t)JC * KMAX + (size_t)JC * P + (size_t)JC * PJ_TCOEF64 * 3);
        if (pl.smem > 220 * 1024) { set_error("project: lmax=%d too large for the slab tile", lmax); return MODAL_ERR_ARG; }
        pl.fpt = ceil_div(PP, 256);
        if (pl.fpt > 16) { set_error("project: P=%d too large", P); return MODAL_ERR_ARG; }
        // F partials [S][L][P*P] | B [segments][S][P][P*P] | slab bases [L+1] | weight table [points]
        long long npts = 0;
        for (int i = lmin; i <= lmax; i++) npts += tet_row_offset(i, lmax + 1, lmax);
        pl.npts = npts;
        pl.o_B = sizeof(double) * (size_t)S * L * PP;
        MODAL_CUDA(cudaDeviceGetAttribute(&pl.nsm, cudaDevAttrMultiProcessorCount, ctx->device));
        pl.nseg = (int)std::max<long>(1, std::min<long>(std::min(8, L / 32), 1024L * pl.nsm / ((long)S * P * PP)));
        pl.o_sb = pl.o_B + sizeof(double) * (size_t)pl.nseg * S * P * PP;
        pl.o_w = pl.o_sb + sizeof(long long) * (size_t)(L + 1);
        MODAL_TRY(ensure(ctx->scratch, pl.o_w + sizeof(double) * (size_t)npts));
        auto attr = [&](auto kern) -> modal_status {
            MODAL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
            return MODAL_OK;
        };
        if (pl.fpt <= 1) MODAL_TRY(attr(k_project_slab_fp64<1>));
        else if (pl.fpt <= 4) MODAL_TRY(attr(k_project_slab_fp64<4>));
        else if (pl.fpt <= 8) MODAL_TRY(attr(k_project_slab_fp64<8>));
        else MODAL_TRY(attr(k_project_slab_fp64<16>));
    }
    return MODAL_OK;
}

modal_status proj_stage(modal_ctx *ctx, const ProjPlan &pl, const modal_shape *shapes)
{
    const int lmax = ctx->lmax;
    for (int s = 0; s < pl.S; s++) {
        const modal_shape &m = shapes[s];
        if (m.kind != MODAL_SHAPE_SEPARABLE) continue;
        size_t n = (size_t)m.nterms * 3 * (lmax + 1);
        MODAL_CUDA(cudaMemcpyAsync(ctx->shape_tab.as<double>() + pl.desc[s].tab_off, m.tab, sizeof(double) * n,
                                   cudaMemcpyHostToDevice, ctx->stream));
    }
    MODAL_CUDA(cudaMemcpyAsync(ctx->shape_desc.ptr, pl.desc.data(), sizeof(DShape) * pl.S, cudaMemcpyHostToDevice,
                               ctx->stream));
    return MODAL_OK;
}

modal_status proj_record(modal_ctx *ctx, const ProjPlan &pl)
{
    const int lmin = ctx->lmin, lmax = ctx->lmax, L = ctx->L, P = ctx->P, N = ctx->N, PP = P * P, S = pl.S;
    if (pl.prec == MODAL_PREC_SPLIT) return pf_record(ctx, pl);
    k_vl<<<ceil_div(vl_nh(lmax), 256), 256, 0, ctx->stream>>>(lmax, ctx->cl.as<double>(), ctx->vl.as<double>());
    MODAL_TRY(launched(ctx, "vl"));
    uint8_t *b8 = ctx->scratch.as<uint8_t>();
    double *Fbuf = reinterpret_cast<double *>(b8);
    double *B = reinterpret_cast<double *>(b8 + pl.o_B);
    long long *sbase = reinterpret_cast<long long *>(b8 + pl.o_sb);
    double *Wd = reinterpret_cast<double *>(b8 + pl.o_w);
    k_slab_base<<<1, 256, 0, ctx->stream>>>(lmin, lmax, sbase);
    MODAL_TRY(launched(ctx, "slab_base"));
    k_weight_table_fp64<<<dim3(L, ceil_div(L, 8)), 256, 0, ctx->stream>>>(lmin, lmax, ctx->vl.as<double>(), sbase, Wd);
    MODAL_TRY(launched(ctx, "weight_table_fp64"));
    const int KMAX = (lmax - lmin) / 2 + 2;
    auto run = [&](auto kern) -> modal_status {
        kern<<<dim3(S, L), 256, pl.smem, ctx->stream>>>(lmin, lmax, P, KMAX, ctx->slab_order.as<int>(), ctx->q.as<double>(),
                                                        ctx->shape_desc.as<DShape>(), ctx->shape_tab.as<double>(), Wd,
                                                        sbase, Fbuf, pl.ra);
        return launched(ctx, "project_slab_fp64");
    };
    if (pl.fpt <= 1) MODAL_TRY(run(k_project_slab_fp64<1>));
    else if (pl.fpt <= 4) MODAL_TRY(run(k_project_slab_fp64<4>));
    else if (pl.fpt <= 8) MODAL_TRY(run(k_project_slab_fp64<8>));
    else MODAL_TRY(run(k_project_slab_fp64<16>));
    k_project_B<<<dim3(ceil_div((long)S * P * PP, 256), pl.nseg), 256, 0, ctx->stream>>>(L, P, S, ctx->q.as<double>(), Fbuf, B);
    MODAL_TRY(launched(ctx, "project_B"));
    k_project_beta<<<ceil_div((long)S * N, 256), 256, 0, ctx->stream>>>(N, P, S, pl.nseg, ctx->triples.as<int>(), B,
                                                                          ctx->beta.as<double>());
    return launched(ctx, "project_beta");
}

modal_status project_dev(modal_ctx *ctx, int S, const modal_shape *shapes, modal_prec prec, bool careful)
{
    ProjPlan pl;
    MODAL_TRY(proj_plan(ctx, S, shapes, prec, pl, careful));
    MODAL_TRY(proj_stage(ctx, pl, shapes));
    return proj_record(ctx, pl);
}

__global__ void k_wq(int lmax, const double *__restrict__ cl, double *__restrict__ wq)
{
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l > lmax) return;
    wq[l] = (l < 2) ? 0.0 : pow(2.0 * l + 1.0, 1.0 / 6.0) * (1.0 / sqrt(cl[l]));
}

}  // namespace modal

using namespace modal;

extern "C" modal_status modal_gamma_transfer_3d(modal_ctx *c, double deltaphi, double *gamma_t)
{
    if (!c || !gamma_t) { set_error("modal_gamma_transfer_3d: NULL argument"); return MODAL_ERR_ARG; }
    if (!c->have_modes || !c->have_spec || c->tr_xsize < 2) {
        set_error("modal_gamma_transfer_3d: set basis, modes, spectrum and transfer functions first");
        return MODAL_ERR_STATE;
    }
    if (c->lmin < 2) { set_error("modal_gamma_transfer_3d: lmin must be >= 2"); return MODAL_ERR_ARG; }
    MODAL_CUDA(cudaSetDevice(c->device));
    const int S = c->tr_Nprim, N = c->N, lmax = c->lmax;
    // each primordial mode is one radial shape of the FP64 projection
    std::vector<modal_shape> placeholder(S);
    for (int s = 0; s < S; s++) {
        placeholder[s] = modal_shape{};
        placeholder[s].kind = MODAL_SHAPE_BUMP;
        placeholder[s].sigma = 1.0;
    }
    ProjPlan pl;
    MODAL_TRY(proj_plan(c, S, placeholder.data(), MODAL_PREC_FP64, pl));
    for (int s = 0; s < S; s++) {
        pl.desc[s].kind = SHAPE_RADIAL;
        pl.desc[s].nterms = s;
    }
    MODAL_TRY(ensure(c->scratch2, sizeof(double) * (size_t)(lmax + 1)));
    k_wq<<<ceil_div(lmax + 1, 256), 256, 0, c->stream>>>(lmax, c->cl.as<double>(), c->scratch2.as<double>());
    MODAL_TRY(launched(c, "wq"));
    pl.ra.qt = c->tr_qt.as<double>();
    pl.ra.x = c->tr_x.as<double>();
    pl.ra.wq = c->scratch2.as<double>();
    pl.ra.prim = c->tr_prim.as<int>();
    pl.ra.xsize = c->tr_xsize;
    pl.ra.Pp = c->tr_Pp;
    pl.ra.L1 = lmax + 1;
    // the row factors of d_radial_rows sit after the kernel's f and H tiles
    pl.smem += sizeof(double) * ((size_t)JC * 3 * c->tr_xsize + c->tr_xsize);
    if (pl.smem > 220 * 1024) { set_error("modal_gamma_transfer_3d: lmax=%d, xsize=%d too large for the slab tile", lmax, c->tr_xsize); return MODAL_ERR_ARG; }
    {
        auto attr = [&](auto kern) -> modal_status {
            MODAL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
            return MODAL_OK;
        };
        if (pl.fpt <= 1) MODAL_TRY(attr(k_project_slab_fp64<1>));
        else if (pl.fpt <= 4) MODAL_TRY(attr(k_project_slab_fp64<4>));
        else if (pl.fpt <= 8) MODAL_TRY(attr(k_project_slab_fp64<8>));
        else MODAL_TRY(attr(k_project_slab_fp64<16>));
    }
    {
        StageTimer t(c, MODAL_T_GAMMA);
        MODAL_TRY(proj_stage(c, pl, placeholder.data()));
        MODAL_TRY(proj_record(c, pl));
    }
    std::vector<double> b((size_t)S * N);
    MODAL_CUDA(cudaMemcpyAsync(b.data(), c->beta.ptr, sizeof(double) * b.size(), cudaMemcpyDeviceToHost, c->stream));
    MODAL_CUDA(cudaStreamSynchronize(c->stream));
    c->have_beta = false;  // the device beta holds these radial projections, not shapes'
    const double f = 6.0 * deltaphi * deltaphi;  // calculate_gamma_3d.c:434-439
    for (int m = 0; m < N; m++)
        for (int n = 0; n < S; n++) gamma_t[(size_t)m * S + n] = f * b[(size_t)n * N + m];
    return MODAL_OK;
}

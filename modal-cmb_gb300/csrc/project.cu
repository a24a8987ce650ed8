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
// One CTA per slab l1 = i; the tetrapyd rows j are processed JC at a time:
//   phase 1: f(i,j,k) for the JC rows into shared memory (shape evaluated here)
//   phase 2: H[j][c] = sum_k f(i,j,k) q_c(k)
//   phase 3: F_i[b][c] += sum_j q_b(j) H[j][c]          (registers)
// F_i goes to a [S][L][P*P] buffer; a second pass forms B and beta.
#include <algorithm>
#include <vector>
#include "common.cuh"

namespace modal {

__device__ __forceinline__ double d_permsix(int i, int j, int k)
{
    if (i == k && i == j) return 1.0;
    if (i == j || j == k || i == k) return 3.0;
    return 6.0;
}

// calculate_geometric (calculate_geometric.c:59-92) for a point already known
// to satisfy parity and the triangle condition.
__device__ __forceinline__ double d_geo(int l1, int l2, int l3)
{
    double s1 = l1 + l2 + l3 + 1.0, s3 = l1 + l2 + l3 + 1.0 / 3.0, s6 = l1 + l2 + l3 + 1.0 / 6.0;
    double s13 = l2 + l3 - l1 + 1.0 / 3.0, s23 = l3 + l1 - l2 + 1.0 / 3.0, s33 = l1 + l2 - l3 + 1.0 / 3.0;
    double s16 = l2 + l3 - l1 + 1.0 / 6.0, s26 = l3 + l1 - l2 + 1.0 / 6.0, s36 = l1 + l2 - l3 + 1.0 / 6.0;
    const double ipi = 0.318309886183790671537767526745028724;
    double fact = ipi * ipi / 2.0;
    double p1 = fact * ((2.0 * l1 + 1.0) * (2.0 * l2 + 1.0) * (2.0 * l3 + 1.0)) / s1;
    double p2 = s3 / (s13 * s23 * s33);
    double p3 = sqrt(s16 * s26 * s36 / s6);
    return p1 * p2 * p3;
}

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
//   c[t] = (f_t(i) g_t(j) + f_t(j) g_t(i), f_t(i) h_t(j) + f_t(j) h_t(i), g_t(i) h_t(j) + g_t(j) h_t(i))
// the value at k is (1/6) sum_t (c0 h_t(k) + c1 g_t(k) + c2 f_t(k)): three loads
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
    return acc * (1.0 / 6.0);
}

// v_l = (2l+1)^{-1/3} w_l, w_l = (2l+1)^{1/6}/sqrt(C_l + N_l/b_l^2), w_0 = w_1 = 0
// (calculate_mode_3D.c:53-62, get_weight :283-290).
__global__ void k_vl(int lmax, const double *__restrict__ cl, double *__restrict__ vl)
{
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l > lmax) return;
    vl[l] = (l < 2) ? 0.0 : pow(2.0 * l + 1.0, -1.0 / 3.0) * (pow(2.0 * l + 1.0, 1.0 / 6.0) / sqrt(cl[l]));
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

// FP64 form of the weight table: the same products in the same order as the
// FP64 point weight, so the projection is unchanged to the last bit.
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
    const double vi = vl[i], vj = vl[j];
    for (int m = lane; m < n; m += 32) {
        const int k = k0 + 2 * m;
        row[m] = d_permsix(i, j, k) * d_geo(i, j, k) * vi * vj * vl[k];
    }
}

template <int FPT>
__global__ void __launch_bounds__(256) k_project_slab_fp64(int lmin, int lmax, int P, int S, int KMAX,
                                                            const int *__restrict__ slab_order,
                                                            const double *__restrict__ q, const double *__restrict__ vl,
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
    const int slab = slab_order[blockIdx.x];
    const int i = lmin + slab;
    const int tid = threadIdx.x;
    const int PP = P * P, L = lmax - lmin + 1, stride = lmax + 1;
    const int par = i & 1;
    for (int s = 0; s < S; s++) {
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
                    c[0] = f[i] * g[j] + f[j] * g[i];  // with h(k)
                    c[1] = f[i] * h[j] + f[j] * h[i];  // with g(k)
                    c[2] = g[i] * h[j] + g[j] * h[i];  // with f(k)
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
            for (int e = tid; e < JC * KMAX; e += 256) {
                int jj = e / KMAX, kk = e - jj * KMAX, j = j0 + jj;
                double val = 0.0;
                if (j <= lmax) {
                    int k = j + par + 2 * kk, k1 = min(i + j, lmax);
                    if (k <= k1)
                        val = Wd[sbase[slab] + tet_row_offset(i, j, lmax) + kk] *
                              (radial ? d_radial_rows(ra, sh.nterms, i, j, k, V + (size_t)jj * 3 * XR, TW)
                               : rowc ? d_sep_rows(sh, tab, stride, k, Cf + (size_t)jj * PJ_TCOEF64 * 3)
                                      : d_shape(sh, tab, stride, i, j, k, ra));
                }
                f[e] = val;
            }
            __syncthreads();
            for (int e = tid; e < JC * P; e += 256) {
                int jj = e / P, c = e - jj * P, j = j0 + jj;
                double acc = 0.0;
                if (j <= lmax) {
                    int kf = j + par, k1 = min(i + j, lmax);
                    int nk = (k1 >= kf) ? (k1 - kf) / 2 + 1 : 0;
                    const double *fr = f + jj * KMAX;
                    const double *qc = q + (size_t)(kf - lmin) * P + c;
                    for (int kk = 0; kk < nk; kk++) acc = fma(fr[kk], qc[(size_t)2 * kk * P], acc);
                }
                H[e] = acc;
            }
            __syncthreads();
#pragma unroll
            for (int t = 0; t < FPT; t++) {
                int e = tid + 256 * t;
                if (e < PP) {
                    int b = e / P, c = e - b * P;
                    double a = 0.0;
                    for (int jj = 0; jj < JC; jj++) {
                        int j = j0 + jj;
                        if (j <= lmax) a = fma(q[(size_t)(j - lmin) * P + b], H[jj * P + c], a);
                    }
                    Facc[t] += a;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int t = 0; t < FPT; t++) {
            int e = tid + 256 * t;
            if (e < PP) Fbuf[((size_t)s * L + slab) * PP + e] = Facc[t];
        }
    }
}

// B[s][a][bc] = sum_slab q[slab][a] Fbuf[s][slab][bc]
__global__ void k_project_B(int L, int P, int S, const double *__restrict__ q, const double *__restrict__ Fbuf,
                            double *__restrict__ B)
{
    const int PP = P * P;
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)S * P * PP) return;
    int s = (int)(e / ((size_t)P * PP));
    int rem = (int)(e - (size_t)s * P * PP);
    int a = rem / PP, bc = rem - a * PP;
    const double *F = Fbuf + (size_t)s * L * PP + bc;
    double acc = 0.0;
    for (int l = 0; l < L; l++) acc = fma(q[(size_t)l * P + a], F[(size_t)l * PP], acc);
    B[e] = acc;
}

// beta[s][r] = (1/6) sum of B over the six orderings of mode r's triple
__global__ void k_project_beta(int N, int P, int S, const int *__restrict__ triples, const double *__restrict__ B,
                               double *__restrict__ beta)
{
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)S * N) return;
    int s = (int)(e / N), r = (int)(e % N);
    int p1 = triples[3 * r], p2 = triples[3 * r + 1], p3 = triples[3 * r + 2];
    const double *b = B + (size_t)s * P * P * P;
#define BB(x, y, z) b[((size_t)(x) * P + (y)) * P + (z)]
    double v = BB(p1, p2, p3) + BB(p2, p3, p1) + BB(p3, p1, p2) + BB(p3, p2, p1) + BB(p2, p1, p3) + BB(p1, p3, p2);
#undef BB
    beta[e] = v / 6e0;
}


// ---------------------------------------------------------------- host side
//
// A projection is planned (shapes validated, every device buffer sized, the
// slab schedule uploaded), its inputs are staged (shape tables and
// descriptors copied to the device), and its device work is recorded on the
// context stream.  The record step allocates nothing and makes no host
// round trip, so modal_project_batch can capture it into a CUDA graph.

modal_status proj_plan(modal_ctx *ctx, int S, const modal_shape *shapes, modal_prec prec, ProjPlan &pl)
{
    const int lmin = ctx->lmin, lmax = ctx->lmax, L = ctx->L, P = ctx->P, N = ctx->N, PP = P * P;
    pl = ProjPlan();
    pl.S = S;
    pl.prec = prec;
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
    {   // FP32 layout (k_pf_tab): per term and factor 16 H8 entries, H8 = groups of 8 lattice points per parity
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
    MODAL_TRY(ensure(ctx->vl, sizeof(double) * (lmax + 1)));
    MODAL_TRY(ensure(ctx->beta, sizeof(double) * (size_t)S * N));
    if (prec == MODAL_PREC_SPLIT) {
        MODAL_TRY(pf_plan(ctx, pl));
    } else {
        // slab schedule: heaviest slabs first
        std::vector<int> order(L);
        std::vector<long long> cnt(L);
        for (int q = 0; q < L; q++) { order[q] = q; cnt[q] = tet_row_offset(lmin + q, lmax + 1, lmax); }
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cnt[a] > cnt[b]; });
        MODAL_TRY(ensure(ctx->slab_order, sizeof(int) * (size_t)L));
        MODAL_CUDA(cudaMemcpyAsync(ctx->slab_order.ptr, order.data(), sizeof(int) * L, cudaMemcpyHostToDevice, ctx->stream));
        const int KMAX = (lmax - lmin) / 2 + 2;
        pl.smem = sizeof(double) * ((size_t)JC * KMAX + (size_t)JC * P + (size_t)JC * PJ_TCOEF64 * 3);
        if (pl.smem > 220 * 1024) { set_error("project: lmax=%d too large for the slab tile", lmax); return MODAL_ERR_ARG; }
        pl.fpt = ceil_div(PP, 256);
        if (pl.fpt > 16) { set_error("project: P=%d too large", P); return MODAL_ERR_ARG; }
        // F partials [S][L][P*P] | B [S][P][P*P] | slab bases [L+1] | weight table [points]
        long long npts = 0;
        for (int i = lmin; i <= lmax; i++) npts += tet_row_offset(i, lmax + 1, lmax);
        pl.npts = npts;
        pl.o_B = sizeof(double) * (size_t)S * L * PP;
        pl.o_sb = pl.o_B + sizeof(double) * (size_t)S * P * PP;
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
    k_vl<<<ceil_div(lmax + 1, 256), 256, 0, ctx->stream>>>(lmax, ctx->cl.as<double>(), ctx->vl.as<double>());
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
        kern<<<L, 256, pl.smem, ctx->stream>>>(lmin, lmax, P, S, KMAX, ctx->slab_order.as<int>(), ctx->q.as<double>(),
                                               ctx->vl.as<double>(), ctx->shape_desc.as<DShape>(),
                                               ctx->shape_tab.as<double>(), Wd, sbase, Fbuf, pl.ra);
        return launched(ctx, "project_slab_fp64");
    };
    if (pl.fpt <= 1) MODAL_TRY(run(k_project_slab_fp64<1>));
    else if (pl.fpt <= 4) MODAL_TRY(run(k_project_slab_fp64<4>));
    else if (pl.fpt <= 8) MODAL_TRY(run(k_project_slab_fp64<8>));
    else MODAL_TRY(run(k_project_slab_fp64<16>));
    k_project_B<<<ceil_div((long)S * P * PP, 256), 256, 0, ctx->stream>>>(L, P, S, ctx->q.as<double>(), Fbuf, B);
    MODAL_TRY(launched(ctx, "project_B"));
    k_project_beta<<<ceil_div((long)S * N, 256), 256, 0, ctx->stream>>>(N, P, S, ctx->triples.as<int>(), B,
                                                                          ctx->beta.as<double>());
    return launched(ctx, "project_beta");
}

modal_status project_dev(modal_ctx *ctx, int S, const modal_shape *shapes, modal_prec prec)
{
    ProjPlan pl;
    MODAL_TRY(proj_plan(ctx, S, shapes, prec, pl));
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

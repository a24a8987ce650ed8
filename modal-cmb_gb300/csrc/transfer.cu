// transfer.cu -- late x primordial transfer Gamma, FP64 on the GPU.
//
// Default path of gamma_mpi.c (calculate_gamma.c):
//   TTweight_l = (2l+1)^{5/6} b_l / sqrt(b_l^2 C_l + N_l)                     (:76-88)
//   M[p][q][x][k] = sum_l P_l(mu_k) TTweight_l q~_p(l,x) q_q(l)                (:254-303)
//   g(m,n,x)      = sum_k w_k perm3(M[p_a][q_b][x][k]), (p) = prim triple of n,
//                   (q) = late triple of m                                       (:512-555)
//   y_x = x^2 g(m,n,x), set to 0 at the first 10 grid points when |y| > 1e-18
//   Gamma_t[m][n] = integrate_cubic_spline(x, y) dphi^2 / (8 pi)                 (:773-934)
// The spline integral is linear in y for fixed nodes: I(y) = sum_x c_x y_x with
// c_x the integral of the spline through the unit vector e_x, computed once on
// the host with the reference's own spline recurrences.  The kernel folds the
// x loop and that weighted sum into one pass per (m, n) tile.
// Device layouts: qt[x][p][l] (l = 0..lmax), mt2[x][k][p][q] (mu-major per x).
#include <algorithm>
#include <cmath>
#include <vector>
#include "common.cuh"
#include "triple.cuh"

namespace modal {

// Integral over [x0, x_{n-1}] of the cubic spline of integrate_cubic_spline
// (calculate_gamma.c:845-934) through (x, y).
static double spline_integral(const double *x, const double *y, int n)
{
    if (n < 2) return 0.0;
    std::vector<double> a(n, 0.0), b(n, 0.0), c(n, 0.0);
    c[0] = x[1] - x[0];
    b[1] = (y[1] - y[0]) / c[0];
    for (int i = 1; i < n - 1; i++) {
        c[i] = x[i + 1] - x[i];
        a[i] = 2.0 * (c[i - 1] + c[i]);
        b[i + 1] = (y[i + 1] - y[i]) / c[i];
        b[i] = b[i + 1] - b[i];
    }
    a[0] = -c[0];
    a[n - 1] = -c[n - 2];
    b[0] = 0.0;
    b[n - 1] = 0.0;
    if (n > 2) {
        b[0] = b[2] / (x[3] - x[1]) - b[1] / (x[2] - x[0]);
        b[n - 1] = b[n - 2] / (x[n - 1] - x[n - 3]) - b[n - 3] / (x[n - 2] - x[n - 4]);
        b[0] = b[0] * c[0] * c[0] / (x[3] - x[0]);
        b[n - 1] = -b[n - 1] * c[n - 2] * c[n - 2] / (x[n - 1] - x[n - 4]);
    }
    for (int i = 1; i < n; i++) {
        double h = c[i - 1] / a[i - 1];
        a[i] -= h * c[i - 1];
        b[i] -= h * b[i - 1];
    }
    b[n - 1] /= a[n - 1];
    for (int i = n - 2; i >= 0; i--) b[i] = (b[i] - c[i] * b[i + 1]) / a[i];
    for (int i = 0; i < n - 1; i++) {
        a[i] = (y[i + 1] - y[i]) / c[i] - c[i] * (b[i + 1] + 2.0 * b[i]);
        c[i] = (b[i + 1] - b[i]) / c[i];
        b[i] = 3.0 * b[i];
    }
    double in = 0.0;
    for (int i = 0; i < n - 1; i++) {
        double d = x[i + 1] - x[i];
        in += d * (y[i] + d * (a[i] / 2.0 + d * (b[i] / 3.0 + d * c[i] / 4.0)));
    }
    return in;
}

// v_l = TTweight_l / (2l+1)^{2/3}: the P_l table on the device carries (2l+1)^{2/3}.
__global__ void k_transfer_weight(int lmax, const double *__restrict__ cl, double *__restrict__ v)
{
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l > lmax) return;
    v[l] = (l > 1) ? pow(2e0 * l + 1e0, 5e0 / 6e0) * (1.0 / sqrt(cl[l])) / pow(2e0 * l + 1e0, 2e0 / 3e0) : 0e0;
}

// mt2[x][k][p][q] = sum_l pl[l][k] v_l qt[x][p][l] q[l-lmin][q]; tile 64 mu x 32 (p,q), l ascending.
constexpr int TR_BK = 64, TR_BU = 32, TR_LC = 16;

// With v2/qt2 (polarised E side): the transfer factor is v_l qt - v2_l qt2.
// qt and qt2 rows have stride qstride (lmax_T + 1).
// FOLD: antisymmetric nodes, even and odd l summed apart at the first half of the nodes (as mij_tile).
template <bool FOLD>
__global__ void __launch_bounds__(256) k_mij_transfer(int nmu, int lmin, int lmax, int P, int Pp,
                                                      const double *__restrict__ pl, const double *__restrict__ q,
                                                      const double *__restrict__ v, const double *__restrict__ qt,
                                                      double *__restrict__ mt2, const double *__restrict__ v2,
                                                      const double *__restrict__ qt2, int qstride)
{
    constexpr int NA = FOLD ? 2 : 1;
    __shared__ double sPl[TR_LC][TR_BK];
    __shared__ double sV[TR_LC][TR_BU];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int k0 = blockIdx.x * TR_BK, u0 = blockIdx.y * TR_BU, xi = blockIdx.z;
    const int L = lmax - lmin + 1, nu = Pp * P, nk = FOLD ? (nmu + 1) / 2 : nmu;
    const double *qtx = qt + (size_t)xi * Pp * qstride;
    const double *qtx2 = qt2 ? qt2 + (size_t)xi * Pp * qstride : nullptr;
    double acc[NA][8];
#pragma unroll
    for (int r = 0; r < 8; r++) acc[0][r] = acc[NA - 1][r] = 0.0;
    for (int l0 = 0; l0 < L; l0 += TR_LC) {
#pragma unroll
        for (int t = 0; t < (TR_LC * TR_BK) / 256; t++) {
            int e = tid + 256 * t, lr = e / TR_BK, kc = e % TR_BK;
            int l = l0 + lr, k = k0 + kc;
            sPl[lr][kc] = (l < L && k < nk) ? pl[(size_t)(lmin + l) * nmu + k] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < (TR_LC * TR_BU) / 256; t++) {
            int e = tid + 256 * t, lr = e / TR_BU, uc = e % TR_BU;
            int l = l0 + lr, u = u0 + uc;
            double val = 0.0;
            if (l < L && u < nu) {
                int p = u / P, qq = u - p * P;
                double t = v[lmin + l] * qtx[(size_t)p * qstride + lmin + l];
                if (qtx2) t -= v2[lmin + l] * qtx2[(size_t)p * qstride + lmin + l];
                val = t * q[(size_t)l * P + qq];
            }
            sV[lr][uc] = val;
        }
        __syncthreads();
#pragma unroll
        for (int lr = 0; lr < TR_LC; lr++) {
            double vv = sV[lr][tx];
#pragma unroll
            for (int r = 0; r < 8; r++) acc[lr & (NA - 1)][r] = fma(sPl[lr][ty + 8 * r], vv, acc[lr & (NA - 1)][r]);
        }
        __syncthreads();
    }
    const int u = u0 + tx;
    if (u >= nu) return;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int k = k0 + ty + 8 * r;
        if (k >= nk) continue;
        const double E = acc[(lmin & 1) ? NA - 1 : 0][r], O = FOLD ? acc[(lmin & 1) ? 0 : NA - 1][r] : 0.0;
        mt2[((size_t)xi * nmu + k) * nu + u] = FOLD ? E + O : acc[0][r];
        if (FOLD && nmu - 1 - k != k) mt2[((size_t)xi * nmu + nmu - 1 - k) * nu + u] = E - O;
    }
}

// One CTA per 32 (n: primordial) x 32 (m: late) tile; thread (tx, ty) owns
// n = n0 + tx and m = m0 + ty + 8 r.
// blockIdx.z takes the radial samples [z xs, min(xsize, (z + 1) xs)); its partial
// sum goes to out + z N Nprim (k_sum_groups adds the groups in a fixed order).
__global__ void __launch_bounds__(256) k_gamma_transfer(int N, int Nprim, int P, int Pp, int nmu, int xsize, int xs, int KC,
                                                        const int *__restrict__ triples, const int *__restrict__ prim,
                                                        const double *__restrict__ mt2, const double *__restrict__ w,
                                                        const double *__restrict__ xvec, const double *__restrict__ cx,
                                                        double scale, double *__restrict__ out)
{
    extern __shared__ double smt[];
    double *sW = smt;        // [KC]
    double *sA = smt + KC;   // [KC][Pp*P]
    const int nu = Pp * P;
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int n = blockIdx.x * 32 + tx;
    int po[3] = {0, 0, 0};
    if (n < Nprim) { po[0] = prim[3 * n] * P; po[1] = prim[3 * n + 1] * P; po[2] = prim[3 * n + 2] * P; }
    int qm[4][3];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = blockIdx.y * 32 + ty + 8 * r;
        for (int b = 0; b < 3; b++) qm[r][b] = (m < N) ? triples[3 * m + b] : 0;
    }
    double res[4] = {0.0, 0.0, 0.0, 0.0};
    const int xb = blockIdx.z * xs, xe = min(xsize, xb + xs);
    out += (size_t)blockIdx.z * N * Nprim;
    for (int xi = xb; xi < xe; xi++) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        const double *src0 = mt2 + (size_t)xi * nmu * nu;
        for (int k0 = 0; k0 < nmu; k0 += KC) {
            const int kc = min(KC, nmu - k0);
            const double *src = src0 + (size_t)k0 * nu;
            for (int e = tid; e < kc * nu; e += 256) sA[e] = src[e];
            if (tid < kc) sW[tid] = w[k0 + tid];
            __syncthreads();
            for (int kk = 0; kk < kc; kk++) {
                const double *A = sA + kk * nu;
                const double wk = sW[kk];
                const double *r1 = A + po[0], *r2 = A + po[1], *r3 = A + po[2];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    double a11 = r1[qm[r][0]], a12 = r1[qm[r][1]], a13 = r1[qm[r][2]];
                    double a21 = r2[qm[r][0]], a22 = r2[qm[r][1]], a23 = r2[qm[r][2]];
                    double a31 = r3[qm[r][0]], a32 = r3[qm[r][1]], a33 = r3[qm[r][2]];
                    double t1 = fma(a23, a32, a22 * a33);
                    double t2 = fma(a23, a31, a21 * a33);
                    double t3 = fma(a22, a31, a21 * a32);
                    acc[r] = fma(wk, fma(a13, t3, fma(a12, t2, a11 * t1)), acc[r]);
                }
            }
            __syncthreads();
        }
        const double x2 = xvec[xi] * xvec[xi], c = cx[xi];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            double y = x2 * acc[r];
            if (xi < 10 && fabs(y) > 1e-18) y = 0.0;  // calculate_gamma.c:803-804
            res[r] = fma(c, y, res[r]);
        }
    }
    if (n >= Nprim) return;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = blockIdx.y * 32 + ty + 8 * r;
        if (m < N) out[(size_t)m * Nprim + n] = res[r] * scale;
    }
}

// out[e] = sum over the G groups of out[g stride + e], g ascending (in place).
__global__ void k_sum_groups(long n, int G, long stride, double *__restrict__ out)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    double s = out[e];
    for (int g = 1; g < G; g++) s += out[(size_t)g * stride + e];
    out[e] = s;
}

// The transfer Gamma from the distinct products of three M entries (triple.cu, U = Pp P entries per
// node and radial sample).  The spline integral is linear, so the samples x >= 10 form one sum over
// (x, k) with weights c_x x^2 w_k, T_sum; each of the first ten keeps its own T_x, because the reference
// drops y_x there when |y_x| > 1e-18 (calculate_gamma.c:803-804).
// w2[xi nmu + k] = x^2 w_k for the first nx samples, c_x x^2 w_k beyond
__global__ void k_transfer_node_weights(int nmu, int xsize, int nx, const double *__restrict__ w,
                                        const double *__restrict__ xvec, const double *__restrict__ cx,
                                        double *__restrict__ w2)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)nmu * xsize) return;
    const int xi = (int)(e / nmu), k = (int)(e - (long)xi * nmu);
    const double x2 = xvec[xi] * xvec[xi];
    w2[e] = (xi < nx ? x2 : cx[xi] * x2) * w[k];
}

// y_x of one (m, n), summed as k_gamma_transfer sums it: a pair's permanent per node, nodes in order.
// p: P times the primordial triple, q: the late triple, A: the sample's [nmu][nu] table.
__device__ __noinline__ double transfer_sample(int nmu, int nu, const int *p, const int *q, const double *__restrict__ A,
                                               const double *__restrict__ w)
{
    double acc = 0.0;
    for (int k = 0; k < nmu; k++, A += nu) {
        const double *r1 = A + p[0], *r2 = A + p[1], *r3 = A + p[2];
        const double a21 = r2[q[0]], a22 = r2[q[1]], a23 = r2[q[2]], a31 = r3[q[0]], a32 = r3[q[1]], a33 = r3[q[2]];
        const double t1 = fma(a23, a32, a22 * a33), t2 = fma(a23, a31, a21 * a33), t3 = fma(a22, a31, a21 * a32);
        acc = fma(w[k], fma(r1[q[2]], t3, fma(r1[q[1]], t2, r1[q[0]] * t1)), acc);
    }
    return acc;
}

// out[m][n]: six entries of T_sum and, one x at a time, of the first nx tables with the zero rule, which
// within 1e-6 (relative) of its threshold goes by the sum of the permanents: both routes then drop the same
// samples.  T: [nx] tables of the first samples, then T_sum (if last), zstride apart.
__global__ void __launch_bounds__(256) k_transfer_gather(int N, int Nprim, int P, int U, long ldT, int nx, int last, size_t zstride,
                                                         const int *__restrict__ triples, const int *__restrict__ prim,
                                                         const double *__restrict__ cx, const double *__restrict__ T,
                                                         int nmu, const double *__restrict__ mt2, const double *__restrict__ w,
                                                         const double *__restrict__ xvec, double scale,
                                                         double *__restrict__ out)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)N * Nprim) return;
    const int m = (int)(e / Nprim), n = (int)(e - (long)m * Nprim);
    const int q[3] = {triples[3 * m], triples[3 * m + 1], triples[3 * m + 2]};
    const int p[3] = {prim[3 * n] * P, prim[3 * n + 1] * P, prim[3 * n + 2] * P};
    const int perm[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}, {1, 0, 2}, {0, 2, 1}};
    size_t at[6];
#pragma unroll
    for (int s = 0; s < 6; s++) at[s] = triple_at(p[0] + q[perm[s][0]], p[1] + q[perm[s][1]], p[2] + q[perm[s][2]], U, ldT);
    double res = 0.0;
    for (int x = 0; x < nx; x++) {
        double y = 0.0;
#pragma unroll
        for (int s = 0; s < 6; s++) y += T[x * zstride + at[s]];
        if (fabs(fabs(y) - 1e-18) <= 1e-24)
            y = xvec[x] * xvec[x] * transfer_sample(nmu, U, p, q, mt2 + (size_t)x * nmu * U, w);
        if (fabs(y) > 1e-18) y = 0.0;
        res = fma(cx[x], y, res);
    }
    if (last) {
        double y = 0.0;
#pragma unroll
        for (int s = 0; s < 6; s++) y += T[(size_t)nx * zstride + at[s]];
        res += y;
    }
    out[e] = res * scale;
}

// Polarised points (gamma_2d_pt_TTE/TEE/EEE, calculate_gamma.c:558-687): the
// 3x3 block has rows = primordial legs and columns = late legs, column b taken
// from the T table (b < nT: FORM 1 TTE nT = 2, FORM 2 TEE nT = 1) or the E
// table (FORM 3 EEE: all E); its permanent, weighted, summed over mu.
template <int FORM>
__global__ void __launch_bounds__(256) k_gamma_transfer_pol(int N, int Nprim, int P, int PE, int Pp, int nmu,
                                                            int xsize, int xs, long gstride, int KC,
                                                            const int *__restrict__ triples,
                                                            const int *__restrict__ prim,
                                                            const double *__restrict__ mtT,
                                                            const double *__restrict__ mtE,
                                                            const double *__restrict__ w,
                                                            const double *__restrict__ xvec,
                                                            const double *__restrict__ cx, double scale,
                                                            double *__restrict__ out)
{
    constexpr int nT = (FORM == 1) ? 2 : (FORM == 2 ? 1 : 0);
    extern __shared__ double smt[];
    const int nuT = (nT > 0) ? Pp * P : 0, nuE = Pp * PE;
    double *sW = smt;               // [KC]
    double *sT = smt + KC;          // [KC][Pp*P]
    double *sE = sT + KC * nuT;     // [KC][Pp*PE]
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int n = blockIdx.x * 32 + tx;
    int pa[3] = {0, 0, 0};
    if (n < Nprim) { pa[0] = prim[3 * n]; pa[1] = prim[3 * n + 1]; pa[2] = prim[3 * n + 2]; }
    int qm[4][3];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = blockIdx.y * 32 + ty + 8 * r;
        for (int b = 0; b < 3; b++) qm[r][b] = (m < N) ? triples[3 * m + b] : 0;
    }
    double res[4] = {0.0, 0.0, 0.0, 0.0};
    const int xb = blockIdx.z * xs, xe = min(xsize, xb + xs);  // this CTA's radial samples (as k_gamma_transfer)
    out += (size_t)blockIdx.z * gstride;
    for (int xi = xb; xi < xe; xi++) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k0 = 0; k0 < nmu; k0 += KC) {
            const int kc = min(KC, nmu - k0);
            if (nT > 0)
                for (int e = tid; e < kc * nuT; e += 256) sT[e] = mtT[((size_t)xi * nmu + k0) * nuT + e];
            for (int e = tid; e < kc * nuE; e += 256) sE[e] = mtE[((size_t)xi * nmu + k0) * nuE + e];
            if (tid < kc) sW[tid] = w[k0 + tid];
            __syncthreads();
            for (int kk = 0; kk < kc; kk++) {
                const double *T = sT + kk * nuT, *E = sE + kk * nuE;
                const double wk = sW[kk];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    double a[3][3];
#pragma unroll
                    for (int x = 0; x < 3; x++)
#pragma unroll
                        for (int b = 0; b < 3; b++)
                            a[x][b] = (b < nT) ? T[pa[x] * P + qm[r][b]] : E[pa[x] * PE + qm[r][b]];
                    const double t1 = fma(a[1][2], a[2][1], a[1][1] * a[2][2]);
                    const double t2 = fma(a[1][2], a[2][0], a[1][0] * a[2][2]);
                    const double t3 = fma(a[1][1], a[2][0], a[1][0] * a[2][1]);
                    acc[r] = fma(wk, fma(a[0][2], t3, fma(a[0][1], t2, a[0][0] * t1)), acc[r]);
                }
            }
            __syncthreads();
        }
        const double x2 = xvec[xi] * xvec[xi], c = cx[xi];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            double y = x2 * acc[r];
            if (xi < 10 && fabs(y) > 1e-18) y = 0.0;  // calculate_gamma.c:803-804 (and :812-826)
            res[r] = fma(c, y, res[r]);
        }
    }
    if (n >= Nprim) return;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = blockIdx.y * 32 + ty + 8 * r;
        if (m < N) out[(size_t)m * Nprim + n] = res[r] * scale;
    }
}

}  // namespace modal

using namespace modal;

// mt2 of the late basis q on lmin..lmax; the transfer factor is v qt, or v qt - v2 qt2.
static modal_status mij_transfer_dev(modal_ctx *c, int lmin, int lmax, int P, const double *q, const double *v,
                                     const double *qt, double *mt2, const double *v2, const double *qt2)
{
    const int nu = c->tr_Pp * P, nk = c->gl_sym ? (c->nmu + 1) / 2 : c->nmu;
    const dim3 g(ceil_div(nk, TR_BK), ceil_div(nu, TR_BU), c->tr_xsize);
    auto run = [&](auto kern) {
        kern<<<g, 256, 0, c->stream>>>(c->nmu, lmin, lmax, P, c->tr_Pp, c->pl.as<double>(), q, v, qt, mt2, v2, qt2, c->lmax + 1);
    };
    if (c->gl_sym) run(k_mij_transfer<true>);
    else run(k_mij_transfer<false>);
    return launched(c, "mij_transfer");
}

// tr_out[N][Nprim] from the distinct products.
static modal_status transfer_triple_dev(modal_ctx *c, double scale)
{
    const int xsize = c->tr_xsize, nmu = c->nmu, U = c->tr_Pp * c->P, N = c->N, Nprim = c->tr_Nprim;
    const int nx = std::min(10, xsize), K2 = (xsize - nx) * nmu;
    const size_t UV = (size_t)U * (U + 1) / 2, n = U * UV;
    const int kper = K2 > 0 ? ceil_div(K2, triple_splits(c, U, K2)) : 1, Zn = K2 > 0 ? ceil_div(K2, kper) : 0;
    const long K = (long)xsize * nmu;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t oz = al(sizeof(double) * K * U), ow = 2 * oz, ot = ow + al(sizeof(double) * K);
    MODAL_TRY(ensure(c->trip, ot + sizeof(double) * (nx + Zn) * n));
    uint8_t *b = c->trip.as<uint8_t>();
    double *X = reinterpret_cast<double *>(b), *Z = reinterpret_cast<double *>(b + oz), *w2 = reinterpret_cast<double *>(b + ow),
           *T = reinterpret_cast<double *>(b + ot);
    const double *cx = c->tr_x.as<double>() + xsize;
    k_transfer_node_weights<<<ceil_div(K, 256), 256, 0, c->stream>>>(nmu, xsize, nx, c->w.as<double>(), c->tr_x.as<double>(), cx, w2);
    MODAL_TRY(launched(c, "transfer_node_weights"));
    MODAL_TRY(triple_rows_dev(c, K, U, 0, c->tr_mt.as<double>(), U, w2, X, Z));
    MODAL_TRY(triple_dev(c, U, nx * nmu, nmu, X, Z, T, n));
    if (K2 > 0) {
        const size_t o = (size_t)nx * nmu * U;
        MODAL_TRY(triple_dev(c, U, K2, kper, X + o, Z + o, T + nx * n, n));
        MODAL_TRY(triple_sum_dev(c, n, Zn, n, T + nx * n));
    }
    k_transfer_gather<<<ceil_div((long)N * Nprim, 256), 256, 0, c->stream>>>(
        N, Nprim, c->P, U, (long)UV, nx, K2 > 0, n, c->triples.as<int>(), c->tr_prim.as<int>(), cx, T, nmu,
        c->tr_mt.as<double>(), c->w.as<double>(), c->tr_x.as<double>(), scale, c->tr_out.as<double>());
    return launched(c, "transfer_gather");
}

extern "C" modal_status modal_set_transfer(modal_ctx *c, int Pp, int xsize, const double *xvec, const double *qtilde,
                                           int Nprim, const int *prim)
{
    if (!c || !c->have_basis) { set_error("modal_set_transfer: set the basis first"); return MODAL_ERR_STATE; }
    if (Pp < 1 || Pp > 64 || xsize < 4 || Nprim < 1 || !xvec || !qtilde || !prim) {
        set_error("modal_set_transfer: Pp=%d xsize=%d (>= 4 points) Nprim=%d", Pp, xsize, Nprim);
        return MODAL_ERR_ARG;
    }
    for (long e = 0; e < 3L * Nprim; e++)
        if (prim[e] < 0 || prim[e] >= Pp) { set_error("modal_set_transfer: primordial mode index %d outside [0,%d)", prim[e], Pp); return MODAL_ERR_ARG; }
    for (int i = 1; i < xsize; i++)
        if (!(xvec[i] > xvec[i - 1])) { set_error("modal_set_transfer: x grid must increase"); return MODAL_ERR_ARG; }
    MODAL_CUDA(cudaSetDevice(c->device));
    // spline weights c_x = integral of the reference spline through e_x
    std::vector<double> cx(xsize), e(xsize, 0.0);
    for (int i = 0; i < xsize; i++) {
        e[i] = 1.0;
        cx[i] = spline_integral(xvec, e.data(), xsize);
        e[i] = 0.0;
    }
    const size_t nq = (size_t)xsize * Pp * (c->lmax + 1);
    MODAL_TRY(ensure(c->tr_x, sizeof(double) * 2 * xsize));
    MODAL_TRY(ensure(c->tr_qt, sizeof(double) * nq));
    MODAL_TRY(ensure(c->tr_prim, sizeof(int) * 3 * (size_t)Nprim));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_x.ptr, xvec, sizeof(double) * xsize, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_x.as<double>() + xsize, cx.data(), sizeof(double) * xsize, cudaMemcpyHostToDevice,
                               c->stream));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_qt.ptr, qtilde, sizeof(double) * nq, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_prim.ptr, prim, sizeof(int) * 3 * Nprim, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaStreamSynchronize(c->stream));
    c->tr_Pp = Pp;
    c->tr_xsize = xsize;
    c->tr_Nprim = Nprim;
    return MODAL_OK;
}

extern "C" modal_status modal_gamma_transfer(modal_ctx *c, double deltaphi, double *gamma_t)
{
    if (!c || !c->have_modes || !c->have_spec || c->tr_xsize < 4) {
        set_error("modal_gamma_transfer: set basis, modes, spectrum and transfer functions first");
        return MODAL_ERR_STATE;
    }
    MODAL_CUDA(cudaSetDevice(c->device));
    if (!c->have_glint) MODAL_TRY(modal_init_glint(c));
    const int P = c->P, Pp = c->tr_Pp, xsize = c->tr_xsize, nmu = c->nmu, N = c->N, Nprim = c->tr_Nprim;
    const int nu = Pp * P;
    MODAL_TRY(ensure(c->tr_mt, sizeof(double) * (size_t)xsize * nmu * nu));
    MODAL_TRY(ensure(c->tr_v, sizeof(double) * (c->lmax + 1)));
    MODAL_TRY(ensure(c->tr_out, sizeof(double) * (size_t)N * Nprim));
    StageTimer t(c, MODAL_T_GAMMA);
    k_transfer_weight<<<ceil_div(c->lmax + 1, 256), 256, 0, c->stream>>>(c->lmax, c->cl.as<double>(), c->tr_v.as<double>());
    MODAL_TRY(launched(c, "transfer_weight"));
    MODAL_TRY(mij_transfer_dev(c, c->lmin, c->lmax, P, c->q.as<double>(), c->tr_v.as<double>(), c->tr_qt.as<double>(),
                               c->tr_mt.as<double>(), nullptr, nullptr));
    const double scale = deltaphi * deltaphi / (8.0 * 3.14159265358979323846);
    auto finish = [&]() -> modal_status {
        t.stop();
        if (gamma_t)
            MODAL_CUDA(cudaMemcpyAsync(gamma_t, c->tr_out.ptr, sizeof(double) * (size_t)N * Nprim, cudaMemcpyDeviceToHost,
                                       c->stream));
        MODAL_CUDA(cudaStreamSynchronize(c->stream));
        return MODAL_OK;
    };
    int KC = (96 * 1024) / (nu * 8);
    if (KC < 1) KC = 1;
    if (KC > 32) KC = 32;
    const size_t smem = sizeof(double) * ((size_t)KC + (size_t)KC * nu);
    if (smem > 200 * 1024) { set_error("modal_gamma_transfer: Pp*P=%d too large for the tile", nu); return MODAL_ERR_ARG; }
    // the distinct products, or (few modes) the permanents of the pairs: 816 x 120 modes at P = 16, Pp = 8,
    // 32 samples and l <= 600 take 24 ms on the first, 55 ms on the second.  Up to eleven and a few more
    // tables of 8 U^2 (U+1) / 2 bytes: at most 16 GB
    if (triple_wins((double)N * Nprim, nu) && 4.0 * nu * nu * (nu + 1.0) * 42 <= 16e9 &&
        (double)xsize * nmu * nu < 2e9) {
        const modal_status st = transfer_triple_dev(c, scale);
        if (st == MODAL_OK) return finish();
        if (st != MODAL_ERR_NOMEM) return st;
    }
    MODAL_CUDA(cudaFuncSetAttribute(k_gamma_transfer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // the (primordial x late) tiles alone fill about two thirds of the SMs at the
    // benchmark sizes: split the radial samples into groups so that the grid holds
    // about 16 CTAs per SM (measured: 4 -> 67 ms, 8 -> 59 ms, 16 -> 57 ms at l <= 600),
    // and add the groups' partial sums afterwards
    int nsm = 0;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    const long tiles = (long)ceil_div(Nprim, 32) * ceil_div(N, 32);
    int XG = (int)std::min<long>(xsize, std::max<long>(1, (16L * nsm + tiles - 1) / tiles));
    const int xs = ceil_div(xsize, XG);
    XG = ceil_div(xsize, xs);
    MODAL_TRY(ensure(c->tr_out, sizeof(double) * (size_t)XG * N * Nprim));
    dim3 gg(ceil_div(Nprim, 32), ceil_div(N, 32), XG);
    k_gamma_transfer<<<gg, 256, smem, c->stream>>>(N, Nprim, P, Pp, nmu, xsize, xs, KC, c->triples.as<int>(),
                                                   c->tr_prim.as<int>(), c->tr_mt.as<double>(), c->w.as<double>(),
                                                   c->tr_x.as<double>(), c->tr_x.as<double>() + xsize, scale,
                                                   c->tr_out.as<double>());
    MODAL_TRY(launched(c, "gamma_transfer"));
    if (XG > 1) {
        const long n = (long)N * Nprim;
        k_sum_groups<<<ceil_div(n, 256), 256, 0, c->stream>>>(n, XG, n, c->tr_out.as<double>());
        MODAL_TRY(launched(c, "sum_groups"));
    }
    return finish();
}

// E-side weights of calculate_gamma.c:142-183 on the host, divided by the
// (2l+1)^{2/3} the device P_l table carries:
//   EEweight_l = (2l+1)^{5/6} b_E / sqrt(s_TT (s_TT s_EE - s_TE^2))
//   wq_l = EEweight_l s_TT,  wl_l = EEweight_l (sqrt(fE/fT) b_TE^2 C_TE + N_TE)
// so that the effective E transfer function is wq_l q~_E - wl_l q~_T.
extern "C" modal_status modal_set_transfer_pol(modal_ctx *c, const double *qtilde_e, const modal_pol_spectra *sp)
{
    if (!c || !qtilde_e || !sp) { set_error("modal_set_transfer_pol: NULL argument"); return MODAL_ERR_ARG; }
    if (c->tr_xsize < 4 || !c->have_pol) {
        set_error("modal_set_transfer_pol: call modal_set_transfer, modal_set_basis_e and modal_set_modes_pol first");
        return MODAL_ERR_STATE;
    }
    if (c->lmax_e > c->lmax) {
        set_error("modal_set_transfer_pol: lmax_E=%d must not exceed lmax_T=%d", c->lmax_e, c->lmax);
        return MODAL_ERR_ARG;
    }
    const double *arr[9] = {sp->cl_tt, sp->cl_te, sp->cl_ee, sp->beam_tt, sp->beam_te, sp->beam_ee,
                            sp->noise_tt, sp->noise_te, sp->noise_ee};
    for (const double *a : arr)
        if (!a) { set_error("modal_set_transfer_pol: a spectrum array is NULL"); return MODAL_ERR_ARG; }
    if (!(sp->fsky_t > 0.0) || !(sp->fsky_e > 0.0)) { set_error("modal_set_transfer_pol: fsky must be > 0"); return MODAL_ERR_ARG; }
    const int lmax = c->lmax;
    std::vector<double> wq(lmax + 1, 0.0), wl(lmax + 1, 0.0);
    for (int l = std::max(c->lmin_e, 2); l <= c->lmax_e; l++) {
        const double s2 = sp->beam_tt[l] * sp->beam_tt[l] * sp->cl_tt[l] + sp->noise_tt[l];
        const double s3 = sp->beam_tt[l] * sp->beam_ee[l] * sp->cl_te[l] + sp->noise_te[l];
        const double s4 = sp->beam_ee[l] * sp->beam_ee[l] * sp->cl_ee[l] + sp->noise_ee[l];
        const double den = s2 * (s2 * s4 - s3 * s3);
        if (!(den > 0.0)) { set_error("modal_set_transfer_pol: TT/TE/EE covariance not positive at l=%d", l); return MODAL_ERR_ARG; }
        const double eew = std::pow(2.0 * l + 1.0, 5.0 / 6.0) * (sp->beam_ee[l] / std::sqrt(den));
        const double lk = std::sqrt(sp->fsky_e / sp->fsky_t) * sp->beam_te[l] * sp->beam_te[l] * sp->cl_te[l] + sp->noise_te[l];
        const double f = std::pow(2.0 * l + 1.0, 2.0 / 3.0);
        wq[l] = eew * s2 / f;
        wl[l] = eew * lk / f;
    }
    MODAL_CUDA(cudaSetDevice(c->device));
    const size_t nq = (size_t)c->tr_xsize * c->tr_Pp * (lmax + 1);
    MODAL_TRY(ensure(c->tr_qte, sizeof(double) * nq));
    MODAL_TRY(ensure(c->tr_we, sizeof(double) * 2 * (lmax + 1)));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_qte.ptr, qtilde_e, sizeof(double) * nq, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_we.ptr, wq.data(), sizeof(double) * (lmax + 1), cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(c->tr_we.as<double>() + (lmax + 1), wl.data(), sizeof(double) * (lmax + 1),
                               cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaStreamSynchronize(c->stream));
    c->tr_pol = true;
    return MODAL_OK;
}

extern "C" modal_status modal_gamma_transfer_pol(modal_ctx *c, double deltaphi, double *gamma_tte, double *gamma_tee,
                                                 double *gamma_eee)
{
    if (!c || !c->have_modes || !c->have_spec || c->tr_xsize < 4 || !c->tr_pol || !c->have_pol) {
        set_error("modal_gamma_transfer_pol: set basis, modes, spectrum, transfer functions and their E side first");
        return MODAL_ERR_STATE;
    }
    MODAL_CUDA(cudaSetDevice(c->device));
    if (!c->have_glint) MODAL_TRY(modal_init_glint(c));
    const int P = c->P, PE = c->P_e, Pp = c->tr_Pp, xsize = c->tr_xsize, nmu = c->nmu, N = c->N, Nprim = c->tr_Nprim;
    const int nuT = Pp * P, nuE = Pp * PE;
    const size_t NP = (size_t)N * Nprim;
    MODAL_TRY(ensure(c->tr_mt, sizeof(double) * (size_t)xsize * nmu * nuT));
    MODAL_TRY(ensure(c->tr_mte, sizeof(double) * (size_t)xsize * nmu * nuE));
    MODAL_TRY(ensure(c->tr_v, sizeof(double) * (c->lmax + 1)));
    MODAL_TRY(ensure(c->tr_out, sizeof(double) * 3 * NP));
    const size_t per_mu = (size_t)nuT + nuE;
    const int KC = (int)std::max<size_t>(1, std::min<size_t>(32, (96 * 1024) / (per_mu * 8 + 8)));
    const size_t smem = sizeof(double) * ((size_t)KC + (size_t)KC * per_mu);
    if (smem > 200 * 1024) { set_error("modal_gamma_transfer_pol: Pp*(P+P_E)=%zu too large for the tile", per_mu); return MODAL_ERR_ARG; }
    StageTimer t(c, MODAL_T_GAMMA);
    k_transfer_weight<<<ceil_div(c->lmax + 1, 256), 256, 0, c->stream>>>(c->lmax, c->cl.as<double>(), c->tr_v.as<double>());
    MODAL_TRY(launched(c, "transfer_weight"));
    MODAL_TRY(mij_transfer_dev(c, c->lmin, c->lmax, P, c->q.as<double>(), c->tr_v.as<double>(), c->tr_qt.as<double>(),
                               c->tr_mt.as<double>(), nullptr, nullptr));
    const double *wq = c->tr_we.as<double>(), *wl = wq + (c->lmax + 1);
    MODAL_TRY(mij_transfer_dev(c, c->lmin_e, c->lmax_e, PE, c->qe.as<double>(), wq, c->tr_qte.as<double>(),
                               c->tr_mte.as<double>(), wl, c->tr_qt.as<double>()));
    int nsm = 0;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    const long tiles = (long)ceil_div(Nprim, 32) * ceil_div(N, 32);
    int XG = (int)std::min<long>(xsize, std::max<long>(1, (16L * nsm + tiles - 1) / tiles));
    const int xs = ceil_div(xsize, XG);
    XG = ceil_div(xsize, xs);
    MODAL_TRY(ensure(c->tr_out, sizeof(double) * 3 * (size_t)XG * NP));  // group g of form f at (3 g + f) NP
    dim3 gg(ceil_div(Nprim, 32), ceil_div(N, 32), XG);
    const double scale = deltaphi * deltaphi / (8.0 * 3.14159265358979323846);
    auto run = [&](auto kern, int f) -> modal_status {
        MODAL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<gg, 256, smem, c->stream>>>(N, Nprim, P, PE, Pp, nmu, xsize, xs, 3 * (long)NP, KC,
                                           c->tri_pol.as<int>() + 3 * (size_t)N * f,
                                           c->tr_prim.as<int>(), c->tr_mt.as<double>(), c->tr_mte.as<double>(),
                                           c->w.as<double>(), c->tr_x.as<double>(), c->tr_x.as<double>() + xsize, scale,
                                           c->tr_out.as<double>() + f * NP);
        MODAL_TRY(launched(c, "gamma_transfer_pol"));
        if (XG > 1) {
            k_sum_groups<<<ceil_div((long)NP, 256), 256, 0, c->stream>>>((long)NP, XG, 3 * (long)NP,
                                                                          c->tr_out.as<double>() + f * NP);
            MODAL_TRY(launched(c, "sum_groups"));
        }
        return MODAL_OK;
    };
    MODAL_TRY(run(k_gamma_transfer_pol<1>, 0));
    MODAL_TRY(run(k_gamma_transfer_pol<2>, 1));
    MODAL_TRY(run(k_gamma_transfer_pol<3>, 2));
    t.stop();
    double *outs[3] = {gamma_tte, gamma_tee, gamma_eee};
    for (int f = 0; f < 3; f++)
        if (outs[f])
            MODAL_CUDA(cudaMemcpyAsync(outs[f], c->tr_out.as<double>() + f * NP, sizeof(double) * NP,
                                       cudaMemcpyDeviceToHost, c->stream));
    MODAL_CUDA(cudaStreamSynchronize(c->stream));
    return MODAL_OK;
}

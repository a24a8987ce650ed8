// gamma_fp64.cu -- plain FP64 form of the two contractions that build Gamma.
//
//  l-contraction (calculate_orthoMij_T, orthogonalisation_late.c:99-129):
//     M[i][j][k] = sum_{l=lmin}^{lmax} gl_Pl[k][l] q_i(l) q_j(l)
//  mu-contraction (calculate_orthol, orthogonalisation_late.c:239-336):
//     Gamma_mn = sum_k w_k/(48 pi) * sum of the six products
//                M[m_a][n_s(a)][k] over the permutations s of (0,1,2),
//  i.e. w_k/(48 pi) times the permanent of the 3x3 block of M(k) with rows
//  (m1,m2,m3) and columns (n1,n2,n3).  Device layouts: pl[l][k] (l-major),
//  mt[k][i][j] (mu-major, so one mu step of the whole P x P table is one
//  contiguous block).
#include "common.cuh"
#include "triple.cuh"

namespace modal {

// --------------------------------------------------------------------------
// l-contraction, FP64 SIMT GEMM over l: out tile 8R (mu) x 32 (p<=q pairs), bound by the FP64 pipe
// (the tile's loads hide behind it).  FOLD: the quadrature is antisymmetric, so with
// P_l(-x) = (-1)^l P_l(x) (exact in the table) the sums over even and over odd l at the first half of
// the nodes give both halves, E + O and E - O, at half the FMAs; else the sum over l in ascending
// order, as the reference.
// --------------------------------------------------------------------------
constexpr int MIJ_BU = 32, MIJ_LC = 16;

template <int R, bool FOLD>
__device__ __forceinline__ void mij_tile(int nmu, int lmin, int lmax, int P, int npair, const double *__restrict__ pl,
                                         const double *__restrict__ q, const int2 *__restrict__ pairs,
                                         double *__restrict__ mt)
{
    constexpr int MIJ_BK = 8 * R, NA = FOLD ? 2 : 1;
    __shared__ double sPl[MIJ_LC][MIJ_BK];
    __shared__ double sV[MIJ_LC][MIJ_BU];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int k0 = blockIdx.x * MIJ_BK, u0 = blockIdx.y * MIJ_BU, nk = FOLD ? (nmu + 1) / 2 : nmu;
    const int L = lmax - lmin + 1;
    double acc[NA][R];
#pragma unroll
    for (int p = 0; p < NA; p++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[p][r] = 0.0;

    for (int l0 = 0; l0 < L; l0 += MIJ_LC) {
#pragma unroll
        for (int t = 0; t < (MIJ_LC * MIJ_BK + 255) / 256; t++) {
            int e = tid + 256 * t;
            if (e >= MIJ_LC * MIJ_BK) break;
            int lr = e / MIJ_BK, kc = e % MIJ_BK;
            int l = l0 + lr, k = k0 + kc;
            sPl[lr][kc] = (l < L && k < nk) ? pl[(size_t)(lmin + l) * nmu + k] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < (MIJ_LC * MIJ_BU) / 256; t++) {
            int e = tid + 256 * t, lr = e / MIJ_BU, uc = e % MIJ_BU;
            int l = l0 + lr, u = u0 + uc;
            double v = 0.0;
            if (l < L && u < npair) {
                int2 pq = pairs[u];
                v = q[(size_t)l * P + pq.x] * q[(size_t)l * P + pq.y];
            }
            sV[lr][uc] = v;
        }
        __syncthreads();
#pragma unroll
        for (int lr = 0; lr < MIJ_LC; lr++) {
            double vv = sV[lr][tx];
#pragma unroll
            for (int r = 0; r < R; r++) acc[lr & (NA - 1)][r] = fma(sPl[lr][ty + 8 * r], vv, acc[lr & (NA - 1)][r]);
        }
        __syncthreads();
    }
    const int u = u0 + tx;
    if (u >= npair) return;
    const int2 pq = pairs[u];
    auto put = [&](int k, double v) {
        double *blk = mt + (size_t)k * P * P;
        blk[pq.x * P + pq.y] = v;
        blk[pq.y * P + pq.x] = v;
    };
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int k = k0 + ty + 8 * r;
        if (k >= nk) continue;
        if (!FOLD) {
            put(k, acc[0][r]);
        } else {
            // the sums start at lmin: acc[0] holds its parity
            const double E = acc[(lmin & 1) ? NA - 1 : 0][r], O = acc[(lmin & 1) ? 0 : NA - 1][r];
            put(k, E + O);
            if (nmu - 1 - k != k) put(nmu - 1 - k, E - O);
        }
    }
}

// The 64-node tile under the name that the allocation-free entry point launches, and the tile of 8R
// nodes for the regular path.
__global__ void __launch_bounds__(256) k_mij_fp64(int nmu, int lmin, int lmax, int P, int npair, const double *__restrict__ pl,
                                                  const double *__restrict__ q, const int2 *__restrict__ pairs,
                                                  double *__restrict__ mt)
{
    mij_tile<8, false>(nmu, lmin, lmax, P, npair, pl, q, pairs, mt);
}

template <int R>
__global__ void __launch_bounds__(256) k_mij_fp64_r(int nmu, int lmin, int lmax, int P, int npair,
                                                    const double *__restrict__ pl, const double *__restrict__ q,
                                                    const int2 *__restrict__ pairs, double *__restrict__ mt)
{
    mij_tile<R, false>(nmu, lmin, lmax, P, npair, pl, q, pairs, mt);
}

__global__ void __launch_bounds__(256) k_mij_fp64_fold(int nmu, int lmin, int lmax, int P, int npair,
                                                       const double *__restrict__ pl, const double *__restrict__ q,
                                                       const int2 *__restrict__ pairs, double *__restrict__ mt)
{
    mij_tile<8, true>(nmu, lmin, lmax, P, npair, pl, q, pairs, mt);
}

// M table [nmu][P][P] of a basis q[L][P] on lmin..lmax (T or E) into out.
modal_status mij_table_dev(modal_ctx *ctx, const double *q, int lmin, int lmax, int P, DevBuf &out)
{
    const int npair = P * (P + 1) / 2;
    MODAL_TRY(ensure(out, sizeof(double) * (size_t)ctx->nmu * P * P));
    MODAL_TRY(ensure(ctx->scratch, sizeof(int2) * npair));
    int2 *h = new int2[npair];
    int u = 0;
    for (int p = 0; p < P; p++)
        for (int qq = p; qq < P; qq++) h[u++] = make_int2(p, qq);
    cudaError_t e = cudaMemcpyAsync(ctx->scratch.ptr, h, sizeof(int2) * npair, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    delete[] h;
    if (e != cudaSuccess) { set_error("mij pairs: %s", cudaGetErrorString(e)); return MODAL_ERR_CUDA; }
    // smaller mu tiles until there are two CTAs per SM: with 24 CTAs (l <= 500, P = 10) the 64-node tile
    // took 295 us, the FP64 pipe of 128 SMs idle.  Folded where half the nodes still fill the GPU with
    // full tiles (l <= 2000, P = 30: 6.1 -> 3.1 ms); below that it would only leave fewer CTAs, and the
    // sum keeps the reference's order.
    int nsm = 0, R = 8;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    const bool fold = ctx->gl_sym && (long)ceil_div((ctx->nmu + 1) / 2, 64) * ceil_div(npair, MIJ_BU) >= 2L * nsm;
    const int nk = fold ? (ctx->nmu + 1) / 2 : ctx->nmu;
    while (R > 1 && (long)ceil_div(nk, 8 * R) * ceil_div(npair, MIJ_BU) < 2L * nsm) R /= 2;
    auto run = [&](auto kern) {
        kern<<<dim3(ceil_div(nk, 8 * R), ceil_div(npair, MIJ_BU)), 256, 0, ctx->stream>>>(
            ctx->nmu, lmin, lmax, P, npair, ctx->pl.as<double>(), q, ctx->scratch.as<int2>(), out.as<double>());
    };
    if (fold) run(k_mij_fp64_fold);
    else if (R == 8) run(k_mij_fp64);
    else if (R == 4) run(k_mij_fp64_r<4>);
    else if (R == 2) run(k_mij_fp64_r<2>);
    else run(k_mij_fp64_r<1>);
    return launched(ctx, "mij_fp64");
}

modal_status mij_dev(modal_ctx *ctx)
{
    return mij_table_dev(ctx, ctx->q.as<double>(), ctx->lmin, ctx->lmax, ctx->P, ctx->mt);
}

modal_status mt_ready(modal_ctx *ctx)
{
    if (ctx->have_mt) return MODAL_OK;
    StageTimer t(ctx, MODAL_T_MIJ);
    MODAL_TRY(mij_dev(ctx));
    ctx->have_mt = true;
    return MODAL_OK;
}

// --------------------------------------------------------------------------
// mu-contraction, FP64.  One CTA per 32x32 tile of (m,n) with tile(m) <= tile(n);
// thread (tx,ty) owns n = n0+tx and m = m0+ty+8r, r < 4.  A chunk of KC mu
// steps of the whole P x P table is staged in shared memory; per (pair, mu):
// 9 shared loads, the permanent in 9 FP64 ops and one FMA with the weight.
// Summation over mu in ascending order.
// --------------------------------------------------------------------------
__global__ void k_wgt48(int nmu, const double *w, double *wg)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nmu) wg[k] = w[k] / (48e0 * 3.14159265358979323846);
}

__global__ void __launch_bounds__(256) k_gamma_fp64(int N, int P, int nmu, int KC, const int *__restrict__ triples,
                                                    const double *__restrict__ mt, const double *__restrict__ wg,
                                                    double *__restrict__ gamma)
{
    const int tm = blockIdx.y, tn = blockIdx.x;
    if (tm > tn) return;
    extern __shared__ double smem[];
    double *sW = smem;       // [KC]
    double *sA = smem + KC;  // [KC][P*P]
    const int PP = P * P;
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int n = tn * 32 + tx;
    int nb0 = 0, nb1 = 0, nb2 = 0;
    if (n < N) { nb0 = triples[3 * n]; nb1 = triples[3 * n + 1]; nb2 = triples[3 * n + 2]; }
    int mo[4][3];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = tm * 32 + ty + 8 * r;
        if (m < N) { mo[r][0] = triples[3 * m] * P; mo[r][1] = triples[3 * m + 1] * P; mo[r][2] = triples[3 * m + 2] * P; }
        else { mo[r][0] = mo[r][1] = mo[r][2] = 0; }
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k0 = 0; k0 < nmu; k0 += KC) {
        const int kc = min(KC, nmu - k0);
        const double *src = mt + (size_t)k0 * PP;
        for (int e = tid; e < kc * PP; e += 256) sA[e] = src[e];
        if (tid < kc) sW[tid] = wg[k0 + tid];
        __syncthreads();
        for (int kk = 0; kk < kc; kk++) {
            const double *A = sA + kk * PP;
            const double wk = sW[kk];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const double *r1 = A + mo[r][0], *r2 = A + mo[r][1], *r3 = A + mo[r][2];
                double a11 = r1[nb0], a12 = r1[nb1], a13 = r1[nb2];
                double a21 = r2[nb0], a22 = r2[nb1], a23 = r2[nb2];
                double a31 = r3[nb0], a32 = r3[nb1], a33 = r3[nb2];
                double t1 = fma(a23, a32, a22 * a33);
                double t2 = fma(a23, a31, a21 * a33);
                double t3 = fma(a22, a31, a21 * a32);
                double pm = fma(a13, t3, fma(a12, t2, a11 * t1));
                acc[r] = fma(wk, pm, acc[r]);
            }
        }
        __syncthreads();
    }
    if (n >= N) return;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int m = tm * 32 + ty + 8 * r;
        if (m < N && m <= n) {
            gamma[(size_t)m * N + n] = acc[r];
            gamma[(size_t)n * N + m] = acc[r];
        }
    }
}

modal_status gamma_fp64_dev(modal_ctx *ctx, int mu0, int nmu)
{
    const int N = ctx->N, P = ctx->P;
    MODAL_TRY(mt_ready(ctx));
    MODAL_TRY(ensure(ctx->gamma, sizeof(double) * (size_t)N * N));
    MODAL_TRY(ensure(ctx->scratch2, sizeof(double) * nmu));
    k_wgt48<<<ceil_div(nmu, 256), 256, 0, ctx->stream>>>(nmu, ctx->w.as<double>() + mu0, ctx->scratch2.as<double>());
    MODAL_TRY(launched(ctx, "wgt48"));
    // the distinct products of three M entries, or (few modes of a large basis) the permanents of the
    // pairs: full lists at l <= 2000 take 98 ms on the first against 665 ms on the second at P = 30
    if (triple_wins(0.5 * N * (N + 1.0), 0.5 * P * (P + 1.0))) {
        const modal_status st = gamma_triple_dev(ctx, mu0, nmu, ctx->scratch2.as<double>());
        if (st != MODAL_ERR_NOMEM) return st;
    }
    int KC = (96 * 1024) / (P * P * 8);
    if (KC < 1) KC = 1;
    if (KC > 32) KC = 32;
    if (ctx->gamma_kc > 0 && sizeof(double) * ((size_t)ctx->gamma_kc * (1 + (size_t)P * P)) <= 200 * 1024)
        KC = ctx->gamma_kc;  // tuned (modal_autotune)
    size_t smem = sizeof(double) * ((size_t)KC + (size_t)KC * P * P);
    if (smem > 200 * 1024) { set_error("gamma_fp64: P=%d too large for the shared-memory tile", P); return MODAL_ERR_ARG; }
    MODAL_CUDA(cudaFuncSetAttribute(k_gamma_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int nt = ceil_div(N, 32);
    dim3 grid(nt, nt);
    k_gamma_fp64<<<grid, 256, smem, ctx->stream>>>(N, P, nmu, KC, ctx->triples.as<int>(),
                                                   ctx->mt.as<double>() + (size_t)mu0 * P * P,
                                                   ctx->scratch2.as<double>(), ctx->gamma.as<double>());
    return launched(ctx, "gamma_fp64");
}

}  // namespace modal

// triple.cu -- FP64 contractions over distinct products of three M entries.
//
// Gamma_mn = sum_k w_k/(48 pi) perm3(M(k)[m_a][n_b])   (orthogonalisation_late.c:239-336)
// evaluated pair by pair costs ten FP64 instructions per (m, n) and node, N^2/2 pairs.  But every
// term of a permanent is a product of three entries of the symmetric P x P table M(k), and there
// are only U (U+1) (U+2) / 6 such products, U = P (P+1) / 2: for the full mode list (N ~ P^3/6)
// about 1/40 of the permanents' multiplications.  So
//   T[u][(v,t)] = sum_k X_u(k) Z_v(k) X_t(k),  u <= v <= t,  X_u(k) = M_ab(mu_k), Z = w X,
// is formed once (one FMA per product and node, all FP64), and Gamma_mn gathers its six entries.
// The transfer Gamma has the same form with the U = Pp P entries of M[p][q] at one radial sample.
//
// Bound: the FP64 pipe, one warp instruction per 16 cycles and SM on GB300, which hides every load
// of these kernels; so the tiles only serve to keep the number of FP64 instructions near one per
// product: 32 u x 64 (v,t) per CTA, the products Z_v X_t formed once per tile (1/32 extra), tiles
// with no u <= v skipped, and within a tile the warps (4 u each) with none.
// Measured: l <= 2000, P = 30 (U = 465, 1.7e7 products, 5.1e10 FMAs): a new basis in 98 ms, 665 ms by
// permanents.
#include <algorithm>
#include <cmath>
#include <vector>
#include "common.cuh"
#include "triple.cuh"

namespace modal {

namespace {

constexpr int TP_BU = 32, TP_BV = 64, TP_KC = 16;

// X[k][u] = base[k stride + off(u)], Z[k][u] = w(k) X[k][u]; off(u) = a P + b for the pair u = (a, b)
// of a symmetric P x P table (P > 0), or u (P = 0).
__global__ void k_triple_rows(long K, int U, int P, const double *__restrict__ base, long stride,
                              const double *__restrict__ w, double *__restrict__ X, double *__restrict__ Z)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= K * U) return;
    const long k = e / U;
    const int u = (int)(e - k * U);
    int a = 0, b = u;
    if (P > 0) tri_unrank(u, P, a, b);
    const double x = base[k * stride + (P > 0 ? a * P + b : u)];
    X[e] = x;
    Z[e] = w[k] * x;
}

// T[u][r] over nodes [z kper, (z + 1) kper) to T + z zstride.  Thread (lane, warp): rows
// 4 warp .. + 3 of the u tile, columns lane and lane + 32 of the (v, t) tile.
__global__ void __launch_bounds__(256) k_triple(int U, int UV, int K, int kper, const double *__restrict__ X,
                                                const double *__restrict__ Z, double *__restrict__ T, size_t zstride)
{
    const int r0 = blockIdx.x * TP_BV, u0 = blockIdx.y * TP_BU;
    int vl, tl;
    tri_unrank(min(r0 + TP_BV, UV) - 1, U, vl, tl);
    if (u0 > vl) return;
    __shared__ __align__(16) double sX[TP_KC][TP_BU];
    __shared__ double sY[TP_KC][TP_BV];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k0 = blockIdx.z * kper, k1 = min(K, k0 + kper);
    // this thread's column of Y and of X
    int v, t;
    tri_unrank(min(r0 + (tid & 63), UV - 1), U, v, t);
    const double *zc = Z + v, *xc = X + t, *uc = X + min(u0 + lane, U - 1);
    double acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0.0;
    double rx[2], ry[4], rz[4];
    auto fetch = [&](int kb) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int k = kb + warp + 8 * i;
            rx[i] = k < k1 ? uc[(size_t)k * U] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int k = kb + (tid >> 6) + 4 * i;
            ry[i] = k < k1 ? xc[(size_t)k * U] : 0.0;
            rz[i] = k < k1 ? zc[(size_t)k * U] : 0.0;
        }
    };
    fetch(k0);
    for (int kb = k0; kb < k1; kb += TP_KC) {
#pragma unroll
        for (int i = 0; i < 2; i++) sX[warp + 8 * i][lane] = rx[i];
#pragma unroll
        for (int i = 0; i < 4; i++) sY[(tid >> 6) + 4 * i][tid & 63] = rz[i] * ry[i];
        __syncthreads();
        if (kb + TP_KC < k1) fetch(kb + TP_KC);
        const int kn = u0 + 4 * warp <= vl ? min(TP_KC, k1 - kb) : 0;  // a warp past every v leaves the pipe to the others
#pragma unroll 4
        for (int kk = 0; kk < kn; kk++) {
            const double2 xa = *reinterpret_cast<const double2 *>(&sX[kk][4 * warp]);
            const double2 xb = *reinterpret_cast<const double2 *>(&sX[kk][4 * warp + 2]);
            const double x[4] = {xa.x, xa.y, xb.x, xb.y}, y0 = sY[kk][lane], y1 = sY[kk][lane + 32];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i][0] = fma(x[i], y0, acc[i][0]);
                acc[i][1] = fma(x[i], y1, acc[i][1]);
            }
        }
        __syncthreads();
    }
    T += blockIdx.z * zstride;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int u = u0 + 4 * warp + i;
        if (u >= U) break;
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (r0 + lane + 32 * c < UV) T[(size_t)u * UV + r0 + lane + 32 * c] = acc[i][c];
    }
}

// T[e] = sum over the Z partials (in order), in place on the first; tiles that k_triple skips hold
// nothing and are never read.
__global__ void k_triple_sum(size_t n, int Z, size_t zstride, double *__restrict__ T)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    double s = T[e];
    for (int z = 1; z < Z; z++) s += T[z * zstride + e];
    T[e] = s;
}

// Gamma_mn from the six sorted-triple entries of T, one thread per (m, n) of a 32 x 32 tile with
// tile(m) <= tile(n); both halves written.
__global__ void __launch_bounds__(256) k_gamma_gather(int N, int P, int U, long ldT, const int *__restrict__ triples,
                                                      const double *__restrict__ T, double *__restrict__ gamma)
{
    const int tm = blockIdx.y, tn = blockIdx.x;
    if (tm > tn) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int n = tn * 32 + tx;
    if (n >= N) return;
    const int nn[3] = {triples[3 * n], triples[3 * n + 1], triples[3 * n + 2]};
    const int perm[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}, {1, 0, 2}, {0, 2, 1}};
    for (int r = 0; r < 4; r++) {
        const int m = tm * 32 + ty + 8 * r;
        if (m >= N || m > n) continue;
        const int mm[3] = {triples[3 * m], triples[3 * m + 1], triples[3 * m + 2]};
        double g = 0.0;
#pragma unroll
        for (int s = 0; s < 6; s++)
            g += T[triple_at(pair_rank(mm[0], nn[perm[s][0]], P), pair_rank(mm[1], nn[perm[s][1]], P),
                             pair_rank(mm[2], nn[perm[s][2]], P), U, ldT)];
        gamma[(size_t)m * N + n] = g;
        gamma[(size_t)n * N + m] = g;
    }
}

// X^T[u][k] = M_ab(mu_k), u = (a, b), from the symmetric P x P rows of the M table.
__global__ void k_triple_cols(int K, int U, int P, const double *__restrict__ mt, double *__restrict__ XT)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)K * U) return;
    const int u = (int)(e / K), k = (int)(e - (long)u * K);
    int a, b;
    tri_unrank(u, P, a, b);
    XT[e] = mt[(size_t)k * P * P + a * P + b];
}

// Adjoint of the gather: T[sorted triple] += G_mn for each of the six terms of every (m, n).
__global__ void k_gamma_scatter(int N, int P, int U, long ldT, const int *__restrict__ triples, const double *__restrict__ G,
                                double *__restrict__ T)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)N * N) return;
    const int m = (int)(e / N), n = (int)(e - (long)m * N);
    const double g = G[e];
    if (g == 0.0) return;
    const int mm[3] = {triples[3 * m], triples[3 * m + 1], triples[3 * m + 2]};
    const int nn[3] = {triples[3 * n], triples[3 * n + 1], triples[3 * n + 2]};
    const int perm[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}, {1, 0, 2}, {0, 2, 1}};
#pragma unroll
    for (int s = 0; s < 6; s++)
        atomicAdd(&T[triple_at(pair_rank(mm[0], nn[perm[s][0]], P), pair_rank(mm[1], nn[perm[s][1]], P),
                               pair_rank(mm[2], nn[perm[s][2]], P), U, ldT)],
                  g);
}

// Adjoint of the contraction over nodes: part[z][a][k] = sum over pairs r = (v, t) of split z of
//   mult(a; {a, v, t}) T[{a, v, t}] X_v(k) X_t(k),
// mult the number of times a stands in the sorted triple (d/dX_a of X_u X_v X_t).  Tile 32 a x 64 k,
// 16 pairs per stage; one FP64 FMA per (a, r, k), the products X_v X_t formed once per tile.
__global__ void __launch_bounds__(256) k_triple_vjp(int U, int UV, int K, int rper, const double *__restrict__ XT,
                                                    const double *__restrict__ T, double *__restrict__ part)
{
    __shared__ __align__(16) double sC[TP_KC][TP_BU];
    __shared__ double sY[TP_KC][TP_BV];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k0 = blockIdx.x * TP_BV, a0 = blockIdx.y * TP_BU;
    const int r0 = blockIdx.z * rper, r1 = min(UV, r0 + rper);
    const int kc = min(k0 + (tid & 63), K - 1), ac = min(a0 + lane, U - 1);
    double acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0.0;
    for (int rb = r0; rb < r1; rb += TP_KC) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = rb + warp + 8 * i;
            double c = 0.0;
            if (r < r1) {
                int v, t;
                tri_unrank(r, U, v, t);
                c = T[triple_at(ac, v, t, U, UV)] * (double)(1 + (ac == v) + (ac == t));
            }
            sC[warp + 8 * i][lane] = c;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = rb + (tid >> 6) + 4 * i;
            double y = 0.0;
            if (r < r1) {
                int v, t;
                tri_unrank(r, U, v, t);
                y = XT[(size_t)v * K + kc] * XT[(size_t)t * K + kc];
            }
            sY[(tid >> 6) + 4 * i][tid & 63] = y;
        }
        __syncthreads();
        const int rn = min(TP_KC, r1 - rb);
#pragma unroll 4
        for (int rr = 0; rr < rn; rr++) {
            const double2 ca = *reinterpret_cast<const double2 *>(&sC[rr][4 * warp]);
            const double2 cb = *reinterpret_cast<const double2 *>(&sC[rr][4 * warp + 2]);
            const double c[4] = {ca.x, ca.y, cb.x, cb.y}, y0 = sY[rr][lane], y1 = sY[rr][lane + 32];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i][0] = fma(c[i], y0, acc[i][0]);
                acc[i][1] = fma(c[i], y1, acc[i][1]);
            }
        }
    }
    part += (size_t)blockIdx.z * U * K;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int a = a0 + 4 * warp + i;
        if (a >= U) break;
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (k0 + lane + 32 * c < K) part[(size_t)a * K + k0 + lane + 32 * c] = acc[i][c];
    }
}

// dX[k][u] = w_k/(48 pi) sum over the splits of part[z][u][k]
__global__ void k_triple_vjp_sum(int U, int K, int Z, const double *__restrict__ w, const double *__restrict__ part,
                                 double *__restrict__ dX)
{
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)U * K) return;
    const int u = (int)(e / K), k = (int)(e - (long)u * K);
    double s = 0.0;
    for (int z = 0; z < Z; z++) s += part[(size_t)z * U * K + e];
    dX[(size_t)k * U + u] = w[k] / (48e0 * 3.14159265358979323846) * s;
}

}  // namespace

bool triple_wins(double pairs, double U)
{
    // FP64 instructions per node: ten per pair, against one per product (tile edges and the products
    // Z_v X_t add about a fifth).  T is kept under 16 GB.
    const double UV = U * (U + 1) / 2;
    return 1.2 * U * (U + 1) * (U + 2) / 6 < 10.0 * pairs && 8.0 * U * UV <= 16e9;
}

modal_status triple_rows_dev(modal_ctx *ctx, long K, int U, int P, const double *base, long stride, const double *w,
                             double *X, double *Z)
{
    k_triple_rows<<<ceil_div(K * U, 256), 256, 0, ctx->stream>>>(K, U, P, base, stride, w, X, Z);
    return launched(ctx, "triple_rows");
}

int triple_splits(const modal_ctx *ctx, int U, long K)
{
    int nsm = 152;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device);
    const long UV = (long)U * (U + 1) / 2;
    // tiles with work: about a third of all, never fewer than one column of them; six CTAs per SM
    // even out the last wave, and a split costs one more pass over T
    const long tiles = std::max<long>(ceil_div(UV, TP_BV), (long)ceil_div(UV, TP_BV) * ceil_div(U, TP_BU) / 3);
    return (int)std::max<long>(1, std::min<long>(std::min<long>(ceil_div(K, 8 * TP_KC), 32), 6L * nsm / tiles));
}

modal_status triple_dev(modal_ctx *ctx, int U, int K, int kper, const double *X, const double *Z, double *T, size_t zstride)
{
    const long UV = (long)U * (U + 1) / 2;
    const dim3 grid(ceil_div(UV, TP_BV), ceil_div(U, TP_BU), ceil_div(K, kper));
    k_triple<<<grid, 256, 0, ctx->stream>>>(U, (int)UV, K, kper, X, Z, T, zstride);
    return launched(ctx, "triple");
}

modal_status triple_sum_dev(modal_ctx *ctx, size_t n, int Z, size_t zstride, double *T)
{
    if (Z <= 1) return MODAL_OK;
    k_triple_sum<<<ceil_div((long)n, 256), 256, 0, ctx->stream>>>(n, Z, zstride, T);
    return launched(ctx, "triple_sum");
}

modal_status gamma_gather_dev(modal_ctx *ctx, int U, const double *T)
{
    const int nt = ceil_div(ctx->N, 32);
    k_gamma_gather<<<dim3(nt, nt), 256, 0, ctx->stream>>>(ctx->N, ctx->P, U, (long)U * (U + 1) / 2, ctx->triples.as<int>(), T,
                                                          ctx->gamma.as<double>());
    return launched(ctx, "gamma_gather");
}

// Plain FP64 Gamma over nodes mu0 .. mu0 + nmu - 1 from the M table; wg: w / (48 pi) of those nodes.
modal_status gamma_triple_dev(modal_ctx *ctx, int mu0, int nmu, const double *wg)
{
    const int P = ctx->P, U = P * (P + 1) / 2;
    const size_t UV = (size_t)U * (U + 1) / 2;
    const int kper = ceil_div(ceil_div(nmu, triple_splits(ctx, U, nmu)), TP_KC) * TP_KC, Zn = ceil_div(nmu, kper);
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t oz = al(sizeof(double) * (size_t)nmu * U), ot = 2 * oz;
    MODAL_TRY(ensure(ctx->trip, ot + sizeof(double) * Zn * U * UV));
    double *X = ctx->trip.as<double>(), *Z = reinterpret_cast<double *>(ctx->trip.as<uint8_t>() + oz),
           *T = reinterpret_cast<double *>(ctx->trip.as<uint8_t>() + ot);
    MODAL_TRY(triple_rows_dev(ctx, nmu, U, P, ctx->mt.as<double>() + (size_t)mu0 * P * P, (long)P * P, wg, X, Z));
    MODAL_TRY(triple_dev(ctx, U, nmu, kper, X, Z, T, U * UV));
    MODAL_TRY(triple_sum_dev(ctx, U * UV, Zn, U * UV, T));
    return gamma_gather_dev(ctx, U, T);
}

// dX[nmu][U] = dL/dX of Gamma's M entries for an upstream G[N][N] = dL/dGamma (device).
modal_status gamma_triple_vjp_dev(modal_ctx *ctx, const double *G, double *dX)
{
    const int P = ctx->P, U = P * (P + 1) / 2, K = ctx->nmu, N = ctx->N;
    const size_t UV = (size_t)U * (U + 1) / 2;
    int nsm = 0;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    // pair splits: about six CTAs per SM
    const long tiles = (long)ceil_div(K, TP_BV) * ceil_div(U, TP_BU);
    const int want = (int)std::max<long>(1, std::min<long>(std::min<long>(32, ceil_div((long)UV, 4 * TP_KC)), 6L * nsm / tiles));
    const int rper = ceil_div(ceil_div((long)UV, want), TP_KC) * TP_KC, Zn = ceil_div((long)UV, rper);
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t ox = al(sizeof(double) * U * UV), op = ox + al(sizeof(double) * (size_t)U * K);
    MODAL_TRY(ensure(ctx->trip, op + sizeof(double) * Zn * (size_t)U * K));
    uint8_t *b = ctx->trip.as<uint8_t>();
    double *T = reinterpret_cast<double *>(b), *XT = reinterpret_cast<double *>(b + ox), *part = reinterpret_cast<double *>(b + op);
    MODAL_CUDA(cudaMemsetAsync(T, 0, sizeof(double) * U * UV, ctx->stream));
    k_gamma_scatter<<<ceil_div((long)N * N, 256), 256, 0, ctx->stream>>>(N, P, U, (long)UV, ctx->triples.as<int>(), G, T);
    MODAL_TRY(launched(ctx, "gamma_scatter"));
    k_triple_cols<<<ceil_div((long)K * U, 256), 256, 0, ctx->stream>>>(K, U, P, ctx->mt.as<double>(), XT);
    MODAL_TRY(launched(ctx, "triple_cols"));
    k_triple_vjp<<<dim3(ceil_div(K, TP_BV), ceil_div(U, TP_BU), Zn), 256, 0, ctx->stream>>>(U, (int)UV, K, rper, XT, T, part);
    MODAL_TRY(launched(ctx, "triple_vjp"));
    k_triple_vjp_sum<<<ceil_div((long)K * U, 256), 256, 0, ctx->stream>>>(U, K, Zn, ctx->w.as<double>(), part, dX);
    return launched(ctx, "triple_vjp_sum");
}

}  // namespace modal

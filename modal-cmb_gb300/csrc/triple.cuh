// triple.cuh -- index arithmetic and entry points of the contractions over
// distinct products of three table entries (triple.cu).
#pragma once
#include "common.cuh"

namespace modal {

// Pairs (a, b), a <= b < n, ordered by a then b: pair r of them, and the rank of a pair.
__host__ __device__ inline void tri_unrank(int r, int n, int &a, int &b)
{
    const float m = 2.f * n + 1.f, d = m * m - 8.f * (float)r;
    int x = (int)(0.5f * (m - sqrtf(d > 0.f ? d : 0.f)));
    if (x < 0) x = 0;
    if (x > n - 1) x = n - 1;
    auto first = [n](int q) { return (long long)q * n - (long long)q * (q - 1) / 2; };
    while (x > 0 && first(x) > r) x--;
    while (x < n - 1 && first(x + 1) <= r) x++;
    a = x;
    b = x + (int)(r - first(x));
}

__host__ __device__ inline int pair_rank(int a, int b, int n)
{
    const int lo = a < b ? a : b, hi = a < b ? b : a;
    return lo * n - lo * (lo - 1) / 2 + hi - lo;
}

// Position of the sorted triple of (x, y, z) in T[u][(v, t)] with leading dimension ld.
__host__ __device__ inline size_t triple_at(int x, int y, int z, int U, long ld)
{
    const int lo = x < y ? (x < z ? x : z) : (y < z ? y : z), hi = x > y ? (x > z ? x : z) : (y > z ? y : z);
    const int mid = x + y + z - lo - hi;
    return (size_t)lo * ld + (size_t)((long long)mid * U - (long long)mid * (mid - 1) / 2 + hi - mid);
}

// Whether forming the distinct products costs less than `pairs` permanents per node.
bool triple_wins(double pairs, double U);
// Node splits that fill the GPU.
int triple_splits(const modal_ctx *ctx, int U, long K);
// X[k][u] and Z[k][u] = w(k) X[k][u] from a table (P > 0: symmetric P x P rows; P = 0: rows of U entries).
modal_status triple_rows_dev(modal_ctx *ctx, long K, int U, int P, const double *base, long stride, const double *w,
                             double *X, double *Z);
// T[z][u][(v, t)] over nodes [z kper, (z + 1) kper), zstride entries between splits.
modal_status triple_dev(modal_ctx *ctx, int U, int K, int kper, const double *X, const double *Z, double *T,
                        size_t zstride);
modal_status triple_sum_dev(modal_ctx *ctx, size_t n, int Z, size_t zstride, double *T);
// ctx->gamma from T[U][U(U+1)/2].
modal_status gamma_gather_dev(modal_ctx *ctx, int U, const double *T);
modal_status gamma_triple_dev(modal_ctx *ctx, int mu0, int nmu, const double *wg);
modal_status gamma_triple_vjp_dev(modal_ctx *ctx, const double *G, double *dX);

}  // namespace modal

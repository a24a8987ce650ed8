// ozgemm.cu -- FP64-accurate matrix products on the FP16 tensor cores.
//
// GB300 runs FP64 at about 1.25 TFLOP/s but FP16 tensor products at about
// 2 PFLOP/s.  Here an FP64 product C = beta C + alpha op(A) op(B) runs on the
// tensor cores by exact integer slicing (the Ozaki scheme: Ozaki, Ogita, Oishi
// and Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", Numer. Algorithms
// 59 (2012)):
//
//   every row r of op(A) (and every column of op(B)) is scaled by a power of
//   two 2^e_r so that its entries lie in (-1, 1), then written as s balanced
//   7-bit digits:  x = 2^e sum_p d_p 2^{-6-7p},  d_p integer in [-64, 64],
//   exact in FP16 (x 2^{6-e+7(s-1)} rounded once to a 55-bit integer, its
//   digits split off with integer arithmetic).  A digit product is at most 2^12 in size, so the FP32
//   tensor-memory accumulator sums up to 4096 of them without rounding; the
//   K dimension is cut into blocks of OZ_KB = 512, and the products of one
//   block with equal p + q = g (at most s of them) share one accumulator,
//   still exact (s * 512 * 2^12 <= 2^24 for s <= 8).
//
//   C = 2^{eA_m + eB_n - 12} sum_{g < s} 2^{-7g} sum_{p+q=g} sum_k dA_p dB_q,
//   products with p + q >= s dropped (below 2^{-7s} of the leading term).
//
// The exact block sums are added in double-FP32 ("double-float": an FP32
// head and tail, Knuth's TwoSum) kept in registers; the tile is converted
// to FP64 once at the end.  Accuracy: about 2^-48 relative to max|row| max|col|
// per K block, the class of an FP64 GEMM over K = 5000 terms.
//
// Kernel k_oz_gemm: persistent, one CTA per SM over the output tiles
// (128 x 128); warp 0 TMA producer (5-stage ring of 32 KB: an A-slice and a
// B-slice chunk of 64 K, 128-byte swizzle), warp 1 MMA issuer (tcgen05.mma
// kind::f16, M = 128, N = 256 over the B chunks of two neighbouring stages, or 128
// where the ring wraps) and TMEM owner, warps 4-11 epilogue (64 columns
// of 32 rows each, the sums in 128 registers).  TMEM: four FP32 accumulators, two
// groups that the epilogue drains while the next two fill.  Two groups at a time
// take half as many operand copies as one (20 instead of 36 pairs of slices for
// s = 8).  Every mbarrier wait is bounded; on expiry the CTA flags an error, stops,
// drains its copies, frees TMEM and returns (MODAL_ERR_TIMEOUT).
//
// What bounds it: for a short K (the trailing updates of the tridiagonalisation,
// K = 64) the epilogue's instructions, 80 per 32 elements and tile after packing two
// columns per FP32 instruction and building the FP64 results as bit patterns; for a
// long K shared memory, which the copies write and the products read (an A chunk met with
// two B chunks by one instruction is read once; rows of 128 bytes instead of 64 halve the
// copies' requests).  Measured, one group at a time, four epilogue warps, sums in tensor memory,
// results by FP64 conversions -> two groups, eight warps, registers, bit patterns -> chunks of
// 64 K and N = 256: trailing update of 4,928 rows 361 -> 186 -> 170 us, a merge's 4,960 x 4,960 x
// 2,480 product 2.54 -> 2.10 -> 1.41 ms, the 220 products of an eigendecomposition of n = 4,960
// 42.1 -> 25.1 -> 20.4 ms.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>
#include "common.cuh"
#include "dfbits.cuh"
#include "ozdigits.cuh"
#include "tc_ptx.cuh"

namespace modal {

namespace {

using namespace tc;

constexpr int OZ_BM = 128, OZ_BN = 128, OZ_BK = 64, OZ_KB = 512, OZ_STAGES = 5;
constexpr int OZ_MAXS = 8;
constexpr uint32_t OZ_A_BYTES = OZ_BM * OZ_BK * 2;  // 16 KB
constexpr uint32_t OZ_B_BYTES = OZ_BN * OZ_BK * 2;  // 16 KB
constexpr uint32_t OZ_STAGE_BYTES = OZ_A_BYTES + OZ_B_BYTES;
constexpr int OZ_EW = 8;                          // epilogue warps: 32 rows x 64 columns of the tile each
constexpr int OZ_THREADS = 128 + 32 * OZ_EW;      // after one warpgroup of copies and products
constexpr int OZ_RIO = 56, OZ_REPI = 216;         // registers of that one and of the epilogue's, out of 168 each
static_assert(128 * OZ_RIO + 32 * OZ_EW * OZ_REPI <= OZ_THREADS * 168, "registers of the launch");
constexpr uint32_t OZ_STAGING = OZ_EW * 32 * 32 * 8;  // epilogue: 32 x 32 double-floats per warp, (r, c) at 32 r + (c ^ r)
constexpr uint32_t OZ_SMEM = OZ_STAGES * OZ_STAGE_BYTES + 1024 + 256 + OZ_STAGING;
constexpr uint32_t OZ_TMEM_COLS = 512;
constexpr long long OZ_WAIT = 1ll << 31;  // ~1 s of clock64 per wait
constexpr uint32_t OZ_IDESC = idesc_f16(OZ_BM, OZ_BN), OZ_IDESC2 = idesc_f16(OZ_BM, 2 * OZ_BN);

// ------------------------------------------------------------------ slicing
// Rows of op(X), R x K: element (r, k) = trans ? X[k*ld + r] : X[r*ld + k].
// Tiles of 32 rows x 32 columns through shared memory (coalesced either way).
__device__ __forceinline__ void oz_load_tile(double (*tile)[33], const double *__restrict__ X, long ld, int trans,
                                             int R, int K, int r0, int k0)
{
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (!trans) {
        for (int rr = ty; rr < 32; rr += 8) {
            const int r = r0 + rr, k = k0 + tx;
            tile[rr][tx] = (r < R && k < K) ? X[(size_t)r * ld + k] : 0.0;
        }
    } else {
        for (int kk = ty; kk < 32; kk += 8) {
            const int r = r0 + tx, k = k0 + kk;
            tile[tx][kk] = (r < R && k < K) ? X[(size_t)k * ld + r] : 0.0;
        }
    }
}

// Row exponents, over K chunks in parallel: ex[r] = max over the row of
// ilogb(|x|) + 1 (atomicMax over the chunks; ex starts at a value below every
// exponent, and an all-zero row keeps it).  grid (Rpad / 32, K chunks).
__global__ void __launch_bounds__(256) k_oz_rowexp(int R, int K, int kchunk, const double *__restrict__ X, long ld,
                                                   int trans, int *__restrict__ ex)
{
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, kb = blockIdx.y * kchunk, ke = min(K, kb + kchunk);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    // the maxima on the bit patterns (integer instructions, not the FP64 pipe)
    unsigned long long mx[4] = {0ull, 0ull, 0ull, 0ull};
    for (int k0 = kb; k0 < ke; k0 += 32) {
        oz_load_tile(tile, X, ld, trans, R, ke, r0, k0);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; j++) mx[j] = dfb::absmax_bits(mx[j], tile[ty + 8 * j][tx]);
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        unsigned long long b = mx[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
        const double v = __longlong_as_double((long long)b);
        const int r = r0 + ty + 8 * j;
        if (tx == 0 && r < R && v > 0.0 && isfinite(v)) atomicMax(ex + r, ilogb(v) + 1);
    }
}

// Slices of the rows of op(X) from their exponents: out: [s][Rpad][Kpad] FP16
// digits.  Rows >= R and columns >= K are zero; a row whose exponent is still
// the starting value (all zero) gets exponent 0.  grid (Rpad / 32, K chunks).
__global__ void __launch_bounds__(256) k_oz_slice(int R, int K, int Rpad, int Kpad, int kchunk,
                                                  const double *__restrict__ X, long ld, int trans, int s,
                                                  __half *__restrict__ out, int *__restrict__ ex)
{
    __shared__ double tile[32][33];
    __shared__ int sexp[32];
    const int r0 = blockIdx.x * 32, kb = blockIdx.y * kchunk, ke = min(Kpad, kb + kchunk);
    if (threadIdx.x < 32) {
        const int r = r0 + threadIdx.x;
        const int e = ex[r];
        sexp[threadIdx.x] = (e < -100000) ? 0 : e;
    }
    __syncthreads();
    if (blockIdx.y == 0 && threadIdx.x < 32) ex[r0 + threadIdx.x] = sexp[threadIdx.x];
    const size_t plane = (size_t)Rpad * Kpad;
    for (int k0 = kb; k0 < ke; k0 += 32) {
        if (k0 < K) oz_load_tile(tile, X, ld, trans, R, K, r0, k0);
        __syncthreads();
        // two neighbouring columns per thread
        const int c = 2 * (threadIdx.x & 15);
        for (int rr = threadIdx.x >> 4; rr < 32; rr += 16) {
            const double x0 = (k0 < K) ? tile[rr][c] : 0.0, x1 = (k0 < K) ? tile[rr][c + 1] : 0.0;
            ozd::store2(x0, x1, 6 - sexp[rr] + 7 * (s - 1), s,
                        reinterpret_cast<__half2 *>(out + (size_t)(r0 + rr) * Kpad + k0 + c), plane / 2);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ GEMM
struct OzArgs {
    int M, N, Kpad, Mpad, Npad, s, nkb, ntiles, lower, kper;
    const int4 *tiles;  // work items: (tile row, tile column, K split index, -)
    double *part;       // K split > 1: partial products [split][M][N]
    const int *ea, *eb;
    double alpha, beta;
    double *C;
    long ldc;
    int *err;
};

// Pairs of floats (packed arithmetic).
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float a, float b)
{
    f2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 upk(f2 v)
{
    float2 x;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x.x), "=f"(x.y) : "l"(v));
    return x;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 v;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}

// double-float a + b (Knuth's TwoSum, then renormalised), two at a time
__device__ __forceinline__ void df_add2(f2 &hi, f2 &lo, f2 b)
{
    const f2 s = add2(hi, b);
    const f2 bb = sub2(s, hi);
    const f2 e = add2(sub2(hi, sub2(s, bb)), sub2(b, bb));
    const f2 t = add2(lo, e);
    hi = add2(s, t);
    lo = sub2(t, sub2(hi, s));
}

// (h + l) 2^er 2^en where the bit patterns do not reach.  A call of its own: inlined, its FP64
// instructions are executed for every element and thrown away.
__device__ __noinline__ double oz_join_far(float h, float l, int er, int en)
{
    return ((double)h + (double)l) * ldexp(1.0, er) * ldexp(1.0, en);
}

// The digit products of one K block run in groups of equal p + q = g, two groups
// g = gh - 1, gh at a time (group 0 alone when s is odd): A's digit p then meets B's digits
// gh - p and gh - 1 - p, the second of which is the first of p + 1.  A stage of the ring
// holds (A_p, B_{gh-1-p}) and keeps its B for the next stage's products.
__device__ __forceinline__ int oz_first_group(int s) { return (s & 1) ? 0 : 1; }

__global__ void __launch_bounds__(OZ_THREADS, 1) k_oz_gemm(const __grid_constant__ CUtensorMap tmA,
                                                           const __grid_constant__ CUtensorMap tmB, OzArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + OZ_STAGES * OZ_STAGE_BYTES);
    uint64_t *full = bars, *empty = bars + OZ_STAGES, *afull = bars + 2 * OZ_STAGES, *aempty = afull + 2;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + 2 * OZ_STAGES + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * OZ_STAGES + 5);
    float2 *stage = reinterpret_cast<float2 *>(smem + OZ_STAGES * OZ_STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = a.s;
    if (threadIdx.x == 0) {
        for (int i = 0; i < OZ_STAGES; i++) {
            mbar_init(smem_u32(&full[i]), 1);
            mbar_init(smem_u32(&empty[i]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&afull[b]), 1);
            mbar_init(smem_u32(&aempty[b]), OZ_EW);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void *)tmem_slot), OZ_TMEM_COLS);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OZ_RIO));
        if (warp == 0) {
            if (lane == 0) {
                long g = 0;
                bool stop = false;
                // the next stage: digit p of A (p >= 0) and digit q of B (q >= 0), columns k .. k + 63
                auto load = [&](int p, int q, int m0, int n0, int k) {
                    const int st = (int)(g % OZ_STAGES);
                    const long it = g / OZ_STAGES;
                    if (it > 0 && !mbar_wait(smem_u32(&empty[st]), (uint32_t)((it - 1) & 1), abort_flag, OZ_WAIT)) {
                        if (!*abort_flag) { *abort_flag = 1; atomicCAS(a.err, 0, 1); }
                        return false;
                    }
                    uint8_t *sa = smem + (size_t)st * OZ_A_BYTES, *sb = smem + OZ_STAGES * OZ_A_BYTES + (size_t)st * OZ_B_BYTES;
                    const uint32_t fb = smem_u32(&full[st]);
                    mbar_expect_tx(fb, (p >= 0 ? OZ_A_BYTES : 0u) + (q >= 0 ? OZ_B_BYTES : 0u));
                    if (p >= 0) tma_load_2d(smem_u32(sa), &tmA, k, p * a.Mpad + m0, fb);
                    if (q >= 0) tma_load_2d(smem_u32(sb), &tmB, k, q * a.Npad + n0, fb);
                    g++;
                    return true;
                };
                for (int t = blockIdx.x; t < a.ntiles && !stop; t += gridDim.x) {
                    const int4 tile = a.tiles[t];
                    const int m0 = tile.x * OZ_BM, n0 = tile.y * OZ_BN;
                    const int kb0 = tile.z * a.kper, kb1 = min(a.nkb, kb0 + a.kper);
                    for (int kb = kb0; kb < kb1 && !stop; kb++) {
                        const int kbeg = kb * OZ_KB, nkc = min(OZ_KB, a.Kpad - kbeg) / OZ_BK;
                        for (int gh = oz_first_group(s); gh < s && !stop; gh += 2)
                            for (int kc = 0; kc < nkc && !stop; kc++) {
                                const int k = kbeg + kc * OZ_BK;
                                if (gh > 0) stop = !load(-1, gh, m0, n0, k);
                                for (int p = 0; p <= gh && !stop; p++) stop = !load(p, gh > 0 ? gh - 1 - p : 0, m0, n0, k);
                            }
                    }
                }
                // drain: the copies of the last stages must land before the CTA exits
                for (long h = (g > OZ_STAGES ? g - OZ_STAGES : 0); h < g; h++) {
                    const int st = (int)(h % OZ_STAGES);
                    const long long t0 = clock64();
                    while (!mbar_try(smem_u32(&full[st]), (uint32_t)((h / OZ_STAGES) & 1)) && clock64() - t0 < OZ_WAIT) {
                    }
                }
            }
        } else if (warp == 1) {
            if (lane == 0) {
                long g = 0, u = 0;
                bool stop = false;
                uint32_t sa = 0, sb = 0;
                auto wait = [&]() {  // the next stage has landed
                    const int st = (int)(g % OZ_STAGES);
                    if (!mbar_wait(smem_u32(&full[st]), (uint32_t)((g / OZ_STAGES) & 1), abort_flag, OZ_WAIT)) {
                        if (!*abort_flag) { *abort_flag = 1; atomicCAS(a.err, 0, 2); }
                        return false;
                    }
                    tc_fence_after();
                    sa = smem_u32(smem + (size_t)st * OZ_A_BYTES);
                    sb = smem_u32(smem + OZ_STAGES * OZ_A_BYTES + (size_t)st * OZ_B_BYTES);
                    g++;
                    return true;
                };
                auto mma = [&](uint32_t d, uint32_t ax, uint32_t bx, uint32_t idesc, uint32_t acc) {
#pragma unroll
                    for (int kk = 0; kk < OZ_BK / 16; kk++) {
                        umma_f16(d, desc_sw128(ax + kk * 32), desc_sw128(bx + kk * 32), idesc, acc);
                        acc = 1;
                    }
                };
                for (int t = blockIdx.x; t < a.ntiles && !stop; t += gridDim.x) {
                    const int kb0 = a.tiles[t].z * a.kper, kb1 = min(a.nkb, kb0 + a.kper);
                    for (int kb = kb0; kb < kb1 && !stop; kb++) {
                        const int kbeg = kb * OZ_KB, nkc = min(OZ_KB, a.Kpad - kbeg) / OZ_BK;
                        for (int gh = oz_first_group(s); gh < s && !stop; gh += 2, u++) {
                            const int buf = (int)(u & 1);
                            const long use = u >> 1;
                            if (use > 0 && !mbar_wait(smem_u32(&aempty[buf]), (uint32_t)((use - 1) & 1), abort_flag, OZ_WAIT)) {
                                if (!*abort_flag) { *abort_flag = 1; atomicCAS(a.err, 0, 4); }
                                stop = true;
                                break;
                            }
                            tc_fence_after();
                            // accumulators of groups gh and gh - 1
                            const uint32_t dh = tmem + (uint32_t)(2 * buf * OZ_BN), dl = dh + OZ_BN;
                            for (int kc = 0; kc < nkc; kc++) {
                                if (gh == 0) {
                                    stop = !wait();
                                    if (stop) break;
                                    mma(dh, sa, sb, OZ_IDESC, kc > 0);
                                    umma_commit(smem_u32(&empty[(g - 1) % OZ_STAGES]));
                                    continue;
                                }
                                stop = !wait();
                                if (stop) break;
                                uint32_t bprev = sb;
                                for (int p = 0; p <= gh; p++) {
                                    stop = !wait();
                                    if (stop) break;
                                    // both groups' products as one, where this stage's B follows the one before
                                    if (p < gh && sb == bprev + OZ_B_BYTES)
                                        mma(dh, sa, bprev, OZ_IDESC2, kc > 0 || p > 0);
                                    else {
                                        mma(dh, sa, bprev, OZ_IDESC, kc > 0 || p > 0);
                                        if (p < gh) mma(dl, sa, sb, OZ_IDESC, kc > 0 || p > 0);
                                    }
                                    bprev = sb;
                                    umma_commit(smem_u32(&empty[(g - 2) % OZ_STAGES]));  // the stage before: its B is done
                                }
                                if (stop) break;
                                umma_commit(smem_u32(&empty[(g - 1) % OZ_STAGES]));
                            }
                            if (!stop) umma_commit(smem_u32(&afull[buf]));
                        }
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(OZ_REPI));
        // epilogue: the warp's TMEM lanes are 32*(warp % 4) .. +31 (rows of the tile), its columns a half
        const int ew = warp - 4, lb = (warp & 3) * 32, cb = (ew >> 2) * 64;
        const uint32_t trow = ((uint32_t)lb << 16) + (uint32_t)cb;
        long u = 0;
        bool stop = false;
        for (int t = blockIdx.x; t < a.ntiles && !stop; t += gridDim.x) {
            const int kb0 = a.tiles[t].z * a.kper, kb1 = min(a.nkb, kb0 + a.kper);
            f2 hs[32], ls[32];  // the row's double-float sums, columns in pairs
#pragma unroll
            for (int j = 0; j < 32; j++) hs[j] = ls[j] = 0ull;
            for (int kb = kb0; kb < kb1 && !stop; kb++) {
                for (int gh = oz_first_group(s); gh < s; gh += 2, u++) {
                    const int buf = (int)(u & 1);
                    const long use = u >> 1;
                    if (!mbar_wait(smem_u32(&afull[buf]), (uint32_t)(use & 1), abort_flag, OZ_WAIT)) {
                        if (!*abort_flag) { *abort_flag = 1; atomicCAS(a.err, 0, 3); }
                        stop = true;
                        break;
                    }
                    tc_fence_after();
#pragma unroll 1
                    for (int gi = gh > 0 ? 0 : 1; gi < 2; gi++) {
                        const float sc = __int_as_float((127 - 7 * (gh - 1 + gi)) << 23);
                        const f2 scale = pk(sc, sc);
                        const uint32_t ta = tmem + trow + (uint32_t)((2 * buf + 1 - gi) * OZ_BN);
#pragma unroll
                        for (int c0 = 0; c0 < 64; c0 += 32) {
                            uint32_t v[32];
                            tmem_ld32(ta + c0, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; j += 2)
                                df_add2(hs[(c0 + j) / 2], ls[(c0 + j) / 2],
                                        mul2(pk(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), scale));
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&aempty[buf]));
                }
            }
            if (stop) break;
            // the tile's result: C = beta C + alpha 2^{eA + eB - 12} (head + tail), or the
            // unscaled partial of this K split.  Each warp stages 32 rows x 32 columns of sums
            // in shared memory and writes them row by row, coalesced.  The scaled parts are built
            // as FP64 bit patterns, so an element costs one FP64 addition, and one more where
            // C is added to (conversions and scalings on the FP64 pipe made it six).
            const int4 tile = a.tiles[t];
            const int mrow = tile.x * OZ_BM + lb;
            const int em = (mrow + lane < a.M) ? a.ea[mrow + lane] - 12 : 0;
            const bool split = a.part != nullptr;
            float2 *st = stage + (size_t)ew * 32 * 32;
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 32) {
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    const float2 h = upk(hs[(c0 + j) / 2]), l = upk(ls[(c0 + j) / 2]);
                    st[lane * 32 + (j ^ lane)] = make_float2(h.x, l.x);
                    st[lane * 32 + ((j + 1) ^ lane)] = make_float2(h.y, l.y);
                }
                __syncwarp();
                const int n = tile.y * OZ_BN + cb + c0 + lane;
                const int en = (n < a.N) ? a.eb[n] : 0;
                // FORM 0: +-result or partial, 1: C +- result, 2: any alpha and beta.  The C values of
                // 16 rows are loaded together before any store (one round trip per 16 rows instead
                // of one per row)
                auto emit = [&](auto form, auto inside) {
                    constexpr int FORM = decltype(form)::value;
                    constexpr bool INSIDE = decltype(inside)::value;  // no element to leave out
                    const long ld = split ? a.N : a.ldc;
                    double *base = (split ? a.part + (size_t)tile.z * a.M * a.N : a.C) + (size_t)mrow * ld + n;
                    const unsigned long long sg = (!split && a.alpha < 0.0) ? 1ull << 63 : 0ull;
#pragma unroll 1
                    for (int r0 = 0; r0 < 32; r0 += 16, base += 16 * ld) {
                        double cv[16];
#pragma unroll
                        for (int rr = 0; rr < 16; rr++) {
                            const int mm = mrow + r0 + rr;
                            const bool ok = INSIDE || (mm < a.M && n < a.N && !(a.lower && n > mm));
                            cv[rr] = (FORM == 1 || (FORM == 2 && a.beta != 0.0)) && ok ? base[rr * ld] : 0.0;
                        }
#pragma unroll
                        for (int rr = 0; rr < 16; rr++) {
                            const int mm = mrow + r0 + rr, e = __shfl_sync(0xffffffffu, em, r0 + rr) + en;
                            const float2 x = st[(r0 + rr) * 32 + (lane ^ (r0 + rr))];
                            if (!INSIDE && (mm >= a.M || n >= a.N || (a.lower && n > mm))) continue;
                            double xh, xl, v;
                            const bool near = dfb::scaled(__float_as_uint(x.x), e, &xh) & dfb::scaled(__float_as_uint(x.y), e, &xl);
                            v = xh + xl;
                            if (!near) v = oz_join_far(x.x, x.y, e - en, en);
                            if (FORM < 2) v = __longlong_as_double((long long)((unsigned long long)__double_as_longlong(v) ^ sg));
                            if (FORM == 1) v = cv[rr] + v;
                            if (FORM == 2) v = fma(a.beta, cv[rr], a.alpha * v);
                            base[rr * ld] = v;
                        }
                    }
                };
                // (warp-uniform) every element of the 32 x 32 block is one of C's
                const int nl = tile.y * OZ_BN + cb + c0 + 31;
                const bool in = mrow + 31 < a.M && nl < a.N && !(a.lower && nl > mrow);
                constexpr std::integral_constant<bool, true> yes{};
                constexpr std::integral_constant<bool, false> no{};
                const bool unit = a.alpha == 1.0 || a.alpha == -1.0;
                if (split || (unit && a.beta == 0.0)) {
                    if (in) emit(std::integral_constant<int, 0>{}, yes);
                    else emit(std::integral_constant<int, 0>{}, no);
                } else if (unit && a.beta == 1.0) {
                    if (in) emit(std::integral_constant<int, 1>{}, yes);
                    else emit(std::integral_constant<int, 1>{}, no);
                } else
                    emit(std::integral_constant<int, 2>{}, no);
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, OZ_TMEM_COLS);
    }
}

// C = beta C + alpha sum_z part_z (K splits added in a fixed order).
__global__ void k_oz_reduce(int M, int N, int ks, const double *__restrict__ part, double alpha, double beta, double *C,
                            long ldc, int lower)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)M * N) return;
    const int m = (int)(e / N), n = (int)(e - (size_t)m * N);
    if (lower && n > m) return;
    double v = 0.0;
    for (int z = 0; z < ks; z++) v += part[(size_t)z * M * N + e];
    double *c = C + (size_t)m * ldc + n;
    *c = (beta == 0.0) ? alpha * v : fma(beta, *c, alpha * v);
}

// ------------------------------------------------------------------ host side
PFN_cuTensorMapEncodeTiled_v12000 g_oz_encode = nullptr;
std::mutex g_oz_mu;

modal_status oz_encoder()
{
    std::lock_guard<std::mutex> lock(g_oz_mu);
    if (g_oz_encode) return MODAL_OK;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
        set_error("cuTensorMapEncodeTiled unavailable: %s", cudaGetErrorString(e));
        return MODAL_ERR_CUDA;
    }
    g_oz_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return MODAL_OK;
}

// 2D FP16 map over [rows][Kpad], box [box_rows][64], 128-byte swizzle.
modal_status oz_map(CUtensorMap *m, const void *base, long rows, int Kpad, int box_rows)
{
    cuuint64_t dims[2] = {(cuuint64_t)Kpad, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)Kpad * 2};
    cuuint32_t box[2] = {(cuuint32_t)OZ_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_oz_encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return MODAL_ERR_CUDA; }
    return MODAL_OK;
}

}  // namespace

// C[M][N] (ld ldc) = beta C + alpha op(A) op(B), op(A) M x K, op(B) K x N, in
// FP64 accuracy class on the tensor cores with o.slices slices (2 <= s <= 8).
//   op(A)(m, k) = transA ? A[k*lda + m] : A[m*lda + k]
//   op(B)(k, n) = transB ? B[n*ldb + k] : B[k*ldb + n]
// o.lower: only entries with n <= m are written (square C); o.diag_tiles > 0:
// only the 128-row tiles (tm, tn) with tm / diag_tiles == tn / diag_tiles
// (the diagonal blocks of that many tiles); o.ksplit: K split over that many
// work items per tile (0: chosen to fill the GPU), partials added in order.
modal_status oz_slice(modal_ctx *ctx, int R, int K, const double *X, long ld, bool trans, int s, int Rpad, int Kpad,
                      __half *out, int *ex)
{
    if (Rpad % OZ_BM || Kpad % 64 || R > Rpad || K > Kpad || s < 2 || s > OZ_MAXS) {
        set_error("oz_slice: bad layout (R=%d Rpad=%d K=%d Kpad=%d s=%d)", R, Rpad, K, Kpad, s);
        return MODAL_ERR_ARG;
    }
    // K split into chunks (multiples of 32) so that the grid has about two CTAs per SM
    int nsm = 0;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    const int rb = Rpad / 32, want = std::max(1, ceil_div(2 * nsm, rb));
    const int kchunk = std::max(32, ceil_div(ceil_div(Kpad, want), 32) * 32);
    const int nkc = ceil_div(Kpad, kchunk);
    MODAL_CUDA(cudaMemsetAsync(ex, 0x80, sizeof(int) * (size_t)Rpad, ctx->stream));  // below every exponent
    k_oz_rowexp<<<dim3(rb, ceil_div(std::max(K, 1), kchunk)), 256, 0, ctx->stream>>>(R, K, kchunk, X, ld, trans ? 1 : 0,
                                                                                     ex);
    MODAL_TRY(launched(ctx, "oz_rowexp"));
    k_oz_slice<<<dim3(rb, nkc), 256, 0, ctx->stream>>>(R, K, Rpad, Kpad, kchunk, X, ld, trans ? 1 : 0, s, out, ex);
    return launched(ctx, "oz_slice");
}

modal_status oz_run(modal_ctx *ctx, const OzOperand &A, const OzOperand &B, int Kpad, int s,
                    const std::vector<int2> *tile_list, double alpha, double beta, double *C, long ldc, const OzOpts &o)
{
    const int M = A.rows, N = B.rows, Mpad = A.rows_pad, Npad = B.rows_pad;
    if (M <= 0 || N <= 0) return MODAL_OK;
    if (s < 2 || s > OZ_MAXS || Mpad % OZ_BM || Npad % OZ_BM || Kpad % 64 || Kpad <= 0) {
        set_error("oz_run: bad layout (Mpad=%d Npad=%d Kpad=%d s=%d)", Mpad, Npad, Kpad, s);
        return MODAL_ERR_ARG;
    }
    MODAL_TRY(oz_encoder());
    const int ntm = Mpad / OZ_BM, ntn = Npad / OZ_BN;
    const int nkb = ceil_div(Kpad, OZ_KB);
    int nsm = 0;
    MODAL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    std::vector<int2> own;
    if (!tile_list) {
        // tile order: column of tiles outer so that consecutive CTAs share B slices in L2
        for (int tn = 0; tn < ntn; tn++)
            for (int tm = 0; tm < ntm; tm++) {
                if (o.lower && tn > tm) continue;
                if (o.diag_tiles > 0 && tm / o.diag_tiles != tn / o.diag_tiles) continue;
                own.push_back(make_int2(tm, tn));
            }
    }
    const std::vector<int2> &base = tile_list ? *tile_list : own;
    if (base.empty()) return MODAL_OK;
    int ks = o.ksplit;
    if (ks <= 0) ks = (int)std::min<long>(nkb, std::max<long>(1, (long)nsm / std::max<size_t>(1, base.size())));
    ks = std::max(1, std::min(ks, nkb));
    const int kper = ceil_div(nkb, ks);
    ks = ceil_div(nkb, kper);
    std::vector<int4> tiles;
    tiles.reserve(base.size() * ks);
    for (int z = 0; z < ks; z++)
        for (const int2 &t : base) tiles.push_back(make_int4(t.x, t.y, z, 0));
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t off = 0;
    const size_t o_t = off; off += al(tiles.size() * sizeof(int4));
    const size_t o_p = off; off += (ks > 1) ? al((size_t)ks * M * N * 8) : 0;
    MODAL_TRY(ensure(ctx->ozrun, off));
    uint8_t *b = ctx->ozrun.as<uint8_t>();
    MODAL_TRY(ensure(ctx->ozerr, 256));
    int *err = ctx->ozerr.as<int>();
    MODAL_CUDA(cudaMemcpyAsync(b + o_t, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice, ctx->stream));
    if (o.check) MODAL_CUDA(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
    CUtensorMap ma, mb;
    MODAL_TRY(oz_map(&ma, A.slices, (long)s * Mpad, Kpad, OZ_BM));
    MODAL_TRY(oz_map(&mb, B.slices, (long)s * Npad, Kpad, OZ_BN));
    OzArgs g;
    g.M = M; g.N = N; g.Kpad = Kpad; g.Mpad = Mpad; g.Npad = Npad; g.s = s;
    g.nkb = nkb;
    g.kper = kper;
    g.ntiles = (int)tiles.size();
    g.lower = o.lower;
    g.tiles = reinterpret_cast<const int4 *>(b + o_t);
    g.part = ks > 1 ? reinterpret_cast<double *>(b + o_p) : nullptr;
    g.ea = A.ex; g.eb = B.ex; g.alpha = alpha; g.beta = beta; g.C = C; g.ldc = ldc; g.err = err;
    MODAL_CUDA(cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM));
    const int grid = std::max(1, std::min(g.ntiles, nsm));
    {
        StageTimer t(ctx, MODAL_T_TC);
        k_oz_gemm<<<grid, OZ_THREADS, OZ_SMEM, ctx->stream>>>(ma, mb, g);
        MODAL_TRY(launched(ctx, "oz_gemm"));
    }
    if (ks > 1) {
        k_oz_reduce<<<ceil_div((long)M * N, 256), 256, 0, ctx->stream>>>(M, N, ks, g.part, alpha, beta, C, ldc, o.lower);
        MODAL_TRY(launched(ctx, "oz_reduce"));
    }
    // unchecked calls leave the (sticky) error word for oz_check
    return o.check ? oz_check(ctx) : MODAL_OK;
}

modal_status oz_gemm_ex(modal_ctx *ctx, int M, int N, int K, double alpha, const double *A, long lda, bool transA,
                        const double *B, long ldb, bool transB, double beta, double *C, long ldc, const OzOpts &o)
{
    if (M <= 0 || N <= 0) return MODAL_OK;
    const int s = o.slices;
    if (s < 2 || s > OZ_MAXS) { set_error("oz_gemm: slices %d outside [2, %d]", s, OZ_MAXS); return MODAL_ERR_ARG; }
    if (K <= 0) {
        if (beta == 1.0) return MODAL_OK;
        set_error("oz_gemm: K = %d with beta != 1", K);
        return MODAL_ERR_ARG;
    }
    const int Mpad = ceil_div(M, OZ_BM) * OZ_BM, Npad = ceil_div(N, OZ_BN) * OZ_BN;
    const int Kpad = ceil_div(K, 64) * 64;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t off = 0;
    const size_t o_a = off; off += al((size_t)s * Mpad * Kpad * 2);
    const size_t o_b = off; off += al((size_t)s * Npad * Kpad * 2);
    const size_t o_ea = off; off += al((size_t)Mpad * 4);
    const size_t o_eb = off; off += al((size_t)Npad * 4);
    MODAL_TRY(ensure(ctx->ozw, off));
    uint8_t *b = ctx->ozw.as<uint8_t>();
    OzOperand oa{reinterpret_cast<__half *>(b + o_a), reinterpret_cast<int *>(b + o_ea), M, Mpad};
    OzOperand ob{reinterpret_cast<__half *>(b + o_b), reinterpret_cast<int *>(b + o_eb), N, Npad};
    MODAL_TRY(oz_slice(ctx, M, K, A, lda, transA, s, Mpad, Kpad, oa.slices, oa.ex));
    // columns of op(B) = rows of op(B)^T: transB ? B[n*ldb + k] (rows of B) : B[k*ldb + n] (columns of B)
    MODAL_TRY(oz_slice(ctx, N, K, B, ldb, !transB, s, Npad, Kpad, ob.slices, ob.ex));
    return oz_run(ctx, oa, ob, Kpad, s, nullptr, alpha, beta, C, ldc, o);
}

modal_status oz_reset(modal_ctx *ctx)
{
    MODAL_TRY(ensure(ctx->ozerr, 256));
    MODAL_CUDA(cudaMemsetAsync(ctx->ozerr.ptr, 0, sizeof(int), ctx->stream));
    return MODAL_OK;
}

modal_status oz_check(modal_ctx *ctx, bool *tail)
{
    if (!ctx->ozerr.ptr) return MODAL_OK;
    int h[2] = {0, 0};
    MODAL_CUDA(cudaMemcpyAsync(h, ctx->ozerr.ptr, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
    MODAL_CUDA(cudaStreamSynchronize(ctx->stream));
    if (tail) *tail = h[1] != 0;
    return oz_status(h[0]);
}

modal_status oz_status(int herr)
{
    if (herr) { set_error("a bounded wait in a tensor-core kernel expired (role %d: 1-4 Ozaki GEMM, 21 and 23 slab projection)", herr); return MODAL_ERR_TIMEOUT; }
    return MODAL_OK;
}

modal_status oz_gemm(modal_ctx *ctx, int M, int N, int K, double alpha, const double *A, long lda, bool transA,
                     const double *B, long ldb, bool transB, double beta, double *C, long ldc, int lower, int s)
{
    OzOpts o;
    o.lower = lower;
    o.slices = s;
    return oz_gemm_ex(ctx, M, N, K, alpha, A, lda, transA, B, ldb, transB, beta, C, ldc, o);
}

}  // namespace modal

using namespace modal;

extern "C" modal_status modal_gemm_f64(modal_ctx *c, int M, int N, int K, double alpha, const double *A, int transA,
                                       const double *B, int transB, double beta, double *C, int slices)
{
    if (!c || M < 1 || N < 1 || K < 1 || !A || !B || !C || slices < 2 || slices > OZ_MAXS) {
        set_error("modal_gemm_f64: bad arguments (M=%d N=%d K=%d slices=%d)", M, N, K, slices);
        return MODAL_ERR_ARG;
    }
    MODAL_CUDA(cudaSetDevice(c->device));
    const size_t na = (size_t)M * K, nb = (size_t)K * N, nc = (size_t)M * N;
    MODAL_TRY(ensure(c->scratch, sizeof(double) * (na + nb + nc)));
    double *dA = c->scratch.as<double>(), *dB = dA + na, *dC = dB + nb;
    MODAL_CUDA(cudaMemcpyAsync(dA, A, sizeof(double) * na, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(dB, B, sizeof(double) * nb, cudaMemcpyHostToDevice, c->stream));
    MODAL_CUDA(cudaMemcpyAsync(dC, C, sizeof(double) * nc, cudaMemcpyHostToDevice, c->stream));
    MODAL_TRY(oz_gemm(c, M, N, K, alpha, dA, transA ? M : K, transA != 0, dB, transB ? K : N, transB != 0, beta, dC, N, 0,
                      slices));
    MODAL_CUDA(cudaMemcpyAsync(C, dC, sizeof(double) * nc, cudaMemcpyDeviceToHost, c->stream));
    MODAL_CUDA(cudaStreamSynchronize(c->stream));
    return MODAL_OK;
}

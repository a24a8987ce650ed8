// project_f32.cu -- single-precision projection of many shapes, both operands of
// the k-contraction on the tcgen05 tensor cores (calculate_mode_3D,
// calculate_mode_3D.c:217-264, over the walk of tetrapyd_tools.c:104-142).
//
// The sum over the tetrapyd i <= j <= k is factorised per slab of the MIDDLE index j:
//   H_s[i][c] = sum_k f_s(i,j,k) q_c(k),   f = W(i,j,k) S_s(i,j,k)
//   F_s[a][c] = sum_i q_a(i) H_s[i][c]
//   B_s[b][a][c] = sum_j q_b(j) F_s[a][c],  beta_r = (1/6) sum of B over the orderings of mode r
// (beta sums B over all six orderings, so which leg the slab takes is free).  With j fixed every
// row i of one parity starts at the same k = j + (i & 1) and ends at min(i + j, lmax): a block of
// 128 such rows is an almost rectangular (row x k) tile, where slabs of fixed i give a band that
// is skewed by one lattice point per row (a 128-row block of the mean row, 167 points at
// l <= 2000, would be 77% padding; here the warps evaluate 13% more points than there are).
//
// One thread owns one row.  It walks k in chunks of 32 lattice points (m = k >> 1), evaluates f in
// FP32 from per-row coefficients in registers (separable: three packed FMAs per term and pair of
// points, the tables at k are the same for the whole warp and come from shared memory; bump: the
// three components of l - cL are linear in k), splits f into three BF16 pieces (8 significant bits
// each, exact) and writes them straight into tensor memory, where they are the A operand (M = 128
// rows) of tcgen05.mma kind::f16.  B (N = basis columns) holds q_c(k) as three BF16 pieces taken
// from FP64, laid out once per call as the shared-memory image, so a chunk is one contiguous bulk
// copy.  Six products (pieces a + b <= 4, numbered from 1) carry each product to about 2^-24.  The
// leading one, f1 q1, has its own FP32 accumulator per chunk: products of 8-bit pieces over 32
// points nearly fit 24 bits, so the tensor core's truncating accumulation loses next to nothing
// there; the other five share a second accumulator for the whole row, where a truncation is 2^-8 of
// that.  (Two TF32 pieces in one accumulator were tried first: 1.3e-7 from the FP64 beta at
// l <= 2000, P = 30, against 5e-8 of the FP32 FMAs this replaces.)  The row's thread adds every
// chunk's accumulator into its H row; F is folded on the CUDA cores once per 128 rows.  These sums are plain
// FP32 where a term meets no more roundings than on CUDA cores and compensated where it would (pf_plan).
//
// What bounds it: issue slots of the row warps (evaluation, split, fold) and, with 12 row warps per
// SM, the latencies between them; so every operand is fetched ahead (ring of three chunks, the
// next half's weights in registers, the fold's basis rows in shared memory) and A is handed over in
// halves of 16 points.  One CTA per SM: three teams (two for P > 32) of four row warps, each with its
// own items, and one warp per team that copies and issues; the row warps take registers over from
// the issuing warps (setmaxnreg 152 / 56 of 128), since a spill to this kernel's small L1 costs an
// L2 round trip.  (Whatever the fold keeps in registers through the passes moves the time by 5%.)  TMEM per team: 48 columns of A, two leading accumulators and one for the rest.
//
// Measured (l <= 2000, P = 30), against the CUDA-core kernel (136 warp instructions per 32 points)
// and the shared-memory-operand tensor-core kernel that it replaces both: 16 separable shapes 33.9 ->
// 15.9 ms, 256 mixed shapes 532 (CUDA cores), 1864 (tensor cores) -> 237 ms; error of beta against
// 64 bits, median and largest over the 128 bumps and 128 separable shapes: 7.5e-8, 8.9e-7 and
// 4.7e-8, 1.3e-7 -> 5.0e-8, 7.2e-7 and 2.5e-8, 4.6e-8.  (The largest was 2.7e-6, and the 256 shapes
// took 8 ms less, with the 1D factors of the weights and of the bumps' exponents rounded to FP32.)
#include <algorithm>
#include <vector>
#include <cuda_bf16.h>
#include "common.cuh"
#include "tc_ptx.cuh"

namespace modal {

namespace {

using namespace tc;

constexpr int PF_ROWS = 128;              // rows per block = tensor-memory lanes
constexpr int PF_KC = 32;                 // lattice points per chunk (two halves of 16)
constexpr int PF_TC = 4;                  // separable terms per pass (row coefficients in registers)
constexpr int PF_SLOTS = 3;               // ring of operand chunks
constexpr long long PF_WAIT = 2000000000LL;  // clock64 cycles, about 1 s

// One shape as the kernel reads it.
struct __align__(16) PfShape {
    // bump, read with the chunks: d/dk of the components of l - c L, (-c1, -c2, 1 - c3), as hi and lo,
    // and -log2(e) / (2 sigma^2), every value twice (packed operands)
    float2 bump[8];
    int kind, nterms;
    long tab_off;        // separable tables from this float offset (pf_tab)
    float ch[3], cl[3];  // bump centre as hi + lo
};

// Rows of slab j with parity p: i = i0 + 2r, r < nr, k = 2m + kp, m0 <= m <= min((i + j - kp) / 2, mtop).
struct PfClass {
    int i0, nr, kp, m0, mtop;
};

__host__ __device__ inline PfClass pf_class(int lmin, int lmax, int j, int p)
{
    PfClass c;
    c.i0 = lmin + ((lmin ^ p) & 1);
    c.nr = (j >= c.i0) ? (j - c.i0) / 2 + 1 : 0;
    c.kp = (j + p) & 1;
    c.m0 = (j + p - c.kp) >> 1;
    c.mtop = (lmax - c.kp) >> 1;
    if (c.m0 > c.mtop) c.nr = 0;
    return c;
}

// Last lattice point of row r of the class.
__host__ __device__ inline int pf_mlast(const PfClass &c, int j, int r)
{
    const int m = (c.i0 + 2 * r + j - c.kp) >> 1;
    return m < c.mtop ? m : c.mtop;
}

// Chunk origin (operand groups of 8 lattice points) and weight-table length (multiple of 8) of block b.
__host__ __device__ inline int pf_mstart(const PfClass &c) { return c.m0 & ~7; }
__host__ __device__ inline int pf_nm(const PfClass &c, int j, int b)
{
    const int last = c.nr - 1 < PF_ROWS * b + PF_ROWS - 1 ? c.nr - 1 : PF_ROWS * b + PF_ROWS - 1;
    return (pf_mlast(c, j, last) - pf_mstart(c) + 8) & ~7;
}

// Weight-table entries of slab j (units of PF_ROWS floats).
__host__ __device__ inline long long pf_slab_len(int lmin, int lmax, int j)
{
    long long n = 0;
    for (int p = 0; p < 2; p++) {
        const PfClass c = pf_class(lmin, lmax, j, p);
        for (int b = 0; b * PF_ROWS < c.nr; b++) n += pf_nm(c, j, b);
    }
    return n;
}

// 1D factors of the point weight, from FP64:
//   geo(l1,l2,l3) = gL(L) g(L - 2 l1) g(L - 2 l2) g(L - 2 l3) prod (2l+1), L = l1 + l2 + l3 (always even),
//   g(x) = sqrt(x + 1/6) / (x + 1/3), gL(L) = (L + 1/3) / (2 pi^2 (L + 1) sqrt(L + 1/6))
// (calculate_geometric.c:59-92 regrouped), v(l) = (2l+1)^{2/3} w_l (calculate_mode_3D.c:53-62).
// g[h] = g(2h), gl[h] = gL(2h), il2[h] = 1/(2h)^2 (bumps), as double-floats: a factor's rounding is
// shared by every point that uses it, and a sum that cancels does not average it away.
__device__ __forceinline__ void pf_tables(int h, int lmax, int nh, const double *__restrict__ cl, float2 *__restrict__ g,
                                          float2 *__restrict__ gl, float2 *__restrict__ il2, float2 *__restrict__ v)
{
    auto df = [](double x) {
        const float hi = (float)x;
        return make_float2(hi, (float)(x - (double)hi));
    };
    if (h < nh) {
        const double x = 2.0 * h;
        g[h] = df(sqrt(x + 1.0 / 6.0) / (x + 1.0 / 3.0));
        gl[h] = df((x + 1.0 / 3.0) / ((x + 1.0) * sqrt(x + 1.0 / 6.0)) * 0.0506605918211688857);
        il2[h] = df(h > 0 ? 1.0 / (x * x) : 0.0);
    }
    if (h <= lmax) v[h] = df((h < 2) ? 0.0 : cbrt(2.0 * h + 1.0) * sqrt(2.0 * h + 1.0) / sqrt(cl[h]));
}

// Product of double-floats, about 2^-46.
__device__ __forceinline__ float2 df_mul(float2 a, float2 b)
{
    const float p = a.x * b.x;
    return make_float2(p, fmaf(a.x, b.y, fmaf(a.y, b.x, fmaf(a.x, b.x, -p))));
}

// Point weights W(i,j,k) = permsix h~^2 prod (2l+1)^{-1/3} w_l of every row block, laid out
// [m / 4][128 rows][4], zero outside the rows.  grid (slabs, 2 parities x blocks); 128 threads.
// Bound by its writes (1.7 GB at l <= 2000); the factors are table look-ups instead of three
// divisions and a square root per point, multiplied as double-floats and rounded once.  Every v takes its
// geometric factor along: v ~ l^{5/6} C_l^{-1/2}, and the product of three alone leaves the FP32 range
// (C_l = 1e-19 at l = 2000) long before the weight does.
__global__ void __launch_bounds__(PF_ROWS) k_pf_weights(int lmin, int lmax, int nbmax, const long long *__restrict__ base,
                                                        const float2 *__restrict__ g, const float2 *__restrict__ gl,
                                                        const float2 *__restrict__ v, float4 *__restrict__ W)
{
    const int j = lmin + blockIdx.x, p = blockIdx.y / nbmax, b = blockIdx.y - p * nbmax;
    const PfClass c = pf_class(lmin, lmax, j, p);
    if (b * PF_ROWS >= c.nr) return;
    long long off = base[blockIdx.x];
    for (int pp = 0; pp < p; pp++) {
        const PfClass cc = pf_class(lmin, lmax, j, pp);
        for (int bb = 0; bb * PF_ROWS < cc.nr; bb++) off += pf_nm(cc, j, bb);
    }
    for (int bb = 0; bb < b; bb++) off += pf_nm(c, j, bb);
    const int r = b * PF_ROWS + threadIdx.x, nm = pf_nm(c, j, b), ms = pf_mstart(c);
    const bool valid = r < c.nr;
    const int i = c.i0 + 2 * (valid ? r : c.nr - 1);
    const int ml = valid ? pf_mlast(c, j, r) : -1;
    // v(i) with permsix, for k = j and for the others
    const float2 vj = v[j], vi1 = df_mul(v[i], make_float2(i == j ? 1.f : 3.f, 0.f)),
                 vi = df_mul(v[i], make_float2(i == j ? 3.f : 6.f, 0.f));
    float4 *o = W + off * (PF_ROWS / 4) + threadIdx.x;
    for (int m4 = 0; m4 < nm; m4 += 4) {
        float w[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int m = ms + m4 + x;
            w[x] = 0.f;
            if (m >= c.m0 && m <= ml) {
                const int k = 2 * m + c.kp;
                const float2 f = df_mul(df_mul(df_mul(df_mul(gl[(i + j + k) >> 1], g[(j + k - i) >> 1]), k == j ? vi1 : vi),
                                               df_mul(g[(k + i - j) >> 1], vj)),
                                        df_mul(g[(i + j - k) >> 1], v[k]));
                w[x] = f.x + f.y;
            }
        }
        o[(size_t)(m4 / 4) * PF_ROWS] = make_float4(w[0], w[1], w[2], w[3]);
    }
}

// B operand image: [parity kp][m / 8][piece][column c < NC][8] BF16 pieces of q_c(2m + kp), zero
// outside the basis; and the padded FP32 basis rows of the slab reduction, qp[l - lmin][NC], and of
// the fold, qt[parity of l][l / 2][NC] (rows outside the basis zero).
__device__ __forceinline__ void pf_basis(long e, int lmin, int lmax, int P, int NC, int M8, int QR,
                                         const double *__restrict__ q, __nv_bfloat16 *__restrict__ Bt, float *__restrict__ qp,
                                         float *__restrict__ qt)
{
    const int c = (int)(e % NC);
    const long x = e / NC;
    if (x < 2L * M8 * 8) {
        const int kp = (int)(x / (M8 * 8)), m = (int)(x % (M8 * 8)), k = 2 * m + kp;
        double v = (k >= lmin && k <= lmax && c < P) ? q[(size_t)(k - lmin) * P + c] : 0.0;
        __nv_bfloat16 *o = Bt + (((size_t)kp * M8 + m / 8) * 3 * NC + c) * 8 + (m & 7);
        for (int pc = 0; pc < 3; pc++) {
            const __nv_bfloat16 h = __double2bfloat16(v);
            o[(size_t)pc * NC * 8] = h;
            v -= (double)__bfloat162float(h);
        }
    }
    if (x <= lmax - lmin) qp[(size_t)x * NC + c] = (c < P) ? (float)q[(size_t)x * P + c] : 0.f;
    if (x < 2L * QR) {
        const int l = 2 * (int)(x % QR) + (int)(x / QR);
        qt[(size_t)x * NC + c] = (l >= lmin && l <= lmax && c < P) ? (float)q[(size_t)(l - lmin) * P + c] : 0.f;
    }
}

__device__ __forceinline__ PfShape pf_shape(const DShape &d)
{
    PfShape f;
    f.kind = d.kind;
    f.nterms = d.nterms;
    f.tab_off = d.tab_off_f;
    // a centre beyond 2^40 is brought down to it together with the width (l / L, at most 1, no longer counts there),
    // so that the squares below stay in the FP32 range
    double c[3] = {d.c1, d.c2, d.c3}, cm = 0.0;
    for (int a = 0; a < 3; a++) {
        if (isinf(c[a])) c[a] = copysign(1e300, c[a]);
        cm = fmax(cm, fabs(c[a]));
    }
    const int down = cm > 0x1p40 ? ilogb(cm) - 40 : 0;
    const double sigma = ldexp(d.sigma, -down);
    for (int a = 0; a < 3; a++) {
        c[a] = ldexp(c[a], -down);
        f.ch[a] = (float)c[a];
        f.cl[a] = (float)(c[a] - (double)f.ch[a]);
        const double b = (a == 2 ? 1.0 : 0.0) - c[a];
        const float bh = (float)b, bl = (float)(b - (double)bh);
        f.bump[2 * a] = make_float2(bh, bh);
        f.bump[2 * a + 1] = make_float2(bl, bl);
    }
    // (a width below 1e-13 is a point: its exponent is bounded, and its tail left out before it could overflow)
    const double ce = fmax(-1.4426950408889634074 / (2.0 * sigma * sigma), -1e25);
    const float ceh = (float)ce, cel = ce < -1e20 ? 0.f : (float)(ce - (double)ceh);
    f.bump[6] = make_float2(ceh, ceh);
    f.bump[7] = make_float2(cel, cel);
    return f;
}

// FP32 table of term t of a separable shape, re-laid from the FP64 [term][f, g, h][l] tables in groups of
// up to four terms (one pass each): group t0 at float offset 3 t0 * 2 * 8 H8, then
// [parity of l][l / 16][term of the group][f, g, h][8]: a chunk of 32 lattice points is contiguous
// and four consecutive points of one factor are one 16-byte load.  tmax[term][f, g, h]: the bits of the
// largest |factor| at l_min .. l_max (infinities and NaN above every number).  One block of 256 threads.
__device__ __forceinline__ void pf_tab(int t, int lmin, int lmax, int H8, const DShape &d, const double *__restrict__ tab64,
                                       float *__restrict__ tabf, unsigned *__restrict__ tmax)
{
    __shared__ unsigned mx[3];
    if (threadIdx.x < 3) mx[threadIdx.x] = 0u;
    __syncthreads();
    const int stride = lmax + 1, t0 = t & ~(PF_TC - 1), ng = min(PF_TC, d.nterms - t0);
    const double *f = tab64 + d.tab_off + (long)t * 3 * stride;
    unsigned b[3] = {0u, 0u, 0u};
    for (int l = threadIdx.x; l < 16 * H8; l += 256) {
        const int m = l >> 1;
        float *o = tabf + d.tab_off_f + (size_t)3 * t0 * 16 * H8 +
                   ((((size_t)(l & 1) * H8 + (m >> 3)) * ng + (t - t0)) * 3) * 8 + (m & 7);
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float v = l <= lmax ? (float)f[x * stride + l] : 0.f;
            o[8 * x] = v;
            if (l >= lmin) b[x] = max(b[x], __float_as_uint(v) & 0x7fffffffu);
        }
    }
#pragma unroll
    for (int x = 0; x < 3; x++) {
        const unsigned w = __reduce_max_sync(0xffffffffu, b[x]);
        if ((threadIdx.x & 31) == 0) atomicMax(mx + x, w);
    }
    __syncthreads();
    if (threadIdx.x < 3) tmax[d.tab_off / stride + 3 * t + threadIdx.x] = mx[threadIdx.x];
}

// What the weights and the slab kernel read, in one launch (four of their own made small batches
// slower): blocks for the 1D factors, for the basis, and one per shape and term.
struct PfSetup {
    int lmin, lmax, P, NC, M8, QR, nh, maxt, nbt, nbb;
    const double *cl, *q, *tab64;
    const DShape *desc;
    float2 *g, *gl, *il2, *v;
    __nv_bfloat16 *Bt;
    float *qp, *qt, *tabf;
    unsigned *tmax;
    PfShape *shapes;
};
__global__ void __launch_bounds__(256) k_pf_setup(const PfSetup a)
{
    int b = blockIdx.x;
    if (b < a.nbt) {
        pf_tables(b * 256 + threadIdx.x, a.lmax, a.nh, a.cl, a.g, a.gl, a.il2, a.v);
        return;
    }
    b -= a.nbt;
    if (b < a.nbb) {
        pf_basis((long)b * 256 + threadIdx.x, a.lmin, a.lmax, a.P, a.NC, a.M8, a.QR, a.q, a.Bt, a.qp, a.qt);
        return;
    }
    b -= a.nbb;
    const int s = b / a.maxt, t = b - s * a.maxt;
    const DShape d = a.desc[s];
    if (d.kind == MODAL_SHAPE_SEPARABLE && t < d.nterms) pf_tab(t, a.lmin, a.lmax, a.M8, d, a.tab64, a.tabf, a.tmax);
    if (t == 0 && threadIdx.x == 0) a.shapes[s] = pf_shape(d);
}

// ---- PTX of this kernel -------------------------------------------------

__device__ __forceinline__ void tmem_st4(uint32_t t, const uint32_t *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3])
                 : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t t, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(t));
}

// D (tensor memory) (+)= A (tensor memory, 128 x 16 BF16) B (shared memory, K-major)
__device__ __forceinline__ void umma_bf16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// Bounded wait for a phase, suspended rather than spinning (a spinning warp takes issue slots from the
// row warps): false when the budget ran out or another role aborted.
__device__ __forceinline__ bool pf_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(100000u)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    if (pf_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!pf_try(bar, parity))
        if (*abort_flag || clock64() - t0 > PF_WAIT) return false;
    return true;
}

// packed FP32 pairs
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Kahan sum: hi - lo += x
__device__ __forceinline__ void kahan2(f2 &hi, f2 &lo, f2 x)
{
    const f2 y = sub2(x, lo), t = add2(hi, y);
    lo = sub2(sub2(t, hi), y);
    hi = t;
}

// Shared-memory descriptor, K-major without swizzle: core matrices of 8 rows x 16 bytes, `lbo`
// bytes between neighbours along K and `sbo` along N.
__device__ __forceinline__ uint64_t desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           ((uint64_t)1 << 46);
}

// Contiguous global -> shared copy (both 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// A weight-table entry: read once per shape, kept out of L1.
__device__ __forceinline__ float4 ld_w(const float4 *p)
{
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Barrier `id` over a team's 128 row threads; returns the OR of v over them.
__device__ __forceinline__ bool rows_bar_or(int id, bool v)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(id)
        : "memory");
    return r != 0;
}

// ---- the slab kernel ----------------------------------------------------

struct PfArgs {
    int lmin, lmax, P, S, SG, G, nitems, M8, QR, teams;
    uint32_t team_smem;        // bytes of a team's shared memory
    const int *order;          // slabs, heaviest first
    const long long *base;     // [L] weight-table offset of each slab (units of 128 floats)
    const PfShape *shapes;
    const float *tabf;
    const float2 *il2;
    const float4 *W;
    const __nv_bfloat16 *Bt;
    const float *qt;
    float *Fbuf;               // [S][L][P*P]
    float *Flo;                // CAREFUL: [CTA][team][SG][tiles per thread][16][128] corrections of F (hi in shared memory)
    int grp, comp;             // rows that the fold adds plainly; whether it compensates the sum of such groups
    int *err;
};

// Item `it` of team `team` (of all CTAs' teams): (slab, shape group), heaviest slabs first, dealt
// out back and forth so that every team gets the same share.
__device__ __forceinline__ int pf_item(const PfArgs &a, int team, int it)
{
    const int n = (int)gridDim.x * a.teams, r = team * (int)gridDim.x + (int)blockIdx.x;
    return it * n + ((it & 1) ? n - 1 - r : r);
}

// This thread's corrections of tile x (of SG tpt) of F.
__device__ __forceinline__ float *pf_flo(const PfArgs &a, int x, int tpt)
{
    return a.Flo + ((size_t)(blockIdx.x * a.teams + (threadIdx.x >> 7)) * a.SG * tpt + x) * 16 * 128 + (threadIdx.x & 127);
}

// The passes of a team in order (items x parities x row blocks x shapes x groups of terms, as the row
// threads' nested loops), walked by the issuing thread for its copies: chunks left in the pass and
// the next chunk's sources.
struct PfWalk {
    int left;                   // chunks of the current pass not yet copied (0: the sequence is over)
    uint32_t tb, tstep;         // bytes of the tables per chunk, step to the next chunk's
    const uint8_t *bsrc, *tsrc;
    int team, it, s0, sgv, j, p, b, sx, ps, np;
    __device__ __forceinline__ void start(const PfArgs &a, int t, int nc)
    {
        team = t;
        it = -1;
        p = 2;
        sgv = sx = ps = np = b = 0;
        pass(a, nc);
    }
    // the next pass
    __device__ __forceinline__ void pass(const PfArgs &a, int nc)
    {
        left = 0;
        PfClass c;
        if (++ps >= np) {
            ps = 0;
            sx++;
        }
        if (sx >= sgv) {
            sx = 0;
            b++;
        }
        for (;;) {
            bool found = false;
            for (; p < 2; p++, b = 0) {
                c = pf_class(a.lmin, a.lmax, j, p);
                if (b * PF_ROWS < c.nr) { found = true; break; }
            }
            if (found) break;
            const int w = pf_item(a, team, ++it);
            if (w >= a.nitems) return;
            s0 = (w % a.G) * a.SG;
            sgv = min(a.SG, a.S - s0);
            j = a.lmin + a.order[w / a.G];
            p = b = sx = ps = 0;
        }
        const PfShape &sh = a.shapes[s0 + sx];
        const int g0 = pf_mstart(c) >> 3, nterms = sh.kind == MODAL_SHAPE_SEPARABLE ? sh.nterms : 0;
        np = max(1, (nterms + PF_TC - 1) / PF_TC);
        left = (pf_nm(c, j, b) + PF_KC - 1) / PF_KC;
        bsrc = reinterpret_cast<const uint8_t *>(a.Bt) + ((size_t)c.kp * a.M8 + g0) * (48 * nc);
        if (nterms > 0) {
            const int t0 = PF_TC * ps, ng = min(PF_TC, nterms - t0);
            tb = tstep = 4u * ng * 96;
            tsrc = reinterpret_cast<const uint8_t *>(a.tabf + sh.tab_off + (size_t)3 * t0 * 16 * a.M8 +
                                                     ((size_t)c.kp * a.M8 + g0) * ng * 24);
        } else {
            tb = sizeof(float2) * 8;
            tstep = 0;
            tsrc = reinterpret_cast<const uint8_t *>(sh.bump);
        }
    }
};

// Row state of a row block.
struct PfRow {
    int b;              // the row block
    int i;              // this thread's row
    int mlw;            // the end of the warp's longest row (-1: no rows)
};

// Chunk geometry in shared and tensor memory.
template <int NC>
struct PfMem {
    static constexpr uint32_t BCH = 4u * 3 * NC * 16;             // B chunk: 4 groups of 8 points x 3 pieces x NC x 16 B
    static constexpr uint32_t TCH = 4u * PF_TC * 3 * 8 * 4;       // tables of one chunk, up to four terms
    static constexpr uint32_t SLOT = BCH + TCH;
    static constexpr uint32_t QB = PF_ROWS * NC * 4;              // basis rows of a row block
    static constexpr int HLD = NC + 4;                            // floats per staged H row (16-byte aligned, conflict-free)
    static constexpr uint32_t D0 = 48;                            // after two halves of A, three pieces of 8 columns each
    static constexpr uint32_t D1 = D0 + 2 * NC;                   // two leading accumulators, then the other products
    static constexpr int TEAMS = D1 + NC <= 160 ? 3 : 2;
    static constexpr uint32_t TCOLS = TEAMS == 3 ? 160 : 256;     // tensor-memory columns of a team
    static constexpr int THREADS = 128 * (TEAMS + 1);
    static constexpr int RROW = TEAMS == 3 ? 152 : 216, RAUX = TEAMS == 3 ? 56 : 72;
    static_assert(TEAMS * RROW + RAUX <= (TEAMS + 1) * (TEAMS == 3 ? 128 : 168), "registers of the launch");
    // kind::f16, D = F32, A = B = BF16, both K-major, M = 128, N = NC
    static constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NC >> 3) << 17) | ((128u >> 4) << 24);
    static_assert(D1 + NC <= TCOLS, "tensor memory");
};

// Barriers and flags of a team, in shared memory.
struct PfSync {
    uint64_t full[PF_SLOTS];  // operand chunk landed
    uint64_t ready[2];        // A half written (four warps)
    uint64_t done[2];         // products of a half complete
    uint64_t qfull;           // basis rows of the row block landed
    int abort_flag;
    uint32_t tmem;
    int first[2];             // row threads -> issuing thread, per chunk parity: PF_PASS, PF_BLOCK, PF_END
    int qrow;                 // first basis row of the new row block
};
static_assert(PfMem<16>::THREADS == PfMem<32>::THREADS && PfMem<48>::THREADS == PfMem<64>::THREADS, "launch shape");
enum { PF_PASS = 1, PF_BLOCK = 2, PF_END = 4 };  // the chunk opens a pass, a row block; no more chunks

// Position in the team's chunk sequence.
struct PfPos {
    uint32_t cc;      // chunks so far
    int slot;         // cc mod PF_SLOTS
    uint32_t phase;   // parity of cc / PF_SLOTS
    __device__ __forceinline__ void next()
    {
        cc++;
        if (++slot == PF_SLOTS) { slot = 0; phase ^= 1; }
    }
};

// Adds an accumulator's columns of this thread's row to H; CAREFUL: with Kahan's compensation in lo[NC] (the
// thread's row of the fold's shared memory, idle during a pass).  With it always, 16 and 256 shapes at l <= 2000,
// P = 30 took 17.4 and 268 ms instead of 16.0 and 234.
template <int NC, bool CAREFUL>
__device__ __forceinline__ void pf_drain(uint32_t t, f2 (&H)[NC / 2], float *lo)
{
    constexpr int CH = CAREFUL && NC <= 32 ? 16 : NC <= 32 ? NC : NC / 2;  // columns per round trip
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += CH) {
        uint32_t r[CH];
#pragma unroll
        for (int x = 0; x < CH; x += 8) tmem_ld8(t + c0 + x, &r[x]);
        tmem_wait_ld();
        if (CAREFUL) {
#pragma unroll
            for (int x = 0; x < CH; x += 4) {
                ulonglong2 l = *reinterpret_cast<ulonglong2 *>(lo + c0 + x);
                kahan2(H[(c0 + x) / 2], l.x, pk(__uint_as_float(r[x]), __uint_as_float(r[x + 1])));
                kahan2(H[(c0 + x) / 2 + 1], l.y, pk(__uint_as_float(r[x + 2]), __uint_as_float(r[x + 3])));
                *reinterpret_cast<ulonglong2 *>(lo + c0 + x) = l;
            }
        } else {
#pragma unroll
            for (int x = 0; x < CH / 2; x++)
                H[c0 / 2 + x] = add2(H[c0 / 2 + x], pk(__uint_as_float(r[2 * x]), __uint_as_float(r[2 * x + 1])));
        }
    }
}

// One pass of a row block: a bump (nt = 0), or nt = 1..4 terms of a separable shape from term t0 on.
// CAREFUL: the points past a row's end are masked and the row sums compensated.
template <int NC, bool CAREFUL>
__device__ __forceinline__ bool pf_pass(const PfArgs &a, const PfShape &sh, int t0, int nt, int j, const PfClass &c,
                                        const PfRow &rw, int nch, bool block, const float4 *__restrict__ Wrow, const uint8_t *sm, PfSync *sy,
                                        uint32_t tA, uint32_t tD1, PfPos &pos, f2 (&H)[NC / 2], float *lo)
{
    using M = PfMem<NC>;
    const uint32_t ready = smem_u32(sy->ready), done = smem_u32(sy->done), full = smem_u32(sy->full);
    volatile int *abort_flag = &sy->abort_flag;
    const int lane = threadIdx.x & 31, ms = pf_mstart(c);
    const int ml = CAREFUL ? pf_mlast(c, j, min(PF_ROWS * rw.b + (int)(threadIdx.x & 127), c.nr - 1)) : 0;
    // the first half's weights
    float4 w[4];
#pragma unroll
    for (int g4 = 0; g4 < 4; g4++)
        if (ms + 8 * (g4 >> 1) <= rw.mlw) w[g4] = ld_w(Wrow + (size_t)g4 * PF_ROWS);
    // row coefficients, as packed pairs: with f, g, h of each term at k, or (hi, lo) of the components
    f2 co[3 * PF_TC];
    const float2 *i2 = a.il2 + ((rw.i + j + c.kp) >> 1);
    if (nt > 0) {
        const float *tab = a.tabf + sh.tab_off + (size_t)3 * t0 * 16 * a.M8;
        const float *ti = tab + (((size_t)(rw.i & 1) * a.M8 + (rw.i >> 4)) * nt * 3) * 8 + ((rw.i >> 1) & 7);
        const float *tj = tab + (((size_t)(j & 1) * a.M8 + (j >> 4)) * nt * 3) * 8 + ((j >> 1) & 7);
#pragma unroll
        for (int t = 0; t < PF_TC; t++)
            if (t < nt) {
                const float fi = __ldg(ti + 24 * t), gi = __ldg(ti + 24 * t + 8), hi = __ldg(ti + 24 * t + 16);
                const float fj = __ldg(tj + 24 * t), gj = __ldg(tj + 24 * t + 8), hj = __ldg(tj + 24 * t + 16);
                const float x = (fi * gj + gi * fj) * (1.f / 6.f), y = (fi * hj + hi * fj) * (1.f / 6.f),
                            z = (gi * hj + hi * gj) * (1.f / 6.f);
                co[3 * t] = pk(z, z);
                co[3 * t + 1] = pk(y, y);
                co[3 * t + 2] = pk(x, x);
            }
    } else {
        // component m of l - c L at k = 0: l_m - c_m (i + j)
        const float s = (float)(rw.i + j), l3[3] = {(float)rw.i, (float)j, 0.f};
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float ch = sh.ch[x], pr = ch * s, pe = fmaf(ch, s, -pr);
            const float d = l3[x] - pr, bb = d - l3[x];
            const float e = (l3[x] - (d - bb)) - (pr + bb);
            const float al = e - pe - sh.cl[x] * s;
            co[2 * x] = pk(d, d);
            co[2 * x + 1] = pk(al, al);
        }
    }
#pragma unroll 1
    for (int n = 0; n < nch; n++, pos.next()) {
        const uint32_t cc = pos.cc;
        if ((threadIdx.x & 127) == 0) {
            sy->first[cc & 1] = n > 0 ? 0 : (block ? PF_PASS | PF_BLOCK : PF_PASS);
            if (n == 0 && block) sy->qrow = c.i0 + 2 * PF_ROWS * rw.b;
        }
        if (!pf_wait(full + 8 * pos.slot, pos.phase, abort_flag)) return false;
        const ulonglong2 *T0 = reinterpret_cast<const ulonglong2 *>(sm + pos.slot * M::SLOT + M::BCH);
        // chunk cc - 2 was complete before this thread wrote the second half of cc - 1; its accumulator is
        // overwritten by the products of this chunk
        if (n >= 2) pf_drain<NC, CAREFUL>(tA + M::D0 + NC * (cc & 1), H, lo);
#pragma unroll 1
        for (int hf = 0; hf < 2; hf++) {
            if (cc > 0) {  // the products that read this half a chunk ago are done
                if (!pf_wait(done + 8 * hf, (cc - 1) & 1, abort_flag)) return false;
                tc_fence_after();
            }
#pragma unroll
            for (int g8 = 0; g8 < 2; g8++) {
                const int mg = ms + PF_KC * n + 16 * hf + 8 * g8;
                uint32_t p1[4] = {0u, 0u, 0u, 0u}, p2[4] = {0u, 0u, 0u, 0u}, p3[4] = {0u, 0u, 0u, 0u};
                if (mg <= rw.mlw) {
                    f2 v[4];
                    if (nt > 0) {
                        const ulonglong2 *T = T0 + (size_t)(2 * hf + g8) * nt * 6;
#pragma unroll
                        for (int t = 0; t < PF_TC; t++)
                            if (t < nt) {
#pragma unroll
                                for (int x = 0; x < 3; x++) {
                                    const ulonglong2 q0 = T[(3 * t + x) * 2], q1 = T[(3 * t + x) * 2 + 1];
                                    const f2 q[4] = {q0.x, q0.y, q1.x, q1.y};
#pragma unroll
                                    for (int y = 0; y < 4; y++)
                                        v[y] = (t == 0 && x == 0) ? mul2(co[0], q[y]) : fma2(co[3 * t + x], q[y], v[y]);
                                }
                            }
                    } else {
                        const float k0 = (float)(2 * mg + c.kp);
                        const f2 kb = pk(k0, k0 + 2.f);
                        float2 il[8];
#pragma unroll
                        for (int y = 0; y < 8; y++) il[y] = __ldg(i2 + mg + y);
#pragma unroll
                        for (int x = 0; x < 3; x++) {
                            const ulonglong2 bb = T0[x];
#pragma unroll
                            for (int y = 0; y < 4; y++) {
                                const f2 kf = y == 0 ? kb : add2(kb, pk(4.f * y, 4.f * y));
                                const f2 d = add2(fma2(bb.x, kf, co[2 * x]), fma2(bb.y, kf, co[2 * x + 1]));
                                v[y] = x == 0 ? mul2(d, d) : fma2(d, d, v[y]);
                            }
                        }
                        const ulonglong2 ce = T0[3];
#pragma unroll
                        for (int y = 0; y < 4; y++) {
                            // r^2 / L^2 and the exponent, both constants with their tails
                            const float2 ia = il[2 * y], ib = il[2 * y + 1];
                            const f2 t = fma2(v[y], pk(ia.x, ib.x), mul2(v[y], pk(ia.y, ib.y)));
                            float e0, e1;
                            upk(fma2(t, ce.x, mul2(t, ce.y)), e0, e1);
                            v[y] = pk(ex2(e0), ex2(e1));
                        }
                    }
                    {
                        const float4 wa = w[2 * g8], wb = w[2 * g8 + 1];
                        v[0] = mul2(v[0], pk(wa.x, wa.y));
                        v[1] = mul2(v[1], pk(wa.z, wa.w));
                        v[2] = mul2(v[2], pk(wb.x, wb.y));
                        v[3] = mul2(v[3], pk(wb.z, wb.w));
                    }
                    if (mg < c.m0) {
                        // before the rows start (below lmin the caller's tables may hold anything); past a
                        // row's end the weight is zero and, unless CAREFUL, the shape finite
#pragma unroll
                        for (int y = 0; y < 4; y++) {
                            float v0, v1;
                            upk(v[y], v0, v1);
                            v[y] = pk(mg + 2 * y >= c.m0 ? v0 : 0.f, mg + 2 * y + 1 >= c.m0 ? v1 : 0.f);
                        }
                    }
                    if (CAREFUL) {
#pragma unroll
                        for (int y = 0; y < 4; y++) {
                            float v0, v1;
                            upk(v[y], v0, v1);
                            v[y] = pk(mg + 2 * y <= ml ? v0 : 0.f, mg + 2 * y + 1 <= ml ? v1 : 0.f);
                        }
                    }
                    // v = f1 + f2 + f3 exactly, 8 significant bits each (truncating splits)
#pragma unroll
                    for (int y = 0; y < 4; y++) {
                        const f2 m1 = pk(-1.f, -1.f);
                        float v0, v1;
                        upk(v[y], v0, v1);
                        p1[y] = __byte_perm(__float_as_uint(v0), __float_as_uint(v1), 0x7632);
                        f2 r = fma2(v[y] & 0xffff0000ffff0000ull, m1, v[y]);
                        upk(r, v0, v1);
                        p2[y] = __byte_perm(__float_as_uint(v0), __float_as_uint(v1), 0x7632);
                        r = fma2(r & 0xffff0000ffff0000ull, m1, r);
                        upk(r, v0, v1);
                        p3[y] = __byte_perm(__float_as_uint(v0), __float_as_uint(v1), 0x7632);
                    }
                }
                // the same group's weights one half on
                if (mg + 16 <= rw.mlw) {
                    w[2 * g8] = ld_w(Wrow + (size_t)((mg + 16 - ms) >> 2) * PF_ROWS);
                    w[2 * g8 + 1] = ld_w(Wrow + (size_t)(((mg + 16 - ms) >> 2) + 1) * PF_ROWS);
                }
                tmem_st4(tA + 24 * hf + 4 * g8, p1);
                tmem_st4(tA + 24 * hf + 8 + 4 * g8, p2);
                tmem_st4(tA + 24 * hf + 16 + 4 * g8, p3);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * hf);
        }
    }
    // the last two chunks, then the row's other products
    if (nch > 1) pf_drain<NC, CAREFUL>(tA + M::D0 + NC * (pos.cc & 1), H, lo);
    if (!pf_wait(done + 8, (pos.cc - 1) & 1, abort_flag)) return false;
    tc_fence_after();
    pf_drain<NC, CAREFUL>(tA + M::D0 + NC * ((pos.cc - 1) & 1), H, lo);
    pf_drain<NC, CAREFUL>(tD1, H, lo);
    tc_fence_before();
    return true;
}

template <int NC, bool CAREFUL>
__global__ void __launch_bounds__(PfMem<NC>::THREADS, 1) k_project_f32(const PfArgs a)
{
    using M = PfMem<NC>;
    extern __shared__ __align__(1024) uint8_t pf_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool aux = warp >= 4 * M::TEAMS;
    const int team = aux ? warp - 4 * M::TEAMS : warp >> 2;
    // a team's memory; idle teams and warps (the launch may use fewer teams) hold team 0's address and touch nothing
    const bool live = team < a.teams;
    uint8_t *pf_sm = pf_smem + (size_t)(live ? team : 0) * a.team_smem;
    float *Qs = reinterpret_cast<float *>(pf_sm + PF_SLOTS * M::SLOT);   // [128][NC] basis rows of the row block
    float *Hs = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(Qs) + M::QB);  // [128][HLD]
    PfSync *sy = reinterpret_cast<PfSync *>(Hs + PF_ROWS * M::HLD);
    float *Fs = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(sy) + 128);  // [SG][tiles per thread][16][128]
    static_assert(sizeof(PfSync) <= 128, "shared-memory layout");
    const int tid = threadIdx.x & 127;
    if (!aux && live && tid == 0) {
        for (int b = 0; b < PF_SLOTS; b++) mbar_init(smem_u32(&sy->full[b]), 1);
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&sy->ready[b]), 4);
            mbar_init(smem_u32(&sy->done[b]), 1);
        }
        mbar_init(smem_u32(&sy->qfull), 1);
        sy->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 * M::TEAMS) {
        tmem_alloc(smem_u32(&sy->tmem), 512);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem0 = reinterpret_cast<const PfSync *>(reinterpret_cast<const uint8_t *>(sy) - (pf_sm - pf_smem))->tmem;
    const uint32_t tmem = tmem0 + M::TCOLS * (uint32_t)(live ? team : 0), d1 = tmem + M::D1;
    bool stop = false;

    if (aux) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(M::RAUX));
        if (live && lane == 0) {
            volatile int *abort_flag = &sy->abort_flag;
            PfWalk ld;
            ld.start(a, team, NC);
            PfPos lp = {0u, 0, 0u}, mp = {0u, 0, 0u};
            const uint32_t sm0 = smem_u32(pf_sm), full = smem_u32(sy->full), ready = smem_u32(sy->ready),
                           done = smem_u32(sy->done);
            auto load = [&]() {  // the next chunk's B operand and tables
                const uint32_t dst = sm0 + lp.slot * M::SLOT, bar = full + 8 * lp.slot;
                mbar_expect_tx(bar, M::BCH + ld.tb);
                bulk_load(dst, ld.bsrc, M::BCH, bar);
                bulk_load(dst + M::BCH, ld.tsrc, ld.tb, bar);
                ld.bsrc += M::BCH;
                ld.tsrc += ld.tstep;
                lp.next();
                if (--ld.left == 0) ld.pass(a, NC);
            };
            for (int x = 0; x < PF_SLOTS - 1 && ld.left > 0; x++) load();
            const uint64_t desc0 = desc_plain(sm0, 48 * NC, 128);
            for (;; mp.next()) {
                const uint32_t cc = mp.cc;
                const uint32_t d0 = tmem + M::D0 + NC * (cc & 1);
                bool ok = pf_wait(ready, cc & 1, abort_flag);
                const int first = ok ? *(volatile int *)&sy->first[cc & 1] : PF_END;
                if (first & PF_END) { stop = !ok; break; }
                ok = pf_wait(full + 8 * mp.slot, mp.phase, abort_flag);
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    // at the second half also: chunk cc - 1 is complete (and cc cannot be yet)
                    if (hf == 1) {
                        ok = ok && pf_wait(ready + 8, cc & 1, abort_flag);
                        if (ok && cc > 0) ok = pf_wait(done + 8, (cc - 1) & 1, abort_flag);
                    }
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t b1 = desc0 + ((mp.slot * M::SLOT + hf * 96u * NC) >> 4), b2 = b1 + NC, b3 = b2 + NC;
                    const uint32_t ta = tmem + 24 * hf;
                    umma_bf16_ts(d0, ta, b1, M::IDESC, hf ? 1u : 0u);
                    umma_bf16_ts(d1, ta + 16, b1, M::IDESC, hf ? 1u : (uint32_t)!(first & PF_PASS));
                    umma_bf16_ts(d1, ta + 8, b2, M::IDESC, 1u);
                    umma_bf16_ts(d1, ta, b3, M::IDESC, 1u);
                    umma_bf16_ts(d1, ta + 8, b1, M::IDESC, 1u);
                    umma_bf16_ts(d1, ta, b2, M::IDESC, 1u);
                    umma_commit(done + 8 * hf);
                }
                if (!ok) {
                    if (!*abort_flag) { *abort_flag = 1; atomicCAS(a.err, 0, 21); }
                    stop = true;
                    break;
                }
                // chunk cc - 1's slot takes chunk cc + 2
                if (ld.left > 0) load();
                if (first & PF_BLOCK) {
                    // a new row block: every row warp is past the last fold, its basis rows come in
                    const int par = sy->qrow & 1, r0 = sy->qrow >> 1;
                    const uint32_t bytes = (uint32_t)min(PF_ROWS, a.QR - r0) * NC * 4;
                    mbar_expect_tx(smem_u32(&sy->qfull), bytes);
                    bulk_load(smem_u32(Qs), a.qt + ((size_t)par * a.QR + r0) * NC, bytes, smem_u32(&sy->qfull));
                }
            }
            if (stop) {
                // copies and products still in flight finish before shared and tensor memory are given back
                const long long t0 = clock64();
                while (clock64() - t0 < 20000000LL) {
                }
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(M::RROW));
        const int P = a.P, PP = P * P, L = a.lmax - a.lmin + 1, bar = 1 + team;
        const uint32_t tA = tmem + ((uint32_t)(tid & 96) << 16), tD1 = d1 + ((uint32_t)(tid & 96) << 16);
        // fold: 4 x 4 tiles of F, the 128 rows split over thread groups when there are few tiles
        const int nb4 = (P + 3) >> 2, nt = nb4 * nb4;
        const int ntp = nt <= 16 ? 16 : (nt <= 32 ? 32 : (nt <= 64 ? 64 : 128));
        const int rs = PF_ROWS / ntp, tpt = (nt + 127) / 128, rper = PF_ROWS / rs;
        PfPos pos = {0u, 0, 0u};
        uint32_t nq = 0;  // row blocks so far
        for (int it = 0; live && !stop; it++) {
            const int w = pf_item(a, team, it);
            if (w >= a.nitems) break;
            const int slab = a.order[w / a.G], s0 = (w % a.G) * a.SG, sgv = min(a.SG, a.S - s0), j = a.lmin + slab;
            for (int e = 0; e < sgv * tpt * 16; e++) Fs[e * 128 + tid] = 0.f;
            rows_bar_or(bar, false);  // a slab without rows (l_min = l_max odd) passes no other barrier before its sums
            long long woff = a.base[slab];
            for (int p = 0; p < 2 && !stop; p++) {
                const PfClass c = pf_class(a.lmin, a.lmax, j, p);
                for (int b = 0; b * PF_ROWS < c.nr && !stop; b++, nq++) {
                    const int nm = pf_nm(c, j, b), nch = (nm + PF_KC - 1) / PF_KC;
                    const int r = b * PF_ROWS + tid, rw0 = b * PF_ROWS + (tid & 96);
                    PfRow rw;
                    rw.b = b;
                    rw.i = c.i0 + 2 * min(r, c.nr - 1);
                    rw.mlw = rw0 < c.nr ? pf_mlast(c, j, min(rw0 + 31, c.nr - 1)) : -1;
                    const float4 *Wrow = a.W + woff * (PF_ROWS / 4) + tid;
                    for (int sx = 0; sx < sgv && !stop; sx++) {
                        const PfShape &sh = a.shapes[s0 + sx];
                        f2 H[NC / 2];
#pragma unroll
                        for (int x = 0; x < NC / 2; x++) H[x] = 0ull;
                        float *lo = CAREFUL ? Hs + tid * M::HLD : nullptr;
                        if (CAREFUL)
#pragma unroll
                            for (int x = 0; x < NC; x += 4) *reinterpret_cast<ulonglong2 *>(lo + x) = make_ulonglong2(0ull, 0ull);
                        bool ok = true;
                        const int nterms = sh.kind == MODAL_SHAPE_SEPARABLE ? sh.nterms : 0;
                        for (int t0 = 0; ok && (t0 == 0 || t0 < nterms); t0 += PF_TC)
                            ok = pf_pass<NC, CAREFUL>(a, sh, t0, min(PF_TC, nterms - t0), j, c, rw, nch, sx == 0 && t0 == 0, Wrow, pf_sm, sy, tA, tD1, pos, H, lo);
                        if (ok && sx == 0) ok = pf_wait(smem_u32(&sy->qfull), nq & 1, &sy->abort_flag);
                        if (!ok) { sy->abort_flag = 1; atomicCAS(a.err, 0, 23); }
                        // fold: F[a][c] += sum over the block's rows of q_a(i) H[i][c], in groups of rows (pf_plan)
#pragma unroll
                        for (int x = 0; x < NC / 2; x += 2)
                            *reinterpret_cast<ulonglong2 *>(Hs + tid * M::HLD + 2 * x) = make_ulonglong2(H[x], H[x + 1]);
                        stop = rows_bar_or(bar, !ok);
                        const int nrow = min(PF_ROWS, c.nr - b * PF_ROWS);
                        // the thread's number is read again, so that less of the fold stays in registers through the
                        // passes (not for 64 columns, which then spill)
                        int ft = threadIdx.x;
                        if (NC < 64) asm volatile("mov.u32 %0, %%tid.x;" : "=r"(ft));
                        for (int tt = 0; tt < tpt; tt++) {
                            const int tid = ft & 127;
                            const int ti = (tid & (ntp - 1)) + 128 * tt, sp = tid / ntp;
                            if (ti >= nt) break;
                            const int bt = ti / nb4, ct = ti - bt * nb4, rend = min(nrow, (sp + 1) * rper);
                            const float *qq = Qs + 4 * bt, *hq = Hs + 4 * ct;
                            float *f = Fs + (size_t)(sx * tpt + tt) * 16 * 128 + tid;
                            float *fl = CAREFUL ? pf_flo(a, sx * tpt + tt, tpt) : nullptr;
                            f2 hi[4][2], lk[4][2], acc[4][2];
#pragma unroll
                            for (int x = 0; x < 4; x++)
#pragma unroll
                                for (int y = 0; y < 2; y++) {
                                    hi[x][y] = lk[x][y] = 0ull;
                                    const int e = (4 * x + 2 * y) * 128;
                                    if (CAREFUL && woff != a.base[slab]) {  // (not the slab's first row block)
                                        hi[x][y] = pk(f[e], f[e + 128]);
                                        lk[x][y] = pk(fl[e], fl[e + 128]);
                                    }
                                }
#pragma unroll 1
                            for (int g = sp * rper; g < rend; g += a.grp) {
                                const int ge = min(g + a.grp, rend);
#pragma unroll
                                for (int x = 0; x < 4; x++) acc[x][0] = acc[x][1] = 0ull;
#pragma unroll 8
                                for (int q = g; q < ge; q++) {
                                    const float4 qv = *reinterpret_cast<const float4 *>(qq + q * NC);
                                    const ulonglong2 hv = *reinterpret_cast<const ulonglong2 *>(hq + q * M::HLD);
                                    const f2 qa[4] = {pk(qv.x, qv.x), pk(qv.y, qv.y), pk(qv.z, qv.z), pk(qv.w, qv.w)};
#pragma unroll
                                    for (int x = 0; x < 4; x++) {
                                        acc[x][0] = fma2(qa[x], hv.x, acc[x][0]);
                                        acc[x][1] = fma2(qa[x], hv.y, acc[x][1]);
                                    }
                                }
#pragma unroll
                                for (int x = 0; x < 4; x++)
#pragma unroll
                                    for (int y = 0; y < 2; y++) {
                                        if (CAREFUL || a.comp) kahan2(hi[x][y], lk[x][y], acc[x][y]);
                                        else hi[x][y] = add2(hi[x][y], acc[x][y]);
                                    }
                            }
#pragma unroll
                            for (int x = 0; x < 4; x++)
#pragma unroll
                                for (int y = 0; y < 2; y++) {
                                    const int e = (4 * x + 2 * y) * 128;
                                    if (CAREFUL) {
                                        upk(hi[x][y], f[e], f[e + 128]);
                                        upk(lk[x][y], fl[e], fl[e + 128]);
                                    } else {
                                        float v0, v1;
                                        upk(sub2(hi[x][y], lk[x][y]), v0, v1);
                                        f[e] += v0;
                                        f[e + 128] += v1;
                                    }
                                }
                        }
                        stop = rows_bar_or(bar, stop);  // Hs is read before the next pass writes it
                    }
                    woff += nm;
                }
            }
            if (stop) break;
            // (the last barrier passed orders the other threads' sums)
            // One entry per thread and step: with a tile's sixteen by the thread that folds it, few tiles left 16 of
            // the 128 threads to write all (15,000 cycles a work item at P = 6).
            for (int sx = 0; sx < sgv; sx++)
                for (int tt = 0; tt < tpt; tt++) {
                    const float *F = Fs + (size_t)(sx * tpt + tt) * 16 * 128;
                    const float *L0 = CAREFUL ? pf_flo(a, sx * tpt + tt, tpt) - tid : nullptr;
                    const bool corr = CAREFUL && woff != a.base[slab];  // (a slab without rows has no corrections)
                    float *dst = a.Fbuf + ((size_t)(s0 + sx) * L + slab) * PP;
                    for (int u = tid; u < 16 * ntp; u += 128) {
                        const int t0 = u & (ntp - 1), xy = u / ntp, ti = t0 + 128 * tt;
                        const int bt = ti / nb4, bb = 4 * bt + (xy >> 2), c2 = 4 * (ti - bt * nb4) + (xy & 3);
                        if (ti >= nt || bb >= P || c2 >= P) continue;
                        float v = 0.f, lo = 0.f;
                        for (int q = 0; q < rs; q++) {
                            const int e = xy * 128 + t0 + q * ntp;
                            if (CAREFUL) {
                                const float z = F[e] - lo, t = v + z;
                                lo = (t - v) - z;
                                v = t;
                                if (corr) lo += L0[e];
                            } else
                                v += F[e];
                        }
                        dst[bb * P + c2] = v - lo;
                    }
                }
            stop = rows_bar_or(bar, false);  // the sums are read before the next item clears them
        }
        if (live && !stop) {  // no more chunks
            if (tid == 0) sy->first[pos.cc & 1] = PF_END;
            rows_bar_or(bar, false);
            if (lane == 0) mbar_arrive(smem_u32(&sy->ready[0]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 4 * M::TEAMS) {
        tc_fence_after();
        tmem_dealloc(tmem0, 512);
    }
}

// B[seg][s][b][ac] = sum over the slabs of segment seg of q_b(j) F_s[j][ac], FP32 products with
// Kahan sums.  One thread keeps PB sums of one (s, ac), so F is read ceil(P / PB) times.
constexpr int PB = 8;
__global__ void __launch_bounds__(128) k_pf_B(int L, int P, int S, int NC, int nseg, const float *__restrict__ qp,
                                              const float *__restrict__ Fbuf, double *__restrict__ B)
{
    const int PP = P * P, e = blockIdx.x * 128 + threadIdx.x, s = blockIdx.y;
    const int nbg = (P + PB - 1) / PB, seg = blockIdx.z / nbg, b0 = (blockIdx.z - seg * nbg) * PB;
    if (e >= PP) return;
    const int per = (L + nseg - 1) / nseg, l0 = seg * per, l1 = min(L, l0 + per);
    const float *F = Fbuf + (size_t)s * L * PP + e;
    float hi[PB], lo[PB];
#pragma unroll
    for (int x = 0; x < PB; x++) hi[x] = lo[x] = 0.f;
#pragma unroll 4
    for (int l = l0; l < l1; l++) {
        const float f = F[(size_t)l * PP];
        const float4 q0 = __ldg(reinterpret_cast<const float4 *>(qp + (size_t)l * NC + b0));
        const float4 q1 = __ldg(reinterpret_cast<const float4 *>(qp + (size_t)l * NC + b0 + 4));
        const float q[PB] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int x = 0; x < PB; x++) {
            const float y = fmaf(q[x], f, -lo[x]);
            const float t = hi[x] + y;
            lo[x] = (t - hi[x]) - y;
            hi[x] = t;
        }
    }
#pragma unroll
    for (int x = 0; x < PB; x++)
        if (b0 + x < P) B[(((size_t)seg * S + s) * P + b0 + x) * PP + e] = (double)hi[x] - (double)lo[x];
}

// beta[s][r] = (1/6) sum over the segments and the six orderings of mode r of B.  *tail: whether (raise) a
// separable shape may leave the FP32 range at some (l1, l2, l3): its value is at most the sum over the terms of
// max|f| max|g| max|h| (pf_tab's maxima).
__global__ void k_pf_beta(int N, int P, int S, int nseg, const int *__restrict__ triples, const double *__restrict__ B,
                          double *__restrict__ beta, int lmax, const DShape *__restrict__ desc,
                          const unsigned *__restrict__ tmax, bool raise, int *__restrict__ tail)
{
    if (blockIdx.x == 0) {
        bool far = false;
        for (int s = threadIdx.x; raise && s < S; s += blockDim.x) {
            const DShape d = desc[s];
            if (d.kind != MODAL_SHAPE_SEPARABLE) continue;
            const unsigned *m = tmax + d.tab_off / (lmax + 1);
            double bound = 0.0;
            for (int t = 0; t < 3 * d.nterms; t += 3)
                bound += (double)__uint_as_float(m[t]) * (double)__uint_as_float(m[t + 1]) * (double)__uint_as_float(m[t + 2]);
            far |= !(bound <= 1e37);
        }
        far = __syncthreads_or(far);
        if (threadIdx.x == 0) *tail = far;
    }
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)S * N) return;
    const int s = (int)(e / N), r = (int)(e % N);
    const int p1 = triples[3 * r], p2 = triples[3 * r + 1], p3 = triples[3 * r + 2];
    double v = 0.0;
    for (int seg = 0; seg < nseg; seg++) {
        const double *b = B + ((size_t)seg * S + s) * P * P * P;
#define BB(x, y, z) b[((size_t)(x) * P + (y)) * P + (z)]
        v += BB(p1, p2, p3) + BB(p2, p3, p1) + BB(p3, p1, p2) + BB(p3, p2, p1) + BB(p2, p1, p3) + BB(p1, p3, p2);
#undef BB
    }
    beta[e] = v / 6e0;
}

}  // namespace

// use(the slab kernel of the plan)
template <class F>
static modal_status pf_kernel(const ProjPlan &pl, F use)
{
    if (pl.careful) return pl.NC == 16 ? use(k_project_f32<16, true>) : pl.NC == 32 ? use(k_project_f32<32, true>)
                      : pl.NC == 48 ? use(k_project_f32<48, true>) : use(k_project_f32<64, true>);
    return pl.NC == 16 ? use(k_project_f32<16, false>) : pl.NC == 32 ? use(k_project_f32<32, false>)
         : pl.NC == 48 ? use(k_project_f32<48, false>) : use(k_project_f32<64, false>);
}

// Sizes the single-precision projection (buffers, slab schedule, launch shape).
modal_status pf_plan(modal_ctx *ctx, ProjPlan &pl)
{
    const int lmin = ctx->lmin, lmax = ctx->lmax, L = ctx->L, P = ctx->P, S = pl.S, PP = P * P;
    // slab schedule of (lmin, lmax): heaviest slabs first, weight-table offsets
    if (ctx->pf_lmin != lmin || ctx->pf_lmax != lmax) {
        std::vector<long long> base(L);
        long long total = 0;
        for (int s = 0; s < L; s++) {
            base[s] = total;
            total += pf_slab_len(lmin, lmax, lmin + s);
        }
        std::vector<int> order(L);
        for (int s = 0; s < L; s++) order[s] = s;
        auto len = [&](int s) { return (s + 1 < L ? base[s + 1] : total) - base[s]; };
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return len(x) > len(y); });
        ctx->pf_lmin = ctx->pf_lmax = -1;
        MODAL_TRY(ensure(ctx->pf_sched, (sizeof(long long) + sizeof(int)) * (size_t)L));
        MODAL_CUDA(cudaMemcpyAsync(ctx->pf_sched.ptr, base.data(), sizeof(long long) * L, cudaMemcpyHostToDevice, ctx->stream));
        MODAL_CUDA(cudaMemcpyAsync(ctx->pf_sched.as<long long>() + L, order.data(), sizeof(int) * L, cudaMemcpyHostToDevice,
                                   ctx->stream));
        MODAL_CUDA(cudaStreamSynchronize(ctx->stream));
        ctx->pf_lmin = lmin;
        ctx->pf_lmax = lmax;
        ctx->pf_total = total;
    }
    pl.NC = P <= 16 ? 16 : (P <= 32 ? 32 : (P <= 48 ? 48 : 64));
    // teams per SM and shapes per work item: as asked for at most, as many as fit in shared memory
    const int nb4 = (P + 3) / 4, tpt = ceil_div((long)nb4 * nb4, 128);
    const size_t slot = 192 * (size_t)pl.NC + 384 * PF_TC, fper = sizeof(float) * 16 * PF_ROWS * (size_t)tpt;
    pl.smem = PF_SLOTS * slot + sizeof(float) * PF_ROWS * (size_t)(2 * pl.NC + 4) + 128;
    const size_t most = 226 * 1024;
    const int teams = pl.NC <= 32 ? 3 : 2;
    pl.teams = ctx->proj_cpb > 0 ? std::min(ctx->proj_cpb, teams) : teams;
    pl.SG = ctx->proj_sg == 8 ? 8 : 4;
    auto team = [&](int sg) { return (pl.smem + sg * fper + 127) & ~(size_t)127; };
    while (pl.SG > 1 && pl.teams * team(pl.SG) > most) pl.SG--;
    while (pl.teams > 1 && pl.teams * team(pl.SG) > most) pl.teams--;
    MODAL_CUDA(cudaDeviceGetAttribute(&pl.nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    {   // fewer shapes per item where whole rounds of items over the teams take a tenth fewer shapes each
        auto rounds = [&](int sg) { return (long)ceil_div((long)L * ceil_div(S, sg), pl.nsm * pl.teams) * sg; };
        int sg = pl.SG;
        for (int x = pl.SG - 1; x >= 1; x--)
            if (rounds(x) < rounds(sg)) sg = x;
        if (10 * rounds(sg) <= 9 * rounds(pl.SG)) pl.SG = sg;
    }
    pl.team_smem = team(pl.SG);
    pl.smem = (size_t)pl.teams * pl.team_smem;
    pl.QR = lmax / 2 + 1;
    pl.M8 = (lmax / 2 + 1 + 7) / 8 + 4;
    // How the sums between a point and F are kept.  Plain FP32 additions do where a term of the sum meets no more
    // roundings than on CUDA cores, which add 32 points of a row and 16 rows plainly and compensate beyond (52 with
    // the roundings of their compensated sums and stores): two for a chunk's accumulator, one per accumulator of the row,
    // `grp` for a group of rows, seven for the groups of a block and the splits of the rows (one if compensated), one
    // per row block.  l <= 1,700 takes no compensation, l <= 2,500 that of the groups; beyond (or for more than four
    // terms, whose passes multiply the accumulators) the careful kernel compensates all.  Groups compensated: 16 shapes
    // at l <= 2000, P = 30 15.56 -> 15.78 ms; with the blocks compensated as well 16.5 ms and 0.25 -> 0.31 ms at l <= 100.
    int terms = 1;
    for (const DShape &d : pl.desc) terms = std::max(terms, d.nterms);
    const int adds = ceil_div(terms, PF_TC) * (ceil_div(lmax / 4 + 8, PF_KC) + 1) - 1,
              blocks = 2 * ceil_div(lmax / 2 + 1, PF_ROWS) - 1, limit = 52;
    pl.comp = 2 + adds + 16 + 7 + blocks > limit;
    pl.grp = pl.comp && 2 + adds + 16 + 1 + blocks > limit ? 8 : 16;
    if (pl.comp && 2 + adds + pl.grp + 1 + blocks > limit) pl.careful = true;
    // segments of the reduction over slabs: about four CTAs per SM
    const long ctas = (long)ceil_div(PP, 128) * S * ceil_div(P, PB);
    pl.nseg = (int)std::max(1L, std::min(std::min(16L, (long)ceil_div(L, 32)), 4L * pl.nsm / ctas));
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const int nh = 3 * (lmax + 8) / 2 + 16;
    size_t o = 0;
    pl.o_q = o; o += al(sizeof(float) * ((size_t)L + 2 * (size_t)pl.QR) * pl.NC);
    pl.o_v = o; o += al(sizeof(float2) * (lmax + 1));
    pl.o_g = o; o += al(sizeof(float2) * 3 * (size_t)nh);
    pl.o_t = o; o += al(sizeof(float) * (size_t)std::max(4L, pl.tabf_total));
    pl.o_m = o; o += al(sizeof(unsigned) * (size_t)(pl.tab_total / (lmax + 1)));
    pl.o_s = o; o += al(sizeof(PfShape) * (size_t)S);
    pl.o_F = o; o += al(sizeof(float) * (size_t)S * L * PP);
    pl.o_fl = o; o += al(pl.careful ? (size_t)pl.nsm * pl.teams * pl.SG * fper : 0);
    pl.o_B = o; o += al(sizeof(double) * (size_t)pl.nseg * S * P * PP);
    pl.o_bq = o; o += al(sizeof(__nv_bfloat16) * 2 * 3 * 8 * (size_t)pl.M8 * pl.NC);
    pl.o_w = o; o += al(sizeof(float) * PF_ROWS * (size_t)ctx->pf_total);
    MODAL_TRY(ensure(ctx->scratch, o));
    auto attr = [&](auto kern) -> modal_status {
        MODAL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
        return MODAL_OK;
    };
    MODAL_TRY(pf_kernel(pl, attr));
    return oz_reset(ctx);
}

// Enqueues the single-precision projection (capturable: no allocation, no host round trip).
modal_status pf_record(modal_ctx *ctx, const ProjPlan &pl)
{
    const int lmin = ctx->lmin, lmax = ctx->lmax, L = ctx->L, P = ctx->P, N = ctx->N, PP = P * P, S = pl.S, NC = pl.NC;
    uint8_t *b = ctx->scratch.as<uint8_t>();
    float *qp = reinterpret_cast<float *>(b + pl.o_q);
    float *qt = qp + (size_t)L * NC;
    float2 *v = reinterpret_cast<float2 *>(b + pl.o_v);
    const int nh = 3 * (lmax + 8) / 2 + 16;
    float2 *g = reinterpret_cast<float2 *>(b + pl.o_g), *gl = g + nh, *il2 = gl + nh;
    float *tabf = reinterpret_cast<float *>(b + pl.o_t), *Fbuf = reinterpret_cast<float *>(b + pl.o_F);
    PfShape *fs = reinterpret_cast<PfShape *>(b + pl.o_s);
    double *B = reinterpret_cast<double *>(b + pl.o_B);
    __nv_bfloat16 *Bt = reinterpret_cast<__nv_bfloat16 *>(b + pl.o_bq);
    float4 *W = reinterpret_cast<float4 *>(b + pl.o_w);
    unsigned *tmax = reinterpret_cast<unsigned *>(b + pl.o_m);
    int *tail = ctx->ozerr.as<int>() + 1;
    const long long *base = ctx->pf_sched.as<long long>();
    PfSetup u;
    u.lmin = lmin; u.lmax = lmax; u.P = P; u.NC = NC; u.M8 = pl.M8; u.QR = pl.QR; u.nh = nh;
    u.maxt = 1;
    for (const DShape &d : pl.desc) u.maxt = std::max(u.maxt, d.nterms);
    u.nbt = ceil_div(std::max(nh, lmax + 1), 256);
    u.nbb = ceil_div((long)std::max(std::max(16 * pl.M8, L), 2 * pl.QR) * NC, 256);
    u.cl = ctx->cl.as<double>(); u.q = ctx->q.as<double>(); u.tab64 = ctx->shape_tab.as<double>();
    u.desc = ctx->shape_desc.as<DShape>();
    u.g = g; u.gl = gl; u.il2 = il2; u.v = v; u.Bt = Bt; u.qp = qp; u.qt = qt; u.tabf = tabf; u.tmax = tmax;
    u.shapes = fs;
    k_pf_setup<<<u.nbt + u.nbb + S * u.maxt, 256, 0, ctx->stream>>>(u);
    MODAL_TRY(launched(ctx, "pf_setup"));
    const int nbmax = ceil_div((lmax - lmin) / 2 + 1, PF_ROWS);
    k_pf_weights<<<dim3(L, 2 * nbmax), PF_ROWS, 0, ctx->stream>>>(lmin, lmax, nbmax, base, g, gl, v, W);
    MODAL_TRY(launched(ctx, "pf_weights"));
    PfArgs a;
    a.lmin = lmin; a.lmax = lmax; a.P = P; a.S = S; a.SG = pl.SG; a.G = ceil_div(S, pl.SG);
    a.nitems = L * a.G;
    a.M8 = pl.M8;
    a.QR = pl.QR;
    a.Flo = reinterpret_cast<float *>(b + pl.o_fl);
    a.grp = pl.grp;
    a.comp = pl.comp;
    a.order = reinterpret_cast<const int *>(base + L);
    a.base = base;
    a.shapes = fs; a.tabf = tabf; a.il2 = il2; a.W = W; a.Bt = Bt; a.qt = qt; a.Fbuf = Fbuf;
    a.err = ctx->ozerr.as<int>();
    a.teams = pl.teams;
    a.team_smem = (uint32_t)pl.team_smem;
    const int grid = std::min(ceil_div(a.nitems, pl.teams), pl.nsm);
    const int threads = NC <= 32 ? PfMem<32>::THREADS : PfMem<64>::THREADS;
    MODAL_TRY(pf_kernel(pl, [&](auto kern) {
        kern<<<grid, threads, pl.smem, ctx->stream>>>(a);
        return launched(ctx, "project_f32");
    }));
    k_pf_B<<<dim3(ceil_div(PP, 128), S, pl.nseg * ceil_div(P, PB)), 128, 0, ctx->stream>>>(L, P, S, NC, pl.nseg, qp, Fbuf, B);
    MODAL_TRY(launched(ctx, "pf_B"));
    k_pf_beta<<<ceil_div((long)S * N, 256), 256, 0, ctx->stream>>>(N, P, S, pl.nseg, ctx->triples.as<int>(), B,
                                                                     ctx->beta.as<double>(), lmax,
                                                                     ctx->shape_desc.as<DShape>(), tmax, !pl.careful, tail);
    return launched(ctx, "pf_beta");
}

}  // namespace modal

// legendre.cuh -- the quadrature kernels (gl.cu) for their two launchers.
#pragma once

namespace modal {

constexpr int GL_THREADS = 64;  // per block of 32 roots
// nodes and weights; grid ceil((n / 2 + 1) / 32)
__global__ void k_gl_nodes(int n, double *mu, double *w);

constexpr int PL_THREADS = 96;  // per block of 32 nodes
constexpr int PL_SMEM_MAX = 200 * 1024;  // dynamic shared memory: one process-wide limit for every size
// pl[l][k] = pw[l] P_l(mu_k); grid ceil(nmu / 32), 24 (lmax + 1) bytes of dynamic shared memory
__global__ void k_legendre_table(int nmu, int lmax, const double *mu, const double *pw, double *pl);

}  // namespace modal

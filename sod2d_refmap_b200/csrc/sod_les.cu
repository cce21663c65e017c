// LES eddy viscosity (Vreman): sgs_visc (mod_sgs_viscosity.f90:13-125) on the device.
//
// Per element (4 per CTA, one thread per gauss point): the velocity is staged in shared memory
// and differentiated with the same line derivatives and He as the RHS; with hLES = gpvol^(1/3),
// alpha = |grad u|^2 and beta = hLES^2 grad u^T grad u, the point value is
// c_sgs sqrt(max(B(beta), 1e-10) / alpha) where alpha > 1e-10 (B = sum of the principal 2x2
// minors), else the previous mu_sgs; the 3x3x3 convertIJK filter of the entropy viscosity then
// smooths it inside the element, as three 3-point passes (weights and index map are separable).
// Element-local, so the update of musgs_int is in place.
//
// Bounded by memory latency on its inputs (10 metric values, 3 gathered velocities and the old value
// per point).  D comes from a shared table (indexed by lane in the kernel parameters it was copied to
// local memory: 128 bytes of stack, and a chain of local loads under every sum), and the lane order
// is the RHS kernels': 24^3 elements 41 -> 28 us.
#include "sod_internal.cuh"

namespace sod {
namespace les {

constexpr int EPB = 4;

__device__ __forceinline__ int nb_filter(int x) {  // natural index of convertIJK(x+1)
  return (x < 0) ? 1 : ((x > 3) ? 1 : x);
}

__global__ void __launch_bounds__(64 * EPB) k_sgs(int nelem, const int32_t* __restrict__ econn,
                                                 const double* __restrict__ geo, const double* __restrict__ u0,
                                                 const double* __restrict__ u1, const double* __restrict__ u2,
                                                 const __grid_constant__ DMat D, double c_sgs,
                                                 double* __restrict__ musgs) {
  __shared__ double us[EPB][3][FSTRIDE];
  __shared__ double ml[EPB][2][NN];
  __shared__ __align__(16) double Ds[NP1 * NP1];
  const int es = threadIdx.x >> 6, lt = threadIdx.x & 63;
  const int e = blockIdx.x * EPB + es;
  const bool act = e < nelem;
  const int ee = act ? e : nelem - 1;
  // lane bits (i0 j0 i1 j1 k): one shared-memory wavefront per xi and eta line load
  const int i = (lt & 1) | ((lt >> 1) & 2), j = ((lt >> 1) & 1) | ((lt >> 2) & 2), k = lt >> 4;
  const int d = i + 4 * j + 16 * k, s = sidx(i, j, k);
  const int n = econn[(size_t)ee * NN + d];
  const double* G = geo + (size_t)ee * NGEO * NN;
  double H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = G[c * NN + d];
  const double gpv = G[9 * NN + d];
  const double old = musgs[(size_t)ee * NN + d];
  if (threadIdx.x < NP1 * NP1) Ds[threadIdx.x] = D.d[threadIdx.x >> 2][threadIdx.x & 3];
  us[es][0][s] = u0[n];
  us[es][1][s] = u1[n];
  us[es][2][s] = u2[n];
  __syncthreads();
  double gu[3][3];  // gu[c][r] = d u_c / d x_r
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const double* f = &us[es][0][0] + (dir == 0 ? sidx(0, j, k) : (dir == 1 ? sidx(i, 0, k) : sidx(i, j, 0)));
    const int st = dir == 0 ? 1 : (dir == 1 ? 4 : PLANE);
    const double* w = Ds + 4 * (dir == 0 ? i : (dir == 1 ? j : k));
    double l[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int m = 0; m < NP1; ++m)
#pragma unroll
      for (int c = 0; c < 3; ++c) l[c] += w[m] * f[c * FSTRIDE + m * st];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) gu[c][r] = dir == 0 ? H[3 * r] * l[c] : gu[c][r] + H[3 * r + dir] * l[c];
  }
  const double hLES = cbrt(gpv);
  double alpha = 0.0, V[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      V[a][b] = (gu[0][a] * gu[0][b] + gu[1][a] * gu[1][b] + gu[2][a] * gu[2][b]) * (hLES * hLES);
      alpha += gu[a][b] * gu[a][b];
    }
  const double B = V[0][0] * V[1][1] + V[0][0] * V[2][2] + V[1][1] * V[2][2] - V[0][1] * V[0][1] -
                   V[0][2] * V[0][2] - V[1][2] * V[1][2];
  double* m0 = ml[es][0];
  double* m1 = ml[es][1];
  m0[d] = alpha > 1.0e-10 ? c_sgs * sqrt(fmax(B, 1.0e-10) / alpha) : old;
  __syncthreads();
  m1[d] = 0.25 * m0[nb_filter(i - 1) + 4 * j + 16 * k] + 0.5 * m0[d] + 0.25 * m0[nb_filter(i + 1) + 4 * j + 16 * k];
  __syncthreads();
  // m0 was last read before the barrier above
  m0[d] = 0.25 * m1[i + 4 * nb_filter(j - 1) + 16 * k] + 0.5 * m1[d] + 0.25 * m1[i + 4 * nb_filter(j + 1) + 16 * k];
  __syncthreads();
  const double acc =
      0.25 * m0[i + 4 * j + 16 * nb_filter(k - 1)] + 0.5 * m0[d] + 0.25 * m0[i + 4 * j + 16 * nb_filter(k + 1)];
  if (act) musgs[(size_t)e * NN + d] = acc;
}

}  // namespace les

int launch_sgs(SodMesh* m, const double* u, cudaStream_t st) {
  const size_t N = m->npoin;
  const int grid = (m->nelem + les::EPB - 1) / les::EPB;
  les::k_sgs<<<grid, 64 * les::EPB, 0, st>>>(m->nelem, m->econn, m->geo64, u, u + N, u + 2 * N, m->D, m->prm.c_sgs,
                                             m->musgs_int);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

}  // namespace sod

// Per-routine entry points with the reference argument lists (sm_100a).  Each keeps the
// reference's inputs independent (e.g. full_convec_ijk takes u and q separately, and the
// energy-like field E as given) and writes fully overwritten nodal outputs.  Element work
// runs one CTA per element (64 threads = gauss points) in FP64, assembly is the same ordered
// CSR gather of node-major residual rows as the fused path.
//
// The element kernels make one pass over the 12 line points of each node: the products of a
// quartet share the line point's contravariant velocities V(m) = sum_c He(c,dir)(x) u_c(m) and
// W(m) (of q), formed with the output point's metric, so nothing but the nodal fields is staged and
// no product is differentiated by itself.  Lanes are ordered (i0 j0 i1 j1 k): a warp's xi and eta line
// loads then cost one shared-memory wavefront each (see sod_rhs.cu).  20^3 elements:
// convection 78 -> 27 us, diffusion 35 -> 27, scalar 22 -> 17, gather of 5 fields 15 -> 9.
#include "sod_internal.cuh"
#include <cmath>

namespace sod {

int launch_visc_dt(SodMesh* m, const SodState* s, double* dt_out, float* mue32, cudaStream_t st, bool bits_set);

// the thread's point in the lane order (i0 j0 i1 j1 k), and its three lines in a staged field
struct Point {
  int i, j, k, d, s;
  int row[3], line[3];
};
__host__ __device__ constexpr int line_stride(int dir) { return dir == 0 ? 1 : (dir == 1 ? 4 : PLANE); }
__device__ __forceinline__ Point point_of(int lt) {
  Point p;
  p.i = (lt & 1) | ((lt >> 1) & 2);
  p.j = ((lt >> 1) & 1) | ((lt >> 2) & 2);
  p.k = lt >> 4;
  p.d = p.i + 4 * p.j + 16 * p.k;
  p.s = sidx(p.i, p.j, p.k);
  p.row[0] = p.i; p.row[1] = p.j; p.row[2] = p.k;
  p.line[0] = sidx(0, p.j, p.k); p.line[1] = sidx(p.i, 0, p.k); p.line[2] = sidx(p.i, p.j, 0);
  return p;
}

// Each kernel is given what it reads: on a small mesh a call is bound by the host's launches, and one struct
// for all with D's row sums in it (312 bytes) cost up to 0.3 us a call.
struct RefArgs {
  int64_t npoin;
  const int32_t* econn;
  const double* geo;
  double* rel;                                  // rows [(e*64 + d)*6 + f]
  DMat D;
  const double* u;
};
struct ConvecArgs : RefArgs {
  const double *q, *rho, *pr, *E;
  double Dsum[NP1];                             // row sums of D
};
struct ScalarArgs : RefArgs {
  const double *q, *eta;
};
struct DiffusionArgs : RefArgs {
  const double *rho, *rho_n, *Tem, *mu_fluid;
  const double *mue, *musgs;                    // internal layout [e][64]
  double Cp, Pr, c_rho, c_ener;
};

// full_convec_ijk (elem_convec.f90:241-435); TOTH: full_convec_ijk_H (elem_convec.f90:48-187),
// whose energy residual is 0.5 (div((E + p) u) + (E + p) div u + u . grad(E + p)) with E the
// total energy; mass and momentum are the same in both.  Both energy quartets (E and k = |u|^2/2, the
// same form) are taken at once on H = E + k.
//
// u, q, rho and H enter the line sums by their differences to the own point, which are small on a resolved
// field; the constant parts are whole sums (div u, div q, u.grad rho) times the own value, and D's row
// sums, which are zero but for the rounding of D's entries.  The differences of H are formed from those of
// E and k: the rounding of E + k itself would be differentiated.  Vortex at 8^3 against extended precision: mass
// 3.1e-15, energy 3.4e-15, momentum less grad p 1.8e-16; with the quartets one by one 6.2e-15, 6.5e-15 and
// 2.3e-16, with whole values in the sums 7.4e-15, 1.2e-14 and 3.3e-16 (and 24 us instead of 27 at 20^3).  On white
// noise, where differences are no smaller than values, momentum 2.5e-16 (quartets 1.8e-16).
template <bool TOTH>
__global__ void __launch_bounds__(64) k_convec_ref(const __grid_constant__ ConvecArgs a) {
  constexpr int F_K = TOTH ? 8 : 9;         // k, after
  __shared__ double f[F_K + 1][FSTRIDE];   // rho, p, E (TOTH: p + E), u, q
  __shared__ double Ds[16], Dsum[NP1];
  const int e = blockIdx.x;
  const Point p = point_of(threadIdx.x);
  if (threadIdx.x < 16) Ds[threadIdx.x] = a.D.d[threadIdx.x >> 2][threadIdx.x & 3];
  if (threadIdx.x < NP1) Dsum[threadIdx.x] = a.Dsum[threadIdx.x];
  const int n = a.econn[(int64_t)e * NN + p.d];
  const int64_t N = a.npoin;
  const double* G = a.geo + (int64_t)e * NGEO * NN;
  double H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = G[c * NN + p.d];
  const double gpv = G[9 * NN + p.d];
  double u[3], q[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) { u[c] = a.u[n + N * c]; q[c] = a.q[n + N * c]; }
  const double rho = a.rho[n], El = a.E[n], pr = a.pr[n];
  const double Ex = TOTH ? pr + El : El, kx = 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  const double Hx = TOTH ? Ex : Ex + kx;
  f[0][p.s] = rho; f[1][p.s] = pr; f[2][p.s] = Ex;
  if (!TOTH) f[F_K][p.s] = kx;
#pragma unroll
  for (int c = 0; c < 3; ++c) { f[3 + c][p.s] = u[c]; f[6 + c][p.s] = q[c]; }
  __syncthreads();
  double divU = 0.0, divQ = 0.0, ugr = 0.0;      // div u, div q, u.grad rho
  double A[3] = {0, 0, 0};                       // div(q_c u) + rho div(u_c u) + q.grad u_c + u.grad q_c, of the differences
  double gP[3] = {0, 0, 0};
  double Ea = 0.0, Er = 0.0;                     // div(rho H u) + rho div(H u) + q.grad H + u.grad(rho H) (TOTH: div(H u) + u.grad H) and div(rho u), likewise
  double sV = 0.0, sW = 0.0;                     // D's row sums times V and W
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const double h0 = H[dir], h1 = H[3 + dir], h2 = H[6 + dir];
    const double Vx = h0 * u[0] + h1 * u[1] + h2 * u[2], Wx = h0 * q[0] + h1 * q[1] + h2 * q[2];
    double lu[3] = {0, 0, 0}, lq[3] = {0, 0, 0}, lr = 0.0, lp = 0.0, lH = 0.0, lrH = 0.0;
#pragma unroll
    for (int m = 0; m < NP1; ++m) {
      const double* v = &f[0][0] + p.line[dir] + m * line_stride(dir);
      const double w = Ds[4 * p.row[dir] + m];
      const double u_[3] = {v[3 * FSTRIDE], v[4 * FSTRIDE], v[5 * FSTRIDE]};
      const double q_[3] = {v[6 * FSTRIDE], v[7 * FSTRIDE], v[8 * FSTRIDE]};
      const double r_ = v[0];
      const double wV = w * (h0 * u_[0] + h1 * u_[1] + h2 * u_[2]);
      const double dr = r_ - rho;
      lr += w * dr;
      lp += w * v[FSTRIDE];
      double dH = v[2 * FSTRIDE] - Ex;
      if (!TOTH) dH += v[F_K * FSTRIDE] - kx;
      lH += w * dH;
      if (TOTH) {
        Ea += wV * dH;
      } else {
        const double wVr = wV * r_;
        Er += wV * dr;
        Ea += (wVr + wV * rho) * dH;
        lrH += (w * r_) * dH;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double du = u_[c] - u[c], dq = q_[c] - q[c];
        A[c] += wV * (dq + rho * du);
        lu[c] += w * du;
        lq[c] += w * dq;
      }
    }
    sV += Vx * Dsum[p.row[dir]];
    sW += Wx * Dsum[p.row[dir]];
    divU += h0 * lu[0] + h1 * lu[1] + h2 * lu[2];
    divQ += h0 * lq[0] + h1 * lq[1] + h2 * lq[2];
    ugr += Vx * lr;
    gP[0] += h0 * lp;
    gP[1] += h1 * lp;
    gP[2] += h2 * lp;
    Ea += TOTH ? Vx * lH : Wx * lH + Vx * lrH;
#pragma unroll
    for (int c = 0; c < 3; ++c) A[c] += Wx * lu[c] + Vx * lq[c];
  }
  // the constant parts
  divU += sV;
  divQ += sW;
  ugr += rho * sV;
  const double Rm = 0.5 * (divQ + rho * divU + ugr);
  const double Re = TOTH ? 0.5 * (Ea + Hx * (2.0 * divU + sV))
                         : 0.25 * (Ea + Hx * (Er + divQ + 3.0 * rho * divU + 2.0 * ugr + sW));
  const double cu = divQ + rho * divU + ugr + sW, cq = 2.0 * divU + sV;
  double Rmo[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) Rmo[c] = 0.25 * (A[c] + u[c] * cu + q[c] * cq) + gP[c];
  store_res6<double>(a.rel, (size_t)e * NN + p.d, gpv * Rm, gpv * Rmo[0], gpv * Rmo[1], gpv * Rmo[2], gpv * Re, 0.0);
}

// generic_scalar_convec_ijk (elem_convec.f90:488-556)
__global__ void __launch_bounds__(64) k_scalar_ref(const __grid_constant__ ScalarArgs a) {
  __shared__ double f[7][FSTRIDE];
  __shared__ double Ds[16];
  const int e = blockIdx.x;
  const Point p = point_of(threadIdx.x);
  if (threadIdx.x < 16) Ds[threadIdx.x] = a.D.d[threadIdx.x >> 2][threadIdx.x & 3];
  const int n = a.econn[(int64_t)e * NN + p.d];
  const int64_t N = a.npoin;
  const double* G = a.geo + (int64_t)e * NGEO * NN;
  double H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = G[c * NN + p.d];
  const double gpv = G[9 * NN + p.d];
  double u[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) { u[c] = a.u[n + N * c]; f[1 + c][p.s] = u[c]; f[4 + c][p.s] = a.q[n + N * c]; }
  const double eta = a.eta[n];
  f[0][p.s] = eta;
  __syncthreads();
  double div = 0.0, divU = 0.0, adv = 0.0;
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    double le = 0.0, lu[3] = {0, 0, 0}, lq[3] = {0, 0, 0};
#pragma unroll
    for (int m = 0; m < NP1; ++m) {
      const double* v = &f[0][0] + p.line[dir] + m * line_stride(dir);
      const double w = Ds[4 * p.row[dir] + m];
      le += w * v[0];
#pragma unroll
      for (int c = 0; c < 3; ++c) { lu[c] += w * v[(1 + c) * FSTRIDE]; lq[c] += w * v[(4 + c) * FSTRIDE]; }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      divU += H[3 * c + dir] * lu[c];
      div += H[3 * c + dir] * lq[c];
      adv += (H[3 * c + dir] * u[c]) * le;
    }
  }
  a.rel[(size_t)e * NN + p.d] = gpv * (0.5 * (div + eta * divU + adv));  // one value per element node
}

// full_diffusion_ijk (elem_diffu.f90:44-194)
__global__ void __launch_bounds__(64) k_diffusion_ref(const __grid_constant__ DiffusionArgs a) {
  __shared__ double f[5][FSTRIDE];  // rho, T, u
  __shared__ double V[18][FSTRIDE];
  __shared__ double Ds[16], DTs[16];
  const int e = blockIdx.x;
  const Point p = point_of(threadIdx.x);
  if (threadIdx.x < 16) {
    Ds[threadIdx.x] = a.D.d[threadIdx.x >> 2][threadIdx.x & 3];
    DTs[threadIdx.x] = a.D.d[threadIdx.x & 3][threadIdx.x >> 2];
  }
  const int n = a.econn[(int64_t)e * NN + p.d];
  const int64_t N = a.npoin;
  const double* G = a.geo + (int64_t)e * NGEO * NN;
  double H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = G[c * NN + p.d];
  const double gpv = G[9 * NN + p.d];
  double u[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) { u[c] = a.u[n + N * c]; f[2 + c][p.s] = u[c]; }
  f[0][p.s] = a.rho[n];
  f[1][p.s] = a.Tem[n];
  const double rhon = a.rho_n[n], muf = a.mu_fluid[n];
  const double mue = a.mue[(int64_t)e * NN + p.d];
  const double musgs = a.musgs ? a.musgs[(int64_t)e * NN + p.d] : 0.0;
  __syncthreads();
  double gRho[3] = {0, 0, 0}, gT[3] = {0, 0, 0}, gU[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    double l[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int m = 0; m < NP1; ++m) {
      const double* v = &f[0][0] + p.line[dir] + m * line_stride(dir);
      const double w = Ds[4 * p.row[dir] + m];
#pragma unroll
      for (int c = 0; c < 5; ++c) l[c] += w * v[c * FSTRIDE];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double h = H[3 * r + dir];
      gRho[r] += h * l[0];
      gT[r] += h * l[1];
#pragma unroll
      for (int c = 0; c < 3; ++c) gU[c][r] += h * l[2 + c];
    }
  }
  const double divU = gU[0][0] + gU[1][1] + gU[2][2];
  const double mu_fgp = muf + rhon * musgs, mut = mu_fgp + mue;
  const double twoThirds = 2.0 / 3.0;
  double tau[3][3], tauU[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
#pragma unroll
    for (int c = 0; c < 3; ++c) tau[r][c] = mut * (gU[r][c] + gU[c][r]);
    tau[r][r] = tau[r][r] - mu_fgp * twoThirds * divU;
    tauU[r] = tau[r][0] * u[0] + tau[r][1] * u[1] + tau[r][2] * u[2];
  }
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const double h0 = gpv * H[dir], h1 = gpv * H[3 + dir], h2 = gpv * H[6 + dir];
    auto emit = [&](int v, const double* x) { V[3 * v + dir][p.s] = h0 * x[0] + h1 * x[1] + h2 * x[2]; };
    emit(0, gRho);
    emit(1, tauU);
    emit(2, gT);
    emit(3, tau[0]);
    emit(4, tau[1]);
    emit(5, tau[2]);
  }
  __syncthreads();
  double dv[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int dir = 0; dir < 3; ++dir)
#pragma unroll
    for (int m = 0; m < NP1; ++m) {
      const double w = DTs[4 * p.row[dir] + m];
#pragma unroll
      for (int v = 0; v < 6; ++v) dv[v] += w * V[3 * v + dir][p.line[dir] + m * line_stride(dir)];
    }
  const double nu_e = a.c_rho * mue / rhon;
  const double kappa_e = muf * a.Cp / a.Pr + a.c_ener * mue * a.Cp / a.Pr + a.Cp * rhon * musgs / 0.9;
  store_res6<double>(a.rel, (size_t)e * NN + p.d, nu_e * dv[0], dv[3], dv[4], dv[5], dv[1] + kappa_e * dv[2], 0.0);
}

// ordered gather of the residual rows' five fields
__global__ void __launch_bounds__(256) k_gather_rows5(int npoin, const int32_t* __restrict__ ptr,
                                                      const int32_t* __restrict__ idx, const double* __restrict__ rel,
                                                      double* __restrict__ o0, double* __restrict__ o1,
                                                      double* __restrict__ o4) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= npoin) return;
  double r[6] = {0, 0, 0, 0, 0, 0};
  gather_rows<double>(rel, idx, ptr[n], ptr[n + 1], r);
  o0[n] = r[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) o1[n + (int64_t)npoin * c] = r[1 + c];
  o4[n] = r[4];
}
// the same of one value per element node
__global__ void __launch_bounds__(256) k_gather_one(int npoin, const int32_t* __restrict__ ptr,
                                                    const int32_t* __restrict__ idx, const double* __restrict__ rel,
                                                    double* __restrict__ out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= npoin) return;
  double s = 0.0;
  for (int c = ptr[n]; c < ptr[n + 1]; c += 4) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q < ptr[n + 1]) v[q] = rel[idx[c + q]];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q < ptr[n + 1]) s += v[q];
  }
  out[n] = s;
}

// lumped_solver_scal/vect over the working nodes (mod_solver.f90:23-58): rows without elements
// (periodic slaves, absent from lpoin_w) are left as they are
__global__ void k_lumped(int64_t npoin, int ncomp, const double* __restrict__ Ml, const int32_t* __restrict__ ptr,
                         double* R) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin * ncomp) return;
  const int64_t n = t % npoin;
  if (ptr[n + 1] > ptr[n]) R[t] = R[t] / Ml[n];
}

__global__ void k_sutherland(int64_t npoin, const double* __restrict__ Tem, const double* __restrict__ mf,
                             double* __restrict__ mu) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin) return;
  const double T = Tem[t];
  mu[t] = mf[t] * 0.000001458 * (T * sqrt(T)) / (T + 110.4);
}

// eta sum/max/min -> scal[0] mean, scal[1] norm (single-block deterministic reduction)
__global__ void __launch_bounds__(1024) k_eta_norm(int64_t npoin, int64_t nwork, const int32_t* __restrict__ ptr,
                                                   const double* __restrict__ eta, double* scal, int normalise) {
  __shared__ double sh[3][32];
  double s = 0.0, mx = -1e300, mn = 1e300;
  for (int64_t t = threadIdx.x; t < npoin; t += blockDim.x) {
    if (ptr[t + 1] == ptr[t]) continue;  // over lpoin_w only (mod_entropy_viscosity.f90:43-62)
    const double v = eta[t];
    s += v; mx = fmax(mx, v); mn = fmin(mn, v);
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
  }
  if ((threadIdx.x & 31) == 0) { sh[0][threadIdx.x >> 5] = s; sh[1][threadIdx.x >> 5] = mx; sh[2][threadIdx.x >> 5] = mn; }
  __syncthreads();
  if (threadIdx.x == 0) {
    s = sh[0][0]; mx = sh[1][0]; mn = sh[2][0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { s += sh[0][w]; mx = fmax(mx, sh[1][w]); mn = fmin(mn, sh[2][w]); }
    if (normalise) {
      const double mean = s / (double)nwork;
      scal[0] = mean;
      scal[1] = fmax(mx - mean, mean - mn);
    } else {
      scal[0] = 0.0;
      scal[1] = 1.0;
    }
  }
}

// adapt_dt_cfl (mod_time_ops.f90:31-57): per-element limits, then a single-block min
__global__ void k_dt_elem(int nelem, int64_t npoin, const int32_t* __restrict__ econn, const double* __restrict__ helem,
                          const double* __restrict__ u, const double* __restrict__ cs, const double* __restrict__ muf,
                          const double* __restrict__ musgs, const double* __restrict__ rho, double cfl_conv,
                          double cfl_diff, double* __restrict__ out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nelem) return;
  double L3 = 0.0, maxMU = 0.0;
  for (int d = 0; d < NN; ++d) {
    const int n = econn[(int64_t)e * NN + d];
    double um = fabs(u[n]);
    um = fmax(um, fabs(u[n + npoin]));
    um = fmax(um, fabs(u[n + 2 * npoin]));
    L3 = fmax(L3, um + cs[n]);
    const double sg = musgs ? musgs[(int64_t)e * NN + d] : 0.0;
    maxMU = fmax(maxMU, (rho[n] * sg + muf[n]) / rho[n]);
  }
  const double hh = helem[e] / (double)(2.0 * P + 1);
  out[e] = fmin(cfl_conv * hh / L3, cfl_diff * (hh * hh) / maxMU);
}

__global__ void __launch_bounds__(1024) k_min_reduce(int64_t n, const double* __restrict__ v, double* out) {
  __shared__ double sh[32];
  double mn = 100000000000000.0;
  for (int64_t t = threadIdx.x; t < n; t += blockDim.x) mn = fmin(mn, v[t]);
  for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mn;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mn = fmin(mn, sh[w]);
    *out = fmin(sh[0], mn);
  }
}

__global__ void k_csr_spmv_legacy(int npoin, const int32_t* __restrict__ rdom, const int32_t* __restrict__ cdom,
                                  const double* __restrict__ Mc, const double* __restrict__ v, double* __restrict__ u) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= npoin) return;
  double s = 0.0;
  for (int c = rdom[r]; c < rdom[r + 1]; ++c) s += Mc[c] * v[cdom[c] - 1];
  u[r] = s;
}

static int gather_out(SodMesh* m, double* Rmass, double* Rmom, double* Rener, cudaStream_t st) {
  k_gather_rows5<<<(m->npoin + 255) / 256, 256, 0, st>>>(m->npoin, m->n2e_ptr, m->n2e, (const double*)m->buf.rel, Rmass,
                                                          Rmom, Rener);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

template <typename Args>
static Args ref_args(SodMesh* m, const double* u) {
  Args a{};
  a.npoin = m->npoin;
  a.econn = m->econn;
  a.geo = m->geo64;
  a.rel = (double*)m->buf.rel;
  a.D = m->D;
  a.u = u;
  return a;
}
static ConvecArgs convec_args(SodMesh* m, const double* u, const double* q, const double* rho, const double* pr,
                              const double* E) {
  ConvecArgs a = ref_args<ConvecArgs>(m, u);
  a.q = q; a.rho = rho; a.pr = pr; a.E = E;
  for (int r = 0; r < NP1; ++r) a.Dsum[r] = m->Dsum[r];
  return a;
}

}  // namespace sod

using namespace sod;

extern "C" {

int sod_full_convec_ijk(SodMesh* m, const double* u, const double* q, const double* rho, const double* pr,
                        const double* E, double* Rmass, double* Rmom, double* Rener, sod_stream_t stream) {
  SOD_ARG(m && u && q && rho && pr && E && Rmass && Rmom && Rener, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  k_convec_ref<false><<<m->nelem, 64, 0, st>>>(convec_args(m, u, q, rho, pr, E));
  SOD_CHECK_LAUNCH();
  return gather_out(m, Rmass, Rmom, Rener, st);
}

int sod_full_convec_ijk_H(SodMesh* m, const double* u, const double* q, const double* rho, const double* pr,
                          const double* E, double* Rmass, double* Rmom, double* Rener, sod_stream_t stream) {
  SOD_ARG(m && u && q && rho && pr && E && Rmass && Rmom && Rener, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  k_convec_ref<true><<<m->nelem, 64, 0, st>>>(convec_args(m, u, q, rho, pr, E));
  SOD_CHECK_LAUNCH();
  return gather_out(m, Rmass, Rmom, Rener, st);
}

int sod_generic_scalar_convec_ijk(SodMesh* m, const double* q, const double* eta, const double* u,
                                  double* Rconvec, sod_stream_t stream) {
  SOD_ARG(m && q && eta && u && Rconvec, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  ScalarArgs a = ref_args<ScalarArgs>(m, u);
  a.q = q; a.eta = eta;
  k_scalar_ref<<<m->nelem, 64, 0, st>>>(a);
  SOD_CHECK_LAUNCH();
  k_gather_one<<<(m->npoin + 255) / 256, 256, 0, st>>>(m->npoin, m->n2e_ptr, m->n2e, (const double*)m->buf.rel, Rconvec);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

int sod_full_diffusion_ijk(SodMesh* m, double Cp, double Pr, const double* rho_n, const double* rho,
                           const double* u, const double* Tem, const double* mu_fluid, const double* mu_e,
                           const double* mu_sgs, double* Rmass, double* Rmom, double* Rener, sod_stream_t stream) {
  SOD_ARG(m && rho_n && rho && u && Tem && mu_fluid && mu_e && Rmass && Rmom && Rener, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  // element arrays to the internal layout (mu_sgs into the stage scratch of rsum)
  rc = mesh_ref_to_internal_elem(m, mu_e, m->mue_int, st);
  if (rc) return rc;
  double* musgs_int = nullptr;
  if (mu_sgs) {
    SOD_CUDA(cudaMallocAsync((void**)&musgs_int, sizeof(double) * (size_t)m->nelem * NN, st));
    rc = mesh_ref_to_internal_elem(m, mu_sgs, musgs_int, st);
    if (rc) return rc;
  }
  DiffusionArgs a = ref_args<DiffusionArgs>(m, u);
  a.c_rho = m->prm.c_rho; a.c_ener = m->prm.c_ener;
  a.rho_n = rho_n; a.rho = rho; a.Tem = Tem; a.mu_fluid = mu_fluid; a.mue = m->mue_int; a.musgs = musgs_int;
  a.Cp = Cp; a.Pr = Pr;
  k_diffusion_ref<<<m->nelem, 64, 0, st>>>(a);
  SOD_CHECK_LAUNCH();
  if (musgs_int) SOD_CUDA(cudaFreeAsync(musgs_int, st));
  return gather_out(m, Rmass, Rmom, Rener, st);
}

int sod_lumped_solver(SodMesh* m, double* R, int ncomp, sod_stream_t stream) {
  SOD_ARG(m && R && (ncomp == 1 || ncomp == 3), "lumped solver args");
  int64_t n = (int64_t)m->npoin * ncomp;
  k_lumped<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(m->npoin, ncomp, m->Ml, m->n2e_ptr, R);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

int sod_sutherland_viscosity(int32_t npoin, const double* Tem, const double* mu_factor, double* mu_fluid,
                             sod_stream_t stream) {
  SOD_ARG(npoin > 0 && Tem && mu_factor && mu_fluid, "sutherland args");
  k_sutherland<<<(npoin + 255) / 256, 256, 0, (cudaStream_t)stream>>>(npoin, Tem, mu_factor, mu_fluid);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

int sod_smart_visc_spectral(SodMesh* m, const double* Reta, const double* rho, const double* u, const double* csound,
                            const double* Tem, const double* eta, double* mu_e, sod_stream_t stream) {
  SOD_ARG(m && Reta && rho && u && csound && Tem && eta && mu_e, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  k_eta_norm<<<1, 1024, 0, st>>>(m->npoin, m->npoin_w, m->n2e_ptr, eta, m->buf.scal, m->prm.normalise);
  SOD_CHECK_LAUNCH();
  SodState s{};
  s.Reta = const_cast<double*>(Reta);
  s.rho = const_cast<double*>(rho);
  s.u = const_cast<double*>(u);
  s.csound = const_cast<double*>(csound);
  s.Tem = const_cast<double*>(Tem);
  s.mu_fluid = const_cast<double*>(rho);  // unused without dt
  rc = launch_visc_dt(m, &s, nullptr, nullptr, st, false);
  if (rc) return rc;
  return mesh_internal_to_ref_elem(m, m->mue_int, mu_e, st);
}

int sod_adapt_dt_cfl(SodMesh* m, const double* u, const double* csound, const double* mu_fluid,
                     const double* mu_sgs, const double* rho, double* dt_dev, sod_stream_t stream) {
  SOD_ARG(m && u && csound && mu_fluid && rho && dt_dev, "null argument");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  double* musgs_int = nullptr;
  if (mu_sgs) {
    SOD_CUDA(cudaMallocAsync((void**)&musgs_int, sizeof(double) * (size_t)m->nelem * NN, st));
    rc = mesh_ref_to_internal_elem(m, mu_sgs, musgs_int, st);
    if (rc) return rc;
  }
  double* tmp = (double*)m->buf.rel;  // nelem doubles of scratch
  k_dt_elem<<<(m->nelem + 127) / 128, 128, 0, st>>>(m->nelem, m->npoin, m->econn, m->helem, u, csound, mu_fluid,
                                                     musgs_int, rho, m->prm.cfl_conv, m->prm.cfl_diff, tmp);
  SOD_CHECK_LAUNCH();
  k_min_reduce<<<1, 1024, 0, st>>>(m->nelem, tmp, dt_dev);
  SOD_CHECK_LAUNCH();
  if (musgs_int) SOD_CUDA(cudaFreeAsync(musgs_int, st));
  return SOD_OK;
}

int sod_csr_spmv_scal(int32_t npoin, int32_t nzdom, const int32_t* rdom, const int32_t* cdom, const double* Mc,
                      const double* v, double* u, sod_stream_t stream) {
  SOD_ARG(npoin > 0 && nzdom >= 0 && rdom && cdom && Mc && v && u, "csr args");
  k_csr_spmv_legacy<<<(npoin + 127) / 128, 128, 0, (cudaStream_t)stream>>>(npoin, rdom, cdom, Mc, v, u);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

}  // extern "C"

// Hand-written adjoint (vector-Jacobian product) of the stage RHS and of one RK4 step (sm_100a).
//
// The stage RHS is R(U) = (1/Ml) Gather_e[ gpvol * conv_e(U) + diff_e(U) ] with U = (rho, q, E),
// conv from full_convec_ijk (elem_convec.f90:211-460, energy with h), diff from
// full_diffusion_ijk (elem_diffu.f90:12-198), the stage EOS of time_integ.f90:266-285 and
// Sutherland's law (mod_fluid_viscosity.f90:21-41) - Sutherland is differentiated, the entropy
// viscosity mu_e is frozen at its forward value (it is updated once per step from the state
// after the step, time_integ.f90:492-493), as is dt.
//
// k_rhs_vjp: one element per CTA, one thread per gauss point, FP64.  The convection of the stage
// residual is a sum over line pairs (the two-point form of the quartets, see sod_rhs.cu):
//   R_mass(x) = 1/2 sum_dir sum_l D[x][l] (rho_x + rho_l) (V_x + V_l),   V_l = sum_c He(c,dir)(x) u_c(l)
//   R_f(x)    = 1/4 sum_dir sum_l D[x][l] (rho_x + rho_l) (V_x + V_l) (f_x + f_l),  f = u_c, H = h + k
// so a node's adjoint is one pass over its 12 line points, each taken in both roles: the node as
// the output point x (row D[a][l], own metric and seeds) and as the partner l (column D[l][a], the
// line point's metric and seeds).  That needs the line point's 6 fields, 5 seeds and 3 metric
// values and ~42 FP64 operations; q, rho H and the product fields carry no adjoint of their own.
// The same pass structure gives the forward gradients and the D-line sums of the seeds (the
// transpose of pass 2's D^T); the viscous stress is reversed pointwise and its five gradient
// fields (u, rho, T) go back through He^T and D^T.  32^3, one launch: 218 us; 467 us with the 29 nodal
// product fields each sent back through three line arrays.  Bounded by the L1 data pipe (80% busy)
// and the FP64 pipe (60%) at 12 resident warps per SM (168 registers); 16 warps (128 registers, own
// values parked in shared memory) measured 206 us against 173 us for the call at 27^3.
// Element-node adjoints are assembled by the same ordered CSR gather as the forward path.
#include "sod_internal.cuh"
#include <cmath>

namespace sod {
int ensure_step_buffers(SodMesh* m, bool mixed);
int les_in(SodMesh* m, const SodState* s, cudaStream_t st);
int launch_rhs(SodMesh* m, bool mixed, int epb, const double* rho, const double* q0, const double* q1,
               const double* q2, const double* E, const double* mu_factor, const double* musgs_int, cudaStream_t st);

namespace adj {

constexpr double kC1 = 0.000001458;
constexpr double kS = 110.4;
// shared arrays: nodal fields; seeds over Ml (2 w_mass, w_energy, w_mom x3), nu_e w_mass, kappa
// w_energy; gpvol He (3c + dir); then the contravariant grad rho and grad T.  The adjoint line
// arrays of the five gradient fields (x3 directions) overlay the first 15 once they are read.
enum { F_RHO = 0, F_H, F_T, F_U0, F_U1, F_U2, W_M2, W_E, W_O0, W_O1, W_O2, W_NU, W_KE, F_G, F_V6 = F_G + 9, NF_ALL = F_V6 + 6 };
constexpr int kDtab = 32;  // D rows, then D^T rows

struct VjpArgs {
  int nelem;
  const int32_t* __restrict__ econn;
  const double* __restrict__ geo;
  const double* __restrict__ mue;        // internal [e][64]
  const double* __restrict__ musgs;      // internal [e][64] frozen SGS viscosity, or null
  const double* __restrict__ rho;
  const double* __restrict__ q0;
  const double* __restrict__ q1;
  const double* __restrict__ q2;
  const double* __restrict__ E;
  const double* __restrict__ mu_factor;
  const double* __restrict__ w;          // seeds / Ml: 5 columns of npoin (mass, mom x3, energy)
  int64_t npoin;
  double* out;                           // [(e*64 + d)*NRES + f] element-node adjoints (rho, q x3, E, 0)
  DMat D;
  DevParams prm;
};

__device__ __forceinline__ void load4(const double* p, double (&w)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
}

// Keeps the line passes apart: without it the compiler carries the line values of one pass over to
// the next in registers (up to 192 doubles) and spills them.
__device__ __forceinline__ void pass_fence() { asm volatile("" ::: "memory"); }

// Resident CTAs per SM the register budget must allow: 6 (168 registers, 48 bytes of spill, total enthalpy 4)
// 172 us for the whole call at 27^3; 8 (128 registers) 206 us; 4 without spill 186 us.
#ifndef SOD_VJP_MIN_BLOCKS
#define SOD_VJP_MIN_BLOCKS 6
#endif
// TOTH: flag_total_enthalpy (energy convection of full_convec_ijk_H)
template <bool TOTH>
__global__ void __launch_bounds__(64, SOD_VJP_MIN_BLOCKS) k_rhs_vjp(const VjpArgs a) {
  __shared__ __align__(16) double sm[NF_ALL * FSTRIDE];
  __shared__ __align__(16) double dtab[kDtab];
  const int e = blockIdx.x, lt = threadIdx.x;
  // lane bits (i0 j0 i1 j1 k): one shared-memory wavefront per xi and eta line load (see sod_rhs.cu)
  const int i = (lt & 1) | ((lt >> 1) & 2), j = ((lt >> 1) & 1) | ((lt >> 2) & 2), k = lt >> 4;
  const int d = i + 4 * j + 16 * k, s = sidx(i, j, k);
  if (lt < 32) dtab[lt] = lt < 16 ? a.D.d[lt >> 2][lt & 3] : a.D.d[lt & 3][(lt >> 2) & 3];
  const double* Ge = a.geo + (size_t)e * NGEO * NN;
  const int n = a.econn[(size_t)e * NN + d];
  const int64_t N = a.npoin;
  const double g = a.prm.gamma;
  const double rho = a.rho[n];
  const double qv[3] = {a.q0[n], a.q1[n], a.q2[n]};
  const double Et = a.E[n];
  const double wm = a.w[n], we = a.w[n + 4 * N];
  const double wmo[3] = {a.w[n + N], a.w[n + 2 * N], a.w[n + 3 * N]};
  const double mf = a.mu_factor[n];
  const double mue = a.mue[(size_t)e * NN + d];
  const double musgs = a.musgs ? a.musgs[(size_t)e * NN + d] : 0.0;
  double G[9];  // gpvol He
  {
    const double gpv = Ge[9 * NN + d];
#pragma unroll
    for (int c = 0; c < 9; ++c) G[c] = gpv * Ge[c * NN + d];
  }
  const double irho = 1.0 / rho;
  const double uv[3] = {qv[0] * irho, qv[1] * irho, qv[2] * irho};
  const double kk = 0.5 * (uv[0] * uv[0] + uv[1] * uv[1] + uv[2] * uv[2]);
  const double p = rho * (g - 1.0) * (Et * irho - kk);
  const double h = a.prm.g_gm1 * p * irho;
  const double T = p * irho * a.prm.inv_Rgas;
  const double Ht = h + kk;
  const double CpPr = a.prm.CpPr;
  const double muf = mf * kC1 * (T * sqrt(T)) / (T + kS);
  // elem_diffu.f90: the molecular part of the stress carries rho mu_sgs (mu_fgp), the heat flux
  // Cp/0.9 rho mu_sgs; both enter the reverse sweep through rho
  const double mufgp = muf + rho * musgs;
  {
    sm[F_RHO * FSTRIDE + s] = rho;
    sm[F_H * FSTRIDE + s] = Ht;
    sm[F_T * FSTRIDE + s] = T;
    sm[W_M2 * FSTRIDE + s] = 2.0 * wm;
    sm[W_E * FSTRIDE + s] = we;
    sm[W_NU * FSTRIDE + s] = a.prm.c_rho * mue * irho * wm;
    sm[W_KE * FSTRIDE + s] = (muf * CpPr + a.prm.c_ener * mue * CpPr + a.prm.Cp09 * rho * musgs) * we;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      sm[(F_U0 + c) * FSTRIDE + s] = uv[c];
      sm[(W_O0 + c) * FSTRIDE + s] = wmo[c];
    }
#pragma unroll
    for (int c = 0; c < 9; ++c) sm[(F_G + c) * FSTRIDE + s] = G[c];
  }
  __syncthreads();
  constexpr int stride[3] = {1, 4, PLANE};
  const int line[3] = {sidx(0, j, k), sidx(i, 0, k), sidx(i, j, 0)};
  const int row[3] = {i, j, k};

  // ---------------- convection and pressure: both roles of every line pair ----------------
  double rb = 0.0, Hb = 0.0, pb = 0.0;
  double ub[3] = {0.0, 0.0, 0.0};
  // D along the seed lines of the energy and momentum (the adjoint of pass 2's D^T), back to physical
  // components: adjoints of tau u and tau, gpvol He(r,:) . (D S)
  double tUb[3] = {0.0, 0.0, 0.0};
  double taub[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  {
    double X1 = 0.0, gb = 0.0;
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      double w1[4], w2[4], Y1 = 0.0, l1 = 0.0, lo[3] = {0.0, 0.0, 0.0};
      load4(dtab + 4 * row[dir], w1);
      load4(dtab + 16 + 4 * row[dir], w2);
#pragma unroll
      for (int m = 0; m < NP1; ++m) {
        const double* f = sm + line[dir] + m * stride[dir];
        const double r_ = f[F_RHO * FSTRIDE], H_ = f[F_H * FSTRIDE];
        const double br = rho + r_, bH = Ht + H_;
        const double bu[3] = {uv[0] + f[F_U0 * FSTRIDE], uv[1] + f[F_U1 * FSTRIDE], uv[2] + f[F_U2 * FSTRIDE]};
        const double gl[3] = {f[(F_G + dir) * FSTRIDE], f[(F_G + 3 + dir) * FSTRIDE], f[(F_G + 6 + dir) * FSTRIDE]};
        const double el = f[W_E * FSTRIDE];
        const double ol[3] = {f[W_O0 * FSTRIDE], f[W_O1 * FSTRIDE], f[W_O2 * FSTRIDE]};
        const double bV1 = G[dir] * bu[0] + G[3 + dir] * bu[1] + G[6 + dir] * bu[2];
        const double bV2 = gl[0] * bu[0] + gl[1] * bu[1] + gl[2] * bu[2];
        double Q1 = 2.0 * wm + (wmo[0] * bu[0] + wmo[1] * bu[1] + wmo[2] * bu[2]);
        double Q2 = f[W_M2 * FSTRIDE] + (ol[0] * bu[0] + ol[1] * bu[1] + ol[2] * bu[2]);
        if constexpr (!TOTH) {
          Q1 += we * bH;
          Q2 += el * bH;
        }
        const double c1 = w1[m] * br, c2 = w2[m] * br;
        const double P1 = w1[m] * bV1, P2 = w2[m] * bV2;
        rb += P1 * Q1 + P2 * Q2;
        const double x2 = c2 * bV2;
        X1 += c1 * bV1;
        double y2 = c2 * Q2;
        if constexpr (TOTH) {
          // the energy flux is (G_x + G_l)(V_x + V_l) / 2 with G = rho H
          const double bg = rho * Ht + r_ * H_;
          gb += P1 * we + P2 * el;
          Y1 += c1 * Q1 + 2.0 * (w1[m] * bg) * we;
          y2 += 2.0 * (w2[m] * bg) * el;
        } else {
          Hb += x2 * el;
          Y1 += c1 * Q1;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) ub[c] += x2 * ol[c] + y2 * gl[c];
        pb += w2[m] * (gl[0] * ol[0] + gl[1] * ol[1] + gl[2] * ol[2]);
        l1 += w1[m] * el;
#pragma unroll
        for (int c = 0; c < 3; ++c) lo[c] += w1[m] * ol[c];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double hr = G[3 * r + dir];
        tUb[r] += hr * l1;
#pragma unroll
        for (int c = 0; c < 3; ++c) taub[c][r] += hr * lo[c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) ub[c] += Y1 * G[3 * c + dir];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) ub[c] = 0.25 * (ub[c] + X1 * wmo[c]);
    rb *= 0.25;
    if constexpr (TOTH) {
      rb += 0.5 * Ht * gb;
      Hb = 0.5 * rho * gb;
    } else {
      Hb = 0.25 * (Hb + X1 * we);
    }
  }

  // ---------------- forward gradients, and D along the seed lines ----------------
  pass_fence();
  const double igpv = 1.0 / Ge[9 * NN + d];  // G holds gpvol He; the forward gradients want He
  // (with the other two seeds, of grad rho and grad T)
  double gU[3][3];
  double gRhob[3] = {0.0, 0.0, 0.0}, gTb[3] = {0.0, 0.0, 0.0};
  {
    double gRho[3] = {0.0, 0.0, 0.0}, gT[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) gU[c][r] = 0.0;
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      double w1[4];
      load4(dtab + 4 * row[dir], w1);
      double lr = 0.0, lT = 0.0, lu[3] = {0.0, 0.0, 0.0}, l0 = 0.0, l2 = 0.0;
#pragma unroll
      for (int m = 0; m < NP1; ++m) {
        const double* f = sm + line[dir] + m * stride[dir];
        lr += w1[m] * f[F_RHO * FSTRIDE];
        lT += w1[m] * f[F_T * FSTRIDE];
        l0 += w1[m] * f[W_NU * FSTRIDE];
        l2 += w1[m] * f[W_KE * FSTRIDE];
#pragma unroll
        for (int c = 0; c < 3; ++c) lu[c] += w1[m] * f[(F_U0 + c) * FSTRIDE];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double hr = G[3 * r + dir];
        gRho[r] += hr * lr;
        gT[r] += hr * lT;
        gRhob[r] += hr * l0;
        gTb[r] += hr * l2;
#pragma unroll
        for (int c = 0; c < 3; ++c) gU[c][r] += hr * lu[c];
      }
    }
    // contravariant grad rho and grad T fluxes (gpvol He^T grad) for the weak divergences below
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      const double h0 = G[dir] * igpv, h1 = G[3 + dir] * igpv, h2 = G[6 + dir] * igpv;
      sm[(F_V6 + dir) * FSTRIDE + s] = h0 * gRho[0] + h1 * gRho[1] + h2 * gRho[2];
      sm[(F_V6 + 3 + dir) * FSTRIDE + s] = h0 * gT[0] + h1 * gT[1] + h2 * gT[2];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) gU[c][r] *= igpv;
  }
  // tauU_r = sum_c tau_rc u_c;  tau_rc = (mu_fgp+mue)(du_r/dx_c + du_c/dx_r) - delta_rc mu_fgp 2/3 div u,
  // mu_fgp = muf + rho musgs
  double Tb = 0.0;
  double gUb[3][3];
  {
    const double divU = gU[0][0] + gU[1][1] + gU[2][2];
    const double mut = mufgp + mue;
    double mufgpb = 0.0, tr = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double sg = gU[r][c] + gU[c][r];
        double tau = mut * sg;
        if (r == c) tau -= mufgp * (2.0 / 3.0) * divU;
        ub[c] += tUb[r] * tau;
        taub[r][c] += tUb[r] * uv[c];
        mufgpb += taub[r][c] * sg;
      }
#pragma unroll
    for (int r = 0; r < 3; ++r) tr += taub[r][r];
    mufgpb -= (2.0 / 3.0) * divU * tr;
    const double divUb = -mufgp * (2.0 / 3.0) * tr;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) gUb[r][c] = mut * (taub[r][c] + taub[c][r]) + (r == c ? divUb : 0.0);
    rb += mufgpb * musgs;
    Tb = mufgpb;  // d/d muf, finished below
  }
  __syncthreads();  // every line read of the first 22 arrays done; V6 complete
  // nu_e and kappa belong to the output node (elem_diffu.f90:143-193)
  {
    double w2[3][4];
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) load4(dtab + 16 + 4 * row[dir], w2[dir]);
    double dr = 0.0, dT = 0.0;
#pragma unroll
    for (int dir = 0; dir < 3; ++dir)
#pragma unroll
      for (int m = 0; m < NP1; ++m) {
        const double* f = sm + line[dir] + m * stride[dir];
        dr += w2[dir][m] * f[(F_V6 + dir) * FSTRIDE];
        dT += w2[dir][m] * f[(F_V6 + 3 + dir) * FSTRIDE];
      }
    rb += wm * dr * (-a.prm.c_rho * mue * irho * irho) + we * dT * a.prm.Cp09 * musgs;
    Tb += we * dT * CpPr;
    // gradient adjoints -> iso adjoints (He^T) on the arrays the passes above no longer read
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      const double h0 = G[dir] * igpv, h1 = G[3 + dir] * igpv, h2 = G[6 + dir] * igpv;
      auto put = [&](int f, const double* gb) { sm[(3 * f + dir) * FSTRIDE + s] = h0 * gb[0] + h1 * gb[1] + h2 * gb[2]; };
      put(0, gUb[0]);
      put(1, gUb[1]);
      put(2, gUb[2]);
      put(3, gRhob);
      put(4, gTb);
    }
    __syncthreads();
    double lT = 0.0;
#pragma unroll
    for (int dir = 0; dir < 3; ++dir)
#pragma unroll
      for (int m = 0; m < NP1; ++m) {
        const double* f = sm + line[dir] + m * stride[dir];
#pragma unroll
        for (int c = 0; c < 3; ++c) ub[c] += w2[dir][m] * f[(3 * c + dir) * FSTRIDE];
        rb += w2[dir][m] * f[(9 + dir) * FSTRIDE];
        lT += w2[dir][m] * f[(12 + dir) * FSTRIDE];
      }
    // Sutherland (mod_fluid_viscosity.f90:37)
    const double dmuf_dT = mf * kC1 * (1.5 * sqrt(T) * (T + kS) - T * sqrt(T)) / ((T + kS) * (T + kS));
    Tb = Tb * dmuf_dT + lT;
  }

  // H = h + k, EOS and u = q/rho in reverse (time_integ.f90:266-285)
  double kb = Hb;
  pb += Hb * a.prm.g_gm1 * irho;
  rb += -Hb * h * irho;
  pb += Tb * irho * a.prm.inv_Rgas;
  rb += -Tb * T * irho;
  const double Eb = (g - 1.0) * pb;
  rb += -(g - 1.0) * kk * pb;
  kb += -(g - 1.0) * rho * pb;
  double qb[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    ub[c] += uv[c] * kb;
    qb[c] = ub[c] * irho;
    rb += -uv[c] * qb[c];
  }
  store_res6<double>(a.out, (size_t)e * NN + d, rb, qb[0], qb[1], qb[2], Eb, 0.0);
}

}  // namespace adj
}  // namespace sod

// ---------------------------------------------------------------------------------------------
// node-side kernels of the adjoint: seeds, ordered gathers, stage states
// ---------------------------------------------------------------------------------------------
namespace sod {
namespace adj {

struct Cols5 {
  const double* c[5];
};
struct MCols5 {
  double* c[5];
};

// w = scale * src / Ml (scale = -dt * coef when dt is given, else 1)
__global__ void k_seed(int64_t N, Cols5 src, const double* __restrict__ Ml, const double* __restrict__ dt,
                       double coef, double* __restrict__ w, MCols5 keep) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const double sc = dt ? -(*dt) * coef : 1.0;
  const double inv = 1.0 / Ml[n];
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    const double v = src.c[f][n];
    w[f * N + n] = sc * v * inv;
    if (keep.c[f]) keep.c[f][n] = v;
  }
}

// Ordered gather of the element-node adjoints [e][6][64] (ascending element order, like the
// forward assembly), plus extra ([5][npoin], or null); Ybar = sum; out = Ybar (mode 0),
// out += Ybar (mode 1) or out = ybar + Ybar (mode 2: the first accumulation, so that out needs no copy
// of ybar before it and may be the array ybar was kept from); when wnext is set:
// wnext = -dt (cb * ybar + ca * Ybar) / Ml.
__global__ void __launch_bounds__(256) k_gather_vjp(int64_t N, const int32_t* __restrict__ ptr,
                                                    const int32_t* __restrict__ idx, const double* __restrict__ el,
                                                    MCols5 out, int mode, const double* __restrict__ ybar,
                                                    const double* __restrict__ Ml, const double* __restrict__ dt,
                                                    double cb, double ca, double* __restrict__ wnext,
                                                    const double* __restrict__ extra) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double r[6] = {0, 0, 0, 0, 0, 0};
  gather_rows<double>(el, idx, ptr[n], ptr[n + 1], r);
  if (extra) {  // the wall model's node-level adjoint
#pragma unroll
    for (int f = 0; f < 5; ++f) r[f] += extra[f * N + n];
  }
  double yb[5];
  if (wnext || mode == 2) {
#pragma unroll
    for (int f = 0; f < 5; ++f) yb[f] = ybar[f * N + n];
  }
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    if (mode == 0) out.c[f][n] = r[f];
    else out.c[f][n] = (mode == 1 ? out.c[f][n] : yb[f]) + r[f];
  }
  if (wnext) {
    const double sc = -(*dt) / Ml[n];
#pragma unroll
    for (int f = 0; f < 5; ++f) wnext[f * N + n] = sc * (cb * yb[f] + ca * r[f]);
  }
}

// acc += Ybar (the adjoint of a stage state after the boundary routine's adjoint); when wnext
// is set: wnext = -dt (cb * ybar + ca * Ybar) / Ml
__global__ void __launch_bounds__(256) k_accum_seed(int64_t N, const double* __restrict__ Yb, MCols5 acc,
                                                    const double* __restrict__ ybar, const double* __restrict__ Ml,
                                                    const double* __restrict__ dt, double cb, double ca,
                                                    double* __restrict__ wnext) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double r[5];
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    r[f] = Yb[f * N + n];
    acc.c[f][n] += r[f];
  }
  if (wnext) {
    const double sc = -(*dt) / Ml[n];
#pragma unroll
    for (int f = 0; f < 5; ++f) wnext[f * N + n] = sc * (cb * ybar[f * N + n] + ca * r[f]);
  }
}

// stage state: ys = y - coef * dt * gather(rel)/Ml   (time_integ.f90:301-318)
__global__ void __launch_bounds__(256) k_stage_state(int64_t N, const int32_t* __restrict__ ptr,
                                                     const int32_t* __restrict__ idx, const double* __restrict__ el,
                                                     const double* __restrict__ Ml, const double* __restrict__ dt,
                                                     double coef, Cols5 y, const double* __restrict__ src,
                                                     const double* __restrict__ wmc, double* __restrict__ ys) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double r[6] = {0, 0, 0, 0, 0, 0};
  gather_rows<double>(el, idx, ptr[n], ptr[n + 1], r);
  // same operation order as the forward stage gather, so the stage states match it bit for bit
  const double ml = Ml[n];
  if (src) {
#pragma unroll
    for (int d = 0; d < 3; ++d) r[1 + d] -= ml * src[d * N + n];
  }
  if (wmc) {
#pragma unroll
    for (int d = 0; d < 3; ++d) r[1 + d] += wmc[d * N + n];
  }
  const double da = (*dt) * coef, iml = 1.0 / ml;
#pragma unroll
  for (int f = 0; f < 5; ++f) ys[f * N + n] = y.c[f][n] - da * (r[f] * iml);
}

// y0 - dt sum_s b_s R_s from the stage states (dt R_1 = 2 (y0 - Y2), dt R_2 = 2 (y0 - Y3),
// dt R_3 = y0 - Y4) and R_4 = gather(rel)/Ml (+ the source term): the forward's updated state at
// nodes the routines do not modify
__global__ void __launch_bounds__(256) k_final_pre(int64_t N, const int32_t* __restrict__ ptr,
                                                   const int32_t* __restrict__ idx, const double* __restrict__ el,
                                                   const double* __restrict__ Ml, const double* __restrict__ dt,
                                                   Cols5 y, const double* __restrict__ Y2,
                                                   const double* __restrict__ Y3, const double* __restrict__ Y4,
                                                   const double* __restrict__ src, const double* __restrict__ wmc,
                                                   double* __restrict__ zf) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double r[6] = {0, 0, 0, 0, 0, 0};
  gather_rows<double>(el, idx, ptr[n], ptr[n + 1], r);
  const double ml = Ml[n];
  if (src) {
#pragma unroll
    for (int d = 0; d < 3; ++d) r[1 + d] -= ml * src[d * N + n];
  }
  if (wmc) {
#pragma unroll
    for (int d = 0; d < 3; ++d) r[1 + d] += wmc[d * N + n];
  }
  const double h = (*dt) / 6.0;
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    const double y0 = y.c[f][n];
    const double acc = (y0 - Y2[f * N + n]) / 3.0 + 2.0 * (y0 - Y3[f * N + n]) / 3.0 + (y0 - Y4[f * N + n]) / 3.0;
    zf[f * N + n] = y0 - acc - h * (r[f] / ml);
  }
}

static int launch_vjp(SodMesh* m, const double* rho, const double* q0, const double* q1, const double* q2,
                      const double* E, const double* mu_factor, const double* musgs, const double* w, cudaStream_t st) {
  VjpArgs a;
  a.nelem = m->nelem;
  a.econn = m->econn;
  a.geo = m->geo64;
  a.mue = m->mue_int;
  a.musgs = musgs;
  a.rho = rho; a.q0 = q0; a.q1 = q1; a.q2 = q2; a.E = E;
  a.mu_factor = mu_factor;
  a.w = w;
  a.npoin = m->npoin;
  a.out = reinterpret_cast<double*>(m->buf.rel);
  a.D = m->D;
  a.prm = m->prm;
  if (m->prm.total_enthalpy)
    k_rhs_vjp<true><<<m->nelem, NN, 0, st>>>(a);
  else
    k_rhs_vjp<false><<<m->nelem, NN, 0, st>>>(a);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

static int ensure_adj(SodMesh* m, size_t len) {
  if (m->adj_len >= len) return SOD_OK;
  if (m->adj) cudaFree(m->adj);
  m->adj = nullptr;
  m->adj_len = 0;
  SOD_CUDA(cudaMalloc(&m->adj, len * sizeof(double)));
  m->adj_len = len;
  return SOD_OK;
}

static inline unsigned nblk(int64_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace adj
}  // namespace sod

using namespace sod;
using namespace sod::adj;

extern "C" {

int sod_rhs_vjp(SodMesh* m, const double* rho, const double* q, const double* E, const double* mu_e,
                const double* mu_factor, const double* bar_Rmass, const double* bar_Rmom, const double* bar_Rener,
                double* grad_rho, double* grad_q, double* grad_E, sod_stream_t stream) {
  SOD_ARG(m && rho && q && E && mu_e && mu_factor, "inputs null");
  SOD_ARG(bar_Rmass && bar_Rmom && bar_Rener && grad_rho && grad_q && grad_E, "adjoint arrays null");
  if (m->has_slaves) {
    set_error("sod_rhs_vjp on a mesh with periodic slave rows (lpoin_w) is not supported");
    return SOD_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  const int64_t N = m->npoin;
  rc = ensure_adj(m, 5 * (size_t)N);
  if (rc) return rc;
  rc = mesh_ref_to_internal_elem(m, mu_e, m->mue_int, st);
  if (rc) return rc;
  double* w = m->adj;
  Cols5 src{{bar_Rmass, bar_Rmom, bar_Rmom + N, bar_Rmom + 2 * N, bar_Rener}};
  MCols5 none{{nullptr, nullptr, nullptr, nullptr, nullptr}};
  k_seed<<<nblk(N), 256, 0, st>>>(N, src, m->Ml, nullptr, 1.0, w, none);
  SOD_CHECK_LAUNCH();
  rc = launch_vjp(m, rho, q, q + N, q + 2 * N, E, mu_factor, nullptr, w, st);
  if (rc) return rc;
  const double* wmb = nullptr;
  if (m->wmodel.nw > 0) {
    rc = wall_model_vjp(m, rho, q, E, mu_factor, w, st);
    if (rc) return rc;
    wmb = m->wmodel.wmbar;
  }
  MCols5 out{{grad_rho, grad_q, grad_q + N, grad_q + 2 * N, grad_E}};
  k_gather_vjp<<<nblk(N), 256, 0, st>>>(N, m->n2e_ptr, m->n2e, reinterpret_cast<const double*>(m->buf.rel), out, 0,
                                         nullptr, nullptr, nullptr, 0.0, 0.0, nullptr, wmb);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

int sod_rk4_step_vjp(SodMesh* m, const double* rho, const double* q, const double* E, const double* mu_e,
                     const double* mu_sgs, const double* mu_factor, const double* dt_dev, const double* stages,
                     const double* bar_rho, const double* bar_q, const double* bar_E, double* out_rho, double* out_q,
                     double* out_E, sod_stream_t stream) {
  SOD_ARG(m && rho && q && E && mu_e && mu_factor && dt_dev, "inputs null");
  SOD_ARG(bar_rho && bar_q && bar_E && out_rho && out_q && out_E, "adjoint arrays null");
  if (m->has_slaves) {
    set_error("sod_rk4_step_vjp on a mesh with periodic slave rows (lpoin_w) is not supported");
    return SOD_ERR_UNSUPPORTED;
  }
  // boundaries and buffer zone: the routines' adjoints after every stage VJP and on the seed
  const bool has_bc = m->bc.nb > 0, has_zone = m->zone.nb > 0;
  const bool bc = has_bc || has_zone;
  const bool ff = has_bc && m->bc.nff > 0;
  const bool slip = has_bc && m->bc.has_slip;
  // wall model: its forward term in the stage residuals the adjoint rebuilds, its own adjoint in
  // every stage's gather
  const double* wmc = m->wmodel.nw > 0 ? m->wmodel.contrib : nullptr;
  // far-field nodes with a buffer zone: the final routine's input at the lnbn targets from the
  // stage residuals gathered there (the zone changes the stage states the reconstruction uses)
  const bool ffz = ff && has_zone;
  NvtxRange range("sod rk4 step vjp");
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_step_buffers(m, false);
  if (rc) return rc;
  // LES: the step's frozen mu_sgs in the internal layout (the forward re-derives it per step)
  const double* musgs = nullptr;
  if (m->prm.flag_les == 1 && mu_sgs) {
    SodState tmp{};
    tmp.mu_sgs = const_cast<double*>(mu_sgs);
    rc = les_in(m, &tmp, st);
    if (rc) return rc;
    musgs = m->musgs_int;
  }
  const int64_t N = m->npoin;
  // Y = B(Z(y)) for the buffer zone Z and the boundary routine B; adjoint Z^T B^T
  auto pre_stage = [&](double* ys, int stage_of) -> int {
    if (has_zone)
      if (int r = zone_stage(m, ys, st)) return r;
    return has_bc ? bc_stage(m, ys, stage_of, st) : SOD_OK;
  };
  // y: the state the boundary routine read (its far-field nodes' lnbn rows); app: which of the
  // step's five applications (stages 1-4, the update) for the slip walls
  auto pre_adjoint = [&](double* vbar, const double* y, int app) -> int {
    if (has_bc)
      if (int r = bc_adjoint(m, vbar, y, app, st)) return r;
    return has_zone ? zone_adjoint(m, vbar, st) : SOD_OK;
  };
  // scratch: ybar copy | w | (with boundaries: Y1 | Ybar of a stage) | (far-field: the updated
  // state before the routine) | (ys2 ys3 ys4 when the stages are not given)   (5 columns each)
  const size_t base = bc ? (ff ? 25 : 20) : 10;
  rc = ensure_adj(m, (base + (stages ? 0 : 15)) * (size_t)N);
  if (rc) return rc;
  rc = mesh_ref_to_internal_elem(m, mu_e, m->mue_int, st);
  if (rc) return rc;
  double* yb = m->adj;
  double* w = m->adj + 5 * N;
  double* y1s = bc ? m->adj + 10 * N : nullptr;   // first stage state B(y0)
  double* Ybs = bc ? m->adj + 15 * N : nullptr;   // adjoint of one stage state
  double* zf = ff ? m->adj + 20 * N : nullptr;     // y0 - dt sum b_s R_s, before the final routine
  const double* ys[3];
  const double* rel = reinterpret_cast<const double*>(m->buf.rel);
  Cols5 y0{{rho, q, q + N, q + 2 * N, E}};
  Cols5 Y1 = y0;
  if (bc) {
    for (int f = 0; f < 5; ++f)
      SOD_CUDA(cudaMemcpyAsync(y1s + f * N, y0.c[f], N * sizeof(double), cudaMemcpyDeviceToDevice, st));
    rc = pre_stage(y1s, 1);
    if (rc) return rc;
    Y1 = Cols5{{y1s, y1s + N, y1s + 2 * N, y1s + 3 * N, y1s + 4 * N}};
  }
  if (stages) {
    for (int t = 0; t < 3; ++t) ys[t] = stages + (size_t)t * 5 * N;
  } else {
    // forward recompute of the stage states (mu_e and dt frozen)
    const int epb = rhs_epb(m, false);
    const double acoef[3] = {0.5, 0.5, 1.0};
    Cols5 cur = Y1;
    for (int t = 0; t < 3; ++t) {
      double* b = m->adj + (base + 5 * t) * N;
      if (wmc) {
        rc = wall_model_stage(m, cur.c[0], cur.c[1], cur.c[4], mu_factor, st);
        if (rc) return rc;
      }
      rc = launch_rhs(m, false, epb, cur.c[0], cur.c[1], cur.c[2], cur.c[3], cur.c[4], mu_factor, musgs, st);
      if (rc) return rc;
      if (slip) {
        rc = bc_slip_residuals(m, t + 1, rel, st);
        if (rc) return rc;
      }
      if (ffz) {
        rc = bc_ff_residuals(m, t + 1, rel, st);
        if (rc) return rc;
      }
      k_stage_state<<<nblk(N), 256, 0, st>>>(N, m->n2e_ptr, m->n2e, rel, m->Ml, dt_dev, acoef[t], y0, m->source, wmc,
                                             b);
      SOD_CHECK_LAUNCH();
      if (bc) {
        rc = pre_stage(b, t + 2);
        if (rc) return rc;
      }
      ys[t] = b;
      cur = Cols5{{b, b + N, b + 2 * N, b + 3 * N, b + 4 * N}};
    }
  }
  if (ff || slip) {
    const int epb = rhs_epb(m, false);
    if ((slip || ffz) && stages) {
      // the stage residuals at the slip nodes / lnbn targets (the recompute gathered them already)
      for (int t = 0; t < 3; ++t) {
        const double* yt = t == 0 ? y1s : ys[t - 1];
        if (wmc) {
          rc = wall_model_stage(m, yt, yt + N, yt + 4 * N, mu_factor, st);
          if (rc) return rc;
        }
        rc = launch_rhs(m, false, epb, yt, yt + N, yt + 2 * N, yt + 3 * N, yt + 4 * N, mu_factor, musgs, st);
        if (rc) return rc;
        if (slip) {
          rc = bc_slip_residuals(m, t + 1, rel, st);
          if (rc) return rc;
        }
        if (ffz) {
          rc = bc_ff_residuals(m, t + 1, rel, st);
          if (rc) return rc;
        }
      }
    }
    // the updated state the final routine reads, at the far-field nodes' lnbn nodes (interior:
    // there the stage states equal their pre-routine values, so dt R_s = (y0 - Y_{s+1}) / a_{s+1}
    // for s = 1..3); R_4 from one more RHS evaluation at Y4
    const double* y4 = ys[2];
    if (wmc) {
      rc = wall_model_stage(m, y4, y4 + N, y4 + 4 * N, mu_factor, st);
      if (rc) return rc;
    }
    rc = launch_rhs(m, false, epb, y4, y4 + N, y4 + 2 * N, y4 + 3 * N, y4 + 4 * N, mu_factor, musgs, st);
    if (rc) return rc;
    if (ffz) {
      rc = bc_ff_residuals(m, 4, rel, st);
      if (rc) return rc;
      rc = bc_ff_final(m, rho, q, E, dt_dev, zf, st);
      if (rc) return rc;
    } else if (ff) {
      k_final_pre<<<nblk(N), 256, 0, st>>>(N, m->n2e_ptr, m->n2e, rel, m->Ml, dt_dev, y0, ys[0], ys[1], ys[2],
                                           m->source, wmc, zf);
      SOD_CHECK_LAUNCH();
    }
    if (slip) {
      // slip walls: pre-routine rho, q of the five applications and the velocities they read
      rc = bc_slip_residuals(m, 4, rel, st);
      if (rc) return rc;
      rc = bc_slip_prepare(m, rho, q, y1s, ys[0], ys[1], dt_dev, st);
      if (rc) return rc;
    }
  }
  // reverse sweep: kbar4 = -dt/6 ybar, Ybar4 = J4^T kbar4, kbar3 = -dt (ybar/3 + Ybar4), ...
  // (with boundaries ybar is first mapped through the final routine's adjoint)
  Cols5 src{{bar_rho, bar_q, bar_q + N, bar_q + 2 * N, bar_E}};
  MCols5 keep{{yb, yb + N, yb + 2 * N, yb + 3 * N, yb + 4 * N}};
  if (bc) {
    for (int f = 0; f < 5; ++f)
      SOD_CUDA(cudaMemcpyAsync(keep.c[f], src.c[f], N * sizeof(double), cudaMemcpyDeviceToDevice, st));
    rc = pre_adjoint(yb, zf, 4);
    if (rc) return rc;
    src = Cols5{{yb, yb + N, yb + 2 * N, yb + 3 * N, yb + 4 * N}};
    keep = MCols5{{nullptr, nullptr, nullptr, nullptr, nullptr}};
  }
  k_seed<<<nblk(N), 256, 0, st>>>(N, src, m->Ml, dt_dev, 1.0 / 6.0, w, keep);
  SOD_CHECK_LAUNCH();
  keep = MCols5{{yb, yb + N, yb + 2 * N, yb + 3 * N, yb + 4 * N}};
  MCols5 acc{{out_rho, out_q, out_q + N, out_q + 2 * N, out_E}};
  // with boundaries acc = ybar (copied from the kept columns, so out may alias bar); without, the
  // first stage's gather writes ybar + Ybar4
  if (bc)
    for (int f = 0; f < 5; ++f)
      SOD_CUDA(cudaMemcpyAsync(acc.c[f], keep.c[f], N * sizeof(double), cudaMemcpyDeviceToDevice, st));
  if (slip) {
    // the update's slip walls read the velocity q/rho of y0 itself
    rc = bc_slip_push(m, rho, q, out_rho, out_q, st);
    if (rc) return rc;
  }
  const double cb[4] = {1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0, 0.0};
  const double ca[4] = {1.0, 0.5, 0.5, 0.0};
  for (int stage = 4; stage >= 1; --stage) {
    const Cols5 ysrc = stage == 1 ? Y1
                                  : Cols5{{ys[stage - 2], ys[stage - 2] + N, ys[stage - 2] + 2 * N,
                                           ys[stage - 2] + 3 * N, ys[stage - 2] + 4 * N}};
    rc = launch_vjp(m, ysrc.c[0], ysrc.c[1], ysrc.c[2], ysrc.c[3], ysrc.c[4], mu_factor, musgs, w, st);
    if (rc) return rc;
    const double* wmb = nullptr;
    if (wmc) {
      rc = wall_model_vjp(m, ysrc.c[0], ysrc.c[1], ysrc.c[4], mu_factor, w, st);
      if (rc) return rc;
      wmb = m->wmodel.wmbar;
    }
    const int t = 4 - stage;
    if (!bc) {
      k_gather_vjp<<<nblk(N), 256, 0, st>>>(N, m->n2e_ptr, m->n2e, rel, acc, t == 0 ? 2 : 1, yb, m->Ml, dt_dev, cb[t], ca[t],
                                             stage > 1 ? w : nullptr, wmb);
      SOD_CHECK_LAUNCH();
    } else {
      // Ybar of the post-routine stage state, through the stage routine's adjoint, then accumulated
      MCols5 yc{{Ybs, Ybs + N, Ybs + 2 * N, Ybs + 3 * N, Ybs + 4 * N}};
      k_gather_vjp<<<nblk(N), 256, 0, st>>>(N, m->n2e_ptr, m->n2e, rel, yc, 0, nullptr, nullptr, nullptr, 0.0, 0.0,
                                             nullptr, wmb);
      SOD_CHECK_LAUNCH();
      const double* Ysv = stage == 1 ? y1s : ys[stage - 2];
      if (slip && stage < 4) {
        // stage s + 1's slip walls read the velocity of this stage's post-routine state
        rc = bc_slip_push(m, Ysv, Ysv + N, Ybs, Ybs + N, st);
        if (rc) return rc;
      }
      rc = pre_adjoint(Ybs, Ysv, stage - 1);
      if (rc) return rc;
      k_accum_seed<<<nblk(N), 256, 0, st>>>(N, Ybs, acc, yb, m->Ml, dt_dev, cb[t], ca[t], stage > 1 ? w : nullptr);
      SOD_CHECK_LAUNCH();
    }
  }
  return SOD_OK;
}

int sod_bc_dirichlet_prim_vjp(SodMesh* m, const double* rho, const double* q, const double* E, double* bar_rho,
                              double* bar_q, double* bar_E, sod_stream_t stream) {
  SOD_ARG(m && bar_rho && bar_q && bar_E, "null argument");
  SOD_ARG(m->bc.nb > 0, "no boundary nodes registered (sod_mesh_set_boundaries)");
  if (m->has_slaves) {
    set_error("sod_bc_dirichlet_prim_vjp on a mesh with periodic slave rows (lpoin_w) is not supported");
    return SOD_ERR_UNSUPPORTED;
  }
  SOD_ARG(m->bc.nff == 0 || (rho && q && E), "far-field adjoint needs the state the routine read");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t N = m->npoin;
  int rc = ensure_adj(m, 10 * N);
  if (rc) return rc;
  double* v = m->adj;
  double* y = m->adj + 5 * N;
  const double* bars[3] = {bar_rho, bar_q, bar_E};
  const size_t cnt[3] = {N, 3 * N, N}, off[3] = {0, N, 4 * N};
  for (int t = 0; t < 3; ++t) {
    SOD_CUDA(cudaMemcpyAsync(v + off[t], bars[t], cnt[t] * sizeof(double), cudaMemcpyDeviceToDevice, st));
    if (m->bc.nff > 0) {
      const double* ys[3] = {rho, q, E};
      SOD_CUDA(cudaMemcpyAsync(y + off[t], ys[t], cnt[t] * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
  }
  rc = bc_adjoint(m, v, m->bc.nff > 0 ? y : nullptr, -1, st);
  if (rc) return rc;
  double* outs[3] = {bar_rho, bar_q, bar_E};
  for (int t = 0; t < 3; ++t)
    SOD_CUDA(cudaMemcpyAsync(outs[t], v + off[t], cnt[t] * sizeof(double), cudaMemcpyDeviceToDevice, st));
  return SOD_OK;
}

}  // extern "C"

// Mixed-precision fused element RHS with packed FP32 arithmetic (sm_100a FFMA2).
//
// The reference element loops of full_convec_ijk (elem_convec.f90:211-460), full_diffusion_ijk
// (elem_diffu.f90:12-198) and generic_scalar_convec_ijk (elem_convec.f90:462-570) in FP32 on
// deviation fields.  Assembly, lumped mass, RK state and reductions stay FP64.
//
// The split forms of the reference are two-point flux sums: with D the line derivative
// (sum_m D[x][m] = 0), V(m) = sum_c He(c,dir)(x) u_c(m) the contravariant velocity formed with
// the output point's metric, V^ = (V_x + V_m)/2, r^ = (rho_x + rho_m)/2 and df = f_m - f_x, the
// quartets of elem_convec.f90:412-432 are
//   mass      Rm = rho div u + sum_dir sum_m D[x][m] V^ drho
//   f         f_x Rm + sum_dir sum_m D[x][m] V^ r^ df        f = u_c, H = h + k
//   entropy   eta div u + sum_dir sum_m D[x][m] V^ deta
//   (E+p)     G div u + sum_dir sum_m D[x][m] V^ dG          G = rho H, flag_total_enthalpy
// (both energy quartets on H: they are linear in (h, k)).  One pass over the 12 line points of 4
// slots serves the gradients and every product: no products are staged, none of the q, H, rho H,
// eta, h and k derivatives are formed, and the metric is folded into V before the sums instead of
// after them.
// With eta = (rho L_r + lam) / (gamma - 1), L = log p - gamma log rho, L_r its value at the element's
// node 0 and lam = rho (L - L_r), the entropy residual is (L_r Rm + the same functional of lam) /
// (gamma - 1), so lam (small) is differentiated and L_r enters once, at the end.
//
// Nodal fields are staged in shared memory as float2 pairs: one 8-byte shared load and one packed
// __ffma2_rn serve two fields, and the xi-lines are read as 16-byte loads.  Slots:
//   (u0,u1) (u2,H) (rho,lam) (p,T)                                 the nodal fields
//   u0 u1 u2 in FP64                                               for the velocity gradients
//   (gradRho^,tauU^)x3 (gradT^,tauX^)x3 (tauY^,tauZ^)x3            pass 2, one slot per direction
// ^ marks contravariant fluxes.  Every field is held as its deviation from an element reference
// (node 0, in FP64, before the FP32 cast); p and T from one that is affine in xi.
//
// Measured at 64^3 (262,144 elements, one launch): 0.827 ms, 1.254 ms with the 12 gradient fields
// and 25 staged-factor products of the quartets formed one by one.  Bounded by latency at 20
// resident warps per SM with the L1 data pipe ~70% and the issue slots ~60% busy; HBM floor 0.24 ms.
//
// Precision.  div u cancels by orders of magnitude and multiplies rho, H and eta, so its line sums and
// fold run in FP64.  The viscous terms differentiate twice, so an error in a gradient is raised by the
// ratio of the flux to its divergence, ~n for n elements across a wave: the velocity gradients are those
// FP64 line sums, rounded once, and T, like p, is held as the deviation from an affine reference (what is
// left is second order in the element size).  With both from constant references in FP32 the launch took
// 0.801 ms and the assembled viscous and heat terms were 2 to 3.5 times further from FP64 (shear, 48
// elements, 5% jitter: 1.4e-5 against 4.0e-6; heat flux 3.4e-6 against 1.1e-6).
// The momentum's sums are u . grad u: where it cancels between the three directions (a shear), the
// rounding of each term V^ r^ du counts against a small result.  So V_x rho_x times the precise line sum
// is split off and only the rest, second order in the element size, is summed point by point (14 us of
// the launch): error of a shear's momentum 6e-9 of rho u du/dy where the unsplit sums had 6.2e-8, and in a
// channel, where transport and viscous terms balance, 2.1e-7 of the residual against 2.3e-7 (24^3).
#include "sod_internal.cuh"
#include "sod_step_kernels.cuh"
#include <cmath>
#include <algorithm>

namespace sod {
namespace mx2 {

constexpr double kC1 = 0.000001458;
constexpr double kS = 110.4;
constexpr int NA = 4;    // nodal slots (field pairs)
constexpr int NU = 3;    // FP64 velocity slots
constexpr int NP2 = 9;   // pass-2 slots
constexpr int NSLOT = NA + NU + NP2;
// doubles per element ahead of the slots: rho, u, h, k of node 0; (p, T) of the nodes (0,0,0), (3,0,0),
// (0,3,0), (0,0,3); log p and log rho of node 0; then FP32 references (7 floats) and the slopes of (p, T) (3)
constexpr int R_P = 6, R_LOG = R_P + 8, R_F32 = R_LOG + 2, NREF = R_F32 + 4 + 4;
constexpr int NDTAB = 32;  // doubles per CTA: D and D^T in FP32, then D; rows of 4

__host__ __device__ constexpr size_t smem_bytes(int epb) {
  return sizeof(double) * (NDTAB + (size_t)epb * NREF) + sizeof(float2) * (size_t)epb * NSLOT * FSTRIDE;
}

__device__ __forceinline__ float2 F2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 FMA2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 MUL2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 ADD2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// weak divergence of a pair: sum_m D[m][i] fx(m,j,k) + D[m][j] fy(i,m,k) + D[m][k] fz(i,j,m);
// DT: the table of D^T rows
__device__ __forceinline__ float2 divT2(const float2* fx, const float2* fy, const float2* fz, int i, int j, int k,
                                        const float2* DTx, const float2* DTy, const float2* DTz) {
  const float2* ax = fx + 4 * j + PLANE * k;
  const float4 a01 = *reinterpret_cast<const float4*>(ax);
  const float4 a23 = *reinterpret_cast<const float4*>(ax + 2);
  float2 s = MUL2(DTx[0], make_float2(a01.x, a01.y));
  s = FMA2(DTx[1], make_float2(a01.z, a01.w), s);
  s = FMA2(DTx[2], make_float2(a23.x, a23.y), s);
  s = FMA2(DTx[3], make_float2(a23.z, a23.w), s);
  const float2* ay = fy + i + PLANE * k;
  float2 t = MUL2(DTy[0], ay[0]);
  t = FMA2(DTy[1], ay[4], t);
  t = FMA2(DTy[2], ay[8], t);
  t = FMA2(DTy[3], ay[12], t);
  const float2* az = fz + i + 4 * j;
  float2 u = MUL2(DTz[0], az[0]);
  u = FMA2(DTz[1], az[PLANE], u);
  u = FMA2(DTz[2], az[2 * PLANE], u);
  u = FMA2(DTz[3], az[3 * PLANE], u);
  return ADD2(ADD2(s, t), u);
}

// A table row as 4 (v, v) pairs, doubled in registers: doubled rows in shared memory cost 24 more
// wavefronts per element (0.831 against 0.801 ms at 64^3).
__device__ __forceinline__ void load_row(const float* tab, int x, float2* w) {
  const float4 a = *reinterpret_cast<const float4*>(tab + 4 * x);
  w[0] = F2(a.x); w[1] = F2(a.y); w[2] = F2(a.z); w[3] = F2(a.w);
}

// Resident 64-thread element groups per SM the register budget must allow.  Measured at 64^3 (one
// element per CTA): 10 (96 registers) 0.826 ms, 12 (80, 28 bytes of spill) 0.837, 14 (72, 92 bytes)
// 0.908.
#ifndef SOD_MX2_MIN_CTAS
#define SOD_MX2_MIN_CTAS 10
#endif
// One tile of EPB elements (64 threads each); smem_raw holds smem_bytes(EPB).  Every thread of
// the block calls it (it holds block barriers).
// TOTH: flag_total_enthalpy (energy convection of full_convec_ijk_H)
template <int EPB, bool TOTH>
__device__ __forceinline__ void rhs_mixed2_tile(const RhsArgs& a, int tile, unsigned char* smem_raw) {
  float* dtab = reinterpret_cast<float*>(smem_raw);   // D rows, then D^T rows
  double* dtab64 = reinterpret_cast<double*>(smem_raw) + 16;
  double* refs_all = reinterpret_cast<double*>(smem_raw) + NDTAB;
  float2* buf_all = reinterpret_cast<float2*>(refs_all + EPB * NREF);
  const int tid = threadIdx.x;
  const int es = tid >> 6;
  // Lane bits (i0 j0 i1 j1 k): an 8-byte shared load costs one wavefront instead of two when the
  // lanes l, l ^ 1 (or l, l ^ 2) of every pair read the same address.  In this order the xi lines
  // (lanes that differ in i0) and the eta lines (j0) both do; in the natural order only xi does.
  const int lt = tid & 63;
  const int i = (lt & 1) | ((lt >> 1) & 2), j = ((lt >> 1) & 1) | ((lt >> 2) & 2), k = lt >> 4;
  const int d = i + 4 * j + 16 * k;
  const int e = tile * EPB + es;
  const bool active = e < a.nelem;
  const int ee = active ? e : a.nelem - 1;
  double* refs = refs_all + es * NREF;
  float* rf = reinterpret_cast<float*>(refs + R_F32);
  float2* slopes = reinterpret_cast<float2*>(refs + R_F32 + 4);  // of (p, T) along xi, eta, zeta
  float2* buf = buf_all + (size_t)es * NSLOT * FSTRIDE;
  double* ud = reinterpret_cast<double*>(buf + NA * FSTRIDE);
  float2* p2 = buf + (NA + NU) * FSTRIDE;
  const int s_me = sidx(i, j, k);
  const float* geo = reinterpret_cast<const float*>(a.geo) + (size_t)ee * NGEO * NN;

  // ---- own node: stage EOS in FP64 (time_integ.f90:266-285)
  const int32_t n = a.econn[(size_t)ee * NN + d];
  const double g = a.prm.gamma;
  const double rho = a.rho[n];
  const double qv[3] = {a.q0[n], a.q1[n], a.q2[n]};
  const double Et = a.E[n];
  const float mufac = (float)a.mu_factor[n];
  const float mue = reinterpret_cast<const float*>(a.mue)[(size_t)ee * NN + d];
  float H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = geo[c * NN + d];
  const float gpv = geo[9 * NN + d];
  if (tid < 32) {
    const int r = (tid >> 2) & 3, c = tid & 3;
    dtab[tid] = tid < 16 ? a.Df[r][c] : a.Df[c][r];
    if (tid < 16) dtab64[tid] = a.D.d[r][c];
  }
  // one FP64 reciprocal serves every division of the EOS (the deviations below need FP64)
  const double irho = 1.0 / rho;
  const double uv[3] = {qv[0] * irho, qv[1] * irho, qv[2] * irho};
  const double umag = uv[0] * uv[0] + uv[1] * uv[1] + uv[2] * uv[2];
  const double kk = 0.5 * umag;
  const double e_int = Et * irho - 0.5 * umag;
  const double p = rho * (g - 1.0) * e_int;
  const double h = a.prm.g_gm1 * p * irho;
  const double T = p * irho * a.prm.inv_Rgas;

  // element references: FP64 values of local node 0, and their FP32 copies
  if (d == 0) {
    refs[0] = rho; refs[1] = uv[0]; refs[2] = uv[1]; refs[3] = uv[2];
    refs[4] = h; refs[5] = kk;
    rf[0] = (float)rho; rf[1] = (float)uv[0]; rf[2] = (float)uv[1]; rf[3] = (float)uv[2];
    rf[4] = (float)(h + kk); rf[5] = (float)irho;
    rf[6] = 1.0f / (float)p;
  }
  if (d == 0 || d == 3 || d == 12 || d == 48)
    *reinterpret_cast<double2*>(refs + R_P + (d == 0 ? 0 : (d == 3 ? 2 : (d == 12 ? 4 : 6)))) = make_double2(p, T);
#pragma unroll
  for (int c = 0; c < 3; ++c) ud[c * FSTRIDE + s_me] = uv[c];
  __syncthreads();
  // L_r, by two lanes of the second warp while the others go on (read after the next barrier)
  if ((lt & ~1) == 32) refs[R_LOG + (lt & 1)] = log((lt & 1) ? refs[0] : refs[R_P]);
  // deviations from node 0; L - L_r by log1p of small ratios
  const float drho = (float)(rho - refs[0]);
  const double p0 = refs[R_P], T0 = refs[R_P + 1];
  const float dL = log1pf((float)(p - p0) * rf[6]) - a.prm.gamma_f * log1pf(drho * rf[5]);
  float2 v0, v1, v2, v3;   // own slots
  {
    constexpr double kX = 0.44721359549995793928;  // interior GLL nodes of p = 3: +-sqrt(1/5)
    auto xh = [&](int t) {  // (xi_t + 1)/2
      return t == 0 ? 0.0 : (t == 1 ? 0.5 * (1.0 - kX) : (t == 2 ? 0.5 * (1.0 + kX) : 1.0));
    };
    // f = f_0 + sum_d a_d (xi_d + 1) + f' for f = p, T, a_d from the three corner nodes: D differentiates
    // linear functions exactly, so D f = D f' + a
    auto corner = [&](int t) {
      const double2 c = *reinterpret_cast<const double2*>(refs + R_P + 2 * (t + 1));
      return make_double2(c.x - p0, c.y - T0);
    };
    const double2 cx = corner(0), cy = corner(1), cz = corner(2);
    if (d < 3) {
      const double2 c = d == 0 ? cx : (d == 1 ? cy : cz);
      slopes[d] = make_float2(0.5f * (float)c.x, 0.5f * (float)c.y);
    }
    const double wx = xh(i), wy = xh(j), wz = xh(k);
    v0 = make_float2((float)(uv[0] - refs[1]), (float)(uv[1] - refs[2]));
    v1 = make_float2((float)(uv[2] - refs[3]), (float)((h - refs[4]) + (kk - refs[5])));  // total enthalpy H = h + k
    v2 = make_float2(drho, (rf[0] + drho) * dL);
    v3 = make_float2((float)((p - p0) - (cx.x * wx + cy.x * wy + cz.x * wz)),
                     (float)((T - T0) - (cx.y * wx + cy.y * wy + cz.y * wz)));
    buf[0 * FSTRIDE + s_me] = v0;
    buf[1 * FSTRIDE + s_me] = v1;
    buf[2 * FSTRIDE + s_me] = v2;
    buf[3 * FSTRIDE + s_me] = v3;
  }
  // full node values in FP32: reference + deviation
  const float uR[3] = {rf[1] + v0.x, rf[2] + v0.y, rf[3] + v1.x};
  const float HR = rf[4] + v1.y, rhoR = rf[0] + v2.x;
  const float Tf = (float)T;
  const float muf = mufac * (float)kC1 * (Tf * sqrtf(Tf)) / (Tf + (float)kS);
  // LES: rho mu_sgs as an FP64 product, rounded once.  The two coefficients the fluxes need are formed here,
  // while rho is at hand: with rho mu_sgs itself kept across the line pass, or read again after it, total
  // enthalpy at 64^3 took 0.853 and 0.879 ms instead of 0.821.
  const float rmsgs = a.musgs ? (float)(rho * a.musgs[(size_t)ee * NN + d]) : 0.f;
  const float mufgp = muf + rmsgs;
  const float kappa_e = muf * a.prm.CpPr_f + a.prm.c_ener_f * mue * a.prm.CpPr_f + a.prm.Cp09_f * rmsgs;
  __syncthreads();

  // ---- one pass over the line points: gradients, and the residuals' sums
  float2 gU01[3];                    // physical gradients of (u0, u1)
  float gU2[3], gRho[3], gT[3];
  // sum0 = (mom 0, mom 1), sum1 = (mom 2, energy): sum D V^ r^ df (+ grad p); sum2 = (mass, lam):
  // sum D V^ df
  float2 sum0 = F2(0.f), sum1 = F2(0.f), sum2 = F2(0.f);
  double divU64 = 0.0;
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const float hc[3] = {H[dir], H[3 + dir], H[6 + dir]};
    const float hh[3] = {0.5f * hc[0], 0.5f * hc[1], 0.5f * hc[2]};
    const float Vx = fmaf(hc[2], uR[2], fmaf(hc[1], uR[1], hc[0] * uR[0]));
    const float Vh = 0.5f * Vx;
    const int x = dir == 0 ? i : (dir == 1 ? j : k);
    float2 w[4];
    load_row(dtab, x, w);
    float2 g2, g3;
    float2 lu01;  // line sums of u, from FP64
    float lu2;
    auto point = [&](int m, float2 p0, float2 p1, float2 p2_, float2 p3) {
      if (m == 0) {
        g2 = MUL2(w[0], p2_); g3 = MUL2(w[0], p3);
      } else {
        g2 = FMA2(w[m], p2_, g2); g3 = FMA2(w[m], p3, g3);
      }
      // differences to the own point
      const float2 d0 = ADD2(p0, make_float2(-v0.x, -v0.y)), d1 = ADD2(p1, make_float2(-v1.x, -v1.y)),
                   d2 = ADD2(p2_, make_float2(-v2.x, -v2.y));
      // V^ = V_x + hV; s = D (V^ r^ - V_x rho_x) = D (hV r^ + V_x/2 drho), sv = D V^
      const float hV = fmaf(hh[2], d1.x, fmaf(hh[1], d0.y, hh[0] * d0.x));
      const float rh = fmaf(0.5f, d2.x, rhoR);
      const float2 s = F2(w[m].x * fmaf(hV, rh, Vh * d2.x)), sv = F2(w[m].x * (Vx + hV));
      sum0 = FMA2(s, d0, sum0);
      sum2 = FMA2(sv, d2, sum2);
      if constexpr (TOTH) {
        const float dG = fmaf(rhoR + d2.x, d1.y, HR * d2.x);  // rho_m dH + H drho
        sum1.x = fmaf(s.x, d1.x, sum1.x);
        sum1.y = fmaf(sv.x, dG, sum1.y);
      } else {
        sum1.x = fmaf(s.x, d1.x, sum1.x);
        sum1.y = fmaf(sv.x * rh, d1.y, sum1.y);
      }
    };
    const double* fu = ud + (dir == 0 ? sidx(0, j, k) : (dir == 1 ? sidx(i, 0, k) : sidx(i, j, 0)));
    if (dir == 0) {
      const float2* f = buf + sidx(0, j, k);  // the xi line of the node: 16-byte loads
#pragma unroll
      for (int hh_ = 0; hh_ < 2; ++hh_) {
        const float4 q0 = *reinterpret_cast<const float4*>(f + 2 * hh_);
        const float4 q1 = *reinterpret_cast<const float4*>(f + FSTRIDE + 2 * hh_);
        const float4 q2 = *reinterpret_cast<const float4*>(f + 2 * FSTRIDE + 2 * hh_);
        const float4 q3 = *reinterpret_cast<const float4*>(f + 3 * FSTRIDE + 2 * hh_);
        point(2 * hh_, make_float2(q0.x, q0.y), make_float2(q1.x, q1.y), make_float2(q2.x, q2.y),
              make_float2(q3.x, q3.y));
        point(2 * hh_ + 1, make_float2(q0.z, q0.w), make_float2(q1.z, q1.w), make_float2(q2.z, q2.w),
              make_float2(q3.z, q3.w));
      }
      const double2 wa = *reinterpret_cast<const double2*>(dtab64 + 4 * x),
                  wb = *reinterpret_cast<const double2*>(dtab64 + 4 * x + 2);
#pragma unroll
      for (int c = 0; c < 3; ++c, fu += FSTRIDE) {
        const double2 fa = *reinterpret_cast<const double2*>(fu), fb = *reinterpret_cast<const double2*>(fu + 2);
        const double l = (wa.x * fa.x + wa.y * fa.y) + (wb.x * fb.x + wb.y * fb.y);
        divU64 += (double)hc[c] * l;
        (c == 0 ? lu01.x : (c == 1 ? lu01.y : lu2)) = (float)l;
      }
    } else {
      const float2* f = buf + (dir == 1 ? sidx(i, 0, k) : sidx(i, j, 0));
      const int st = dir == 1 ? 4 : PLANE;
#pragma unroll
      for (int m = 0; m < 4; ++m)
        point(m, f[m * st], f[FSTRIDE + m * st], f[2 * FSTRIDE + m * st], f[3 * FSTRIDE + m * st]);
      const double2 wa = *reinterpret_cast<const double2*>(dtab64 + 4 * x),
                  wb = *reinterpret_cast<const double2*>(dtab64 + 4 * x + 2);
#pragma unroll
      for (int c = 0; c < 3; ++c, fu += FSTRIDE) {
        const double l = (wa.x * fu[0] + wa.y * fu[st]) + (wb.x * fu[2 * st] + wb.y * fu[3 * st]);
        divU64 += (double)hc[c] * l;
        (c == 0 ? lu01.x : (c == 1 ? lu01.y : lu2)) = (float)l;
      }
    }
    g3 = ADD2(g3, slopes[dir]);  // the affine parts of p and T
    // momentum: the part of s taken out above, times the whole line sum
    const float Wx = Vx * rhoR;
    sum0 = FMA2(F2(Wx), lu01, sum0);
    sum1.x = fmaf(Wx, lu2, sum1.x);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      if (dir == 0) {
        gU01[r] = MUL2(F2(hc[r]), lu01); gU2[r] = hc[r] * lu2; gRho[r] = hc[r] * g2.x; gT[r] = hc[r] * g3.y;
      } else {
        gU01[r] = FMA2(F2(hc[r]), lu01, gU01[r]); gU2[r] = fmaf(hc[r], lu2, gU2[r]);
        gRho[r] = fmaf(hc[r], g2.x, gRho[r]); gT[r] = fmaf(hc[r], g3.y, gT[r]);
      }
    }
    sum0.x = fmaf(hc[0], g3.x, sum0.x);
    sum0.y = fmaf(hc[1], g3.x, sum0.y);
    sum1.x = fmaf(hc[2], g3.x, sum1.x);
  }
  // ---- convective residuals
  const float divU = (float)divU64;
  const float Rm = fmaf(rhoR, divU, sum2.x);
  const float Lr = (float)(refs[R_LOG] - g * refs[R_LOG + 1]);
  const float Ret = fmaf(Lr, Rm, fmaf(v2.y, divU, sum2.y)) * a.prm.inv_gm1_f;
  const float Rmo[3] = {fmaf(uR[0], Rm, sum0.x), fmaf(uR[1], Rm, sum0.y), fmaf(uR[2], Rm, sum1.x)};
  const float Ren = TOTH ? fmaf(HR * rhoR, divU, sum1.y) : fmaf(HR, Rm, sum1.y);

  // ---- diffusion pass 1 (elem_diffu.f90:70-140) -> contravariant flux pairs per direction
  {
    const float mut = mufgp + mue;
    const float twoThirds = 2.0f / 3.0f;
    const float gradU[3][3] = {{gU01[0].x, gU01[1].x, gU01[2].x}, {gU01[0].y, gU01[1].y, gU01[2].y},
                               {gU2[0], gU2[1], gU2[2]}};
    float tau[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) tau[r][c] = mut * (gradU[r][c] + gradU[c][r]);
#pragma unroll
    for (int r = 0; r < 3; ++r) tau[r][r] = tau[r][r] - mufgp * twoThirds * divU;
    float tauU[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) tauU[r] = tau[r][0] * uR[0] + tau[r][1] * uR[1] + tau[r][2] * uR[2];
    const float2 g2 = F2(gpv);
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      auto emit = [&](int slot0, float2 f0, float2 f1, float2 f2) {
        const float2 v = FMA2(F2(H[6 + dir]), f2, FMA2(F2(H[3 + dir]), f1, MUL2(F2(H[dir]), f0)));
        p2[(slot0 + dir) * FSTRIDE + s_me] = MUL2(g2, v);
      };
      emit(0, make_float2(gRho[0], tauU[0]), make_float2(gRho[1], tauU[1]), make_float2(gRho[2], tauU[2]));
      emit(3, make_float2(gT[0], tau[0][0]), make_float2(gT[1], tau[0][1]), make_float2(gT[2], tau[0][2]));
      emit(6, make_float2(tau[1][0], tau[2][0]), make_float2(tau[1][1], tau[2][1]), make_float2(tau[1][2], tau[2][2]));
    }
  }
  __syncthreads();  // pass-1 fluxes visible

  // ---- diffusion pass 2 (elem_diffu.f90:142-194)
  float2 DTx[4], DTy[4], DTz[4];
  load_row(dtab + 16, i, DTx);
  load_row(dtab + 16, j, DTy);
  load_row(dtab + 16, k, DTz);
  const float2 vA = divT2(p2 + 0 * FSTRIDE, p2 + 1 * FSTRIDE, p2 + 2 * FSTRIDE, i, j, k, DTx, DTy, DTz);
  const float2 vB = divT2(p2 + 3 * FSTRIDE, p2 + 4 * FSTRIDE, p2 + 5 * FSTRIDE, i, j, k, DTx, DTy, DTz);
  const float2 vC = divT2(p2 + 6 * FSTRIDE, p2 + 7 * FSTRIDE, p2 + 8 * FSTRIDE, i, j, k, DTx, DTy, DTz);
  const float nu_e = a.prm.c_rho_f * mue / rhoR;
  if (active) {
    store_res6<float>(reinterpret_cast<float*>(a.rel), (size_t)e * NN + d, gpv * Rm + nu_e * vA.x,
                      gpv * Rmo[0] + vB.y, gpv * Rmo[1] + vC.x, gpv * Rmo[2] + vC.y,
                      gpv * Ren + (vA.y + kappa_e * vB.x), gpv * Ret);
  }
}

template <int EPB, bool TOTH>
__global__ void __launch_bounds__(64 * EPB, (EPB >= SOD_MX2_MIN_CTAS ? 1 : SOD_MX2_MIN_CTAS / EPB))
    k_rhs_mixed2(const RhsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  rhs_mixed2_tile<EPB, TOTH>(a, blockIdx.x, smem_raw);
}

// One RK stage of the mixed path in one cooperative launch (persistent blocks): the fused RHS
// over element tiles, then persist_stage_tail (gather / stage update; at stage 4 the entropy
// viscosity and dt).
template <int EPB, bool TOTH>
__global__ void __launch_bounds__(64 * EPB, (EPB >= SOD_MX2_MIN_CTAS ? 1 : SOD_MX2_MIN_CTAS / EPB))
    k_stage_mixed2(const StageArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ntiles = (p.r.nelem + EPB - 1) / EPB;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    rhs_mixed2_tile<EPB, TOTH>(p.r, t, smem_raw);
    __syncthreads();  // the next tile reuses the shared memory
  }
  persist_stage_tail<float, EPB>(p, smem_raw);
}

template <int EPB>
static int set_attr() {
  SOD_CUDA(cudaFuncSetAttribute(k_rhs_mixed2<EPB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_rhs_mixed2<EPB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_stage_mixed2<EPB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_stage_mixed2<EPB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(EPB)));
  return SOD_OK;
}

// Cooperative launch of one persistent stage; ctas_per_sm <= 0 asks for the most that fit.
template <int EPB>
static int launch_stage(const StageArgs& p, int ctas_per_sm, int* grid_out, cudaStream_t st) {
  const bool toth = p.r.prm.total_enthalpy != 0;
  const void* fn = toth ? (const void*)k_stage_mixed2<EPB, true> : (const void*)k_stage_mixed2<EPB, false>;
  int occ = 0, dev = 0, nsm = 0;
  SOD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 64 * EPB, smem_bytes(EPB)));
  SOD_CUDA(cudaGetDevice(&dev));
  SOD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  if (occ <= 0) {
    set_error("persistent stage kernel: no resident block fits (EPB %d)", EPB);
    return SOD_ERR_UNSUPPORTED;
  }
  const int per = (ctas_per_sm > 0 && ctas_per_sm < occ) ? ctas_per_sm : occ;
  const int ntiles = (p.r.nelem + EPB - 1) / EPB;
  const int grid = std::min(per * nsm, ntiles);
  if (grid_out) *grid_out = grid;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(64 * EPB);
  cfg.dynamicSmemBytes = smem_bytes(EPB);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<StageArgs*>(&p)};
  SOD_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

template <int EPB>
static int launch(const RhsArgs& a, cudaStream_t st) {
  const int grid = (a.nelem + EPB - 1) / EPB;
  if (a.prm.total_enthalpy)
    k_rhs_mixed2<EPB, true><<<grid, 64 * EPB, smem_bytes(EPB), st>>>(a);
  else
    k_rhs_mixed2<EPB, false><<<grid, 64 * EPB, smem_bytes(EPB), st>>>(a);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

}  // namespace mx2

int init_rhs_mixed2_attrs() {
  static bool done = false;
  if (done) return SOD_OK;
  if (mx2::set_attr<1>() || mx2::set_attr<2>() || mx2::set_attr<4>() || mx2::set_attr<8>()) return SOD_ERR_CUDA;
  done = true;
  return SOD_OK;
}

void stage_mixed2_info(int epb, bool toth, const void** fn, size_t* smem) {
  switch (epb) {
    case 1: *fn = toth ? (const void*)mx2::k_stage_mixed2<1, true> : (const void*)mx2::k_stage_mixed2<1, false>; break;
    case 2: *fn = toth ? (const void*)mx2::k_stage_mixed2<2, true> : (const void*)mx2::k_stage_mixed2<2, false>; break;
    case 8: *fn = toth ? (const void*)mx2::k_stage_mixed2<8, true> : (const void*)mx2::k_stage_mixed2<8, false>; break;
    default: *fn = toth ? (const void*)mx2::k_stage_mixed2<4, true> : (const void*)mx2::k_stage_mixed2<4, false>; epb = 4;
  }
  *smem = mx2::smem_bytes(epb);
}

int launch_stage_mixed2(const StageArgs& p, int epb, int ctas_per_sm, int* grid_out, cudaStream_t st) {
  switch (epb) {
    case 1: return mx2::launch_stage<1>(p, ctas_per_sm, grid_out, st);
    case 2: return mx2::launch_stage<2>(p, ctas_per_sm, grid_out, st);
    case 8: return mx2::launch_stage<8>(p, ctas_per_sm, grid_out, st);
    default: return mx2::launch_stage<4>(p, ctas_per_sm, grid_out, st);
  }
}

int launch_rhs_mixed2(const RhsArgs& a, int epb, cudaStream_t st) {
  switch (epb) {
    case 1: return mx2::launch<1>(a, st);
    case 2: return mx2::launch<2>(a, st);
    case 8: return mx2::launch<8>(a, st);
    default: return mx2::launch<4>(a, st);
  }
}

}  // namespace sod

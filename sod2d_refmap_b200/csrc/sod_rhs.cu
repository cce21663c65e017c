// Fused element RHS (KR), deterministic node gather fused with the lumped-mass solve and the
// RK4 stage update (KG), entropy viscosity + CFL dt (KV), and the RK4 step driver (sm_100a).
//
// KR restates, for one CTA-resident tile of EPB elements, the element loops of
//   full_convec_ijk            elem_convec.f90:211-460   (skew-symmetric split convection)
//   full_diffusion_ijk         elem_diffu.f90:12-198     (viscous + heat + artificial mass)
//   generic_scalar_convec_ijk  elem_convec.f90:462-570   (entropy residual)
//   sutherland_viscosity       mod_fluid_viscosity.f90:21-41
//   the stage EOS of rk_4_main time_integ.f90:266-285
// One thread owns one gauss point (= element node, GLL collocation).  Eight nodal fields are
// staged in shared memory; one pass over the 12 line points of each node forms the gradients the
// diffusion needs and the split-form convection; the weak divergence of the diffusive fluxes is
// applied as D^T to contravariant fluxes precomputed at each gauss point.  Element residuals are
// written to an element-major array and assembled by KG as an ordered CSR gather (no atomics).
//
// Convection: the quartets of elem_convec.f90:412-432 are two-point flux sums.  With D the line
// derivative (sum_m D[x][m] = 0), V(m) = sum_c He(c,dir)(x) u_c(m) the contravariant velocity with
// the output point's metric, V^ = (V_x + V_m)/2, r^ = (rho_x + rho_m)/2 and df = f_m - f_x,
//   mass      Rm = rho div u + sum_dir sum_m D[x][m] V^ drho
//   f         f_x Rm + sum_dir sum_m D[x][m] V^ r^ df        f = u_c, H = h + k
//   entropy   eta div u + sum_dir sum_m D[x][m] V^ deta
//   (E+p)     G div u + sum_dir sum_m D[x][m] V^ dG          G = E + p, flag_total_enthalpy
// (the energy is linear in (h, k) and every h term has a k twin, so both quartets are evaluated on
// H).  These are the reference's sums with the products expanded around the output point, where
// the constant parts vanish but for the row sums of D (its rounding), which are counted: 19 FP64 operations
// per line point instead of ~36, and none of the derivatives of q, H, rho H, eta and their products.
// u and rho enter the line sums as differences too, and u = q / rho is rounded once, since div u differentiates
// that rounding.  Against extended precision, vortex at 8^3: mass 8.0e-15, energy 2.3e-14, entropy 2.0e-14;
// quartets one by one 8.5e-15, 2.8e-14, 2.1e-14; with whole values of u in the sums, q * (1 / rho) and no
// row sums 1.6e-14, 3.3e-14, 2.5e-14 (and 0.993 ms in what follows).
// Measured at 64^3, one launch: 1.03 ms, 1.84 ms with the quartets one by one; bounded by latency at 16
// resident warps with the FP64 pipe and the shared-memory pipe about equally loaded (~700 cycles each per element).
//
// This is the FP64 parity path.  The mixed path (FP32 element arithmetic on deviation fields) is
// k_rhs_mixed2 in sod_rhs_mixed.cu.
#include "sod_internal.cuh"
#include "sod_step_kernels.cuh"
#include <cmath>
#include <algorithm>

namespace sod {

// weak divergence sum_dir sum_m D[m][idx_dir] V_dir(line point m)
__device__ __forceinline__ double divT(const double* fx, const double* fy, const double* fz, int i, int j, int k, const double* DTx,
                                  const double* DTy, const double* DTz) {
  const double* ax = fx + 4 * j + PLANE * k;
  const double* ay = fy + i + PLANE * k;
  const double* az = fz + i + 4 * j;
  return DTx[0] * ax[0] + DTx[1] * ax[1] + DTx[2] * ax[2] + DTx[3] * ax[3] +
         (DTy[0] * ay[0] + DTy[1] * ay[4] + DTy[2] * ay[8] + DTy[3] * ay[12]) +
         (DTz[0] * az[0] + DTz[1] * az[PLANE] + DTz[2] * az[2 * PLANE] + DTz[3] * az[3 * PLANE]);
}

constexpr int NBUF = 8;  // rho, u0, u1, u2, H (TOTH: G), eta, p, T
constexpr int NP2 = 18;  // 6 contravariant fluxes x 3 directions
constexpr int NDTAB = 36;  // per CTA: D rows, then D^T rows, then D's row sums

constexpr size_t rhs_smem_bytes(int epb) {
  return sizeof(double) * (NDTAB + (size_t)epb * (NBUF + NP2) * FSTRIDE);
}

// One tile of EPB elements (64 threads each) of the fused RHS; smem_raw holds
// rhs_smem_bytes(EPB).  Every thread of the block calls it (it holds block barriers).
// TOTH: flag_total_enthalpy (energy convection of full_convec_ijk_H)
template <int EPB, bool TOTH>
__device__ __forceinline__ void rhs_fused_tile(const RhsArgs& a, int tile, unsigned char* smem_raw) {
  double* dtab = reinterpret_cast<double*>(smem_raw);
  const int tid = threadIdx.x;
  const int es = tid >> 6;
  // lane bits (i0 j0 i1 j1 k): the xi and the eta line loads of a warp then cost one shared-memory
  // wavefront per 8-byte load instead of two (pairs of lanes l, l ^ 1 or l, l ^ 2 share addresses)
  const int lt = tid & 63;
  const int i = (lt & 1) | ((lt >> 1) & 2), j = ((lt >> 1) & 1) | ((lt >> 2) & 2), k = lt >> 4;
  const int d = i + 4 * j + 16 * k;
  const int e = tile * EPB + es;
  const bool active = e < a.nelem;
  const int ee = active ? e : a.nelem - 1;
  double* buf = dtab + NDTAB + (size_t)es * (NBUF + NP2) * FSTRIDE;
  double* p2 = buf + NBUF * FSTRIDE;
  const int s_me = sidx(i, j, k);
  const double* geo = reinterpret_cast<const double*>(a.geo) + (size_t)ee * NGEO * NN;

  // ---- own node: stage EOS (time_integ.f90:266-285) and Sutherland (mod_fluid_viscosity.f90:37)
  const int32_t n = a.econn[(size_t)ee * NN + d];
  const double g = a.prm.gamma;
  const double rho = a.rho[n];
  const double qv[3] = {a.q0[n], a.q1[n], a.q2[n]};
  const double Et = a.E[n];
  const double mufac = a.mu_factor[n];
  double H[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) H[c] = geo[c * NN + d];
  const double gpv = geo[9 * NN + d];
  const double mue = reinterpret_cast<const double*>(a.mue)[(size_t)ee * NN + d];
  const double musgs = a.musgs ? a.musgs[(size_t)ee * NN + d] : 0.0;
  if (tid < 32) {
    const int r = (tid >> 2) & 3, c = tid & 3;
    dtab[tid] = tid < 16 ? a.D.d[r][c] : a.D.d[c][r];
    if (tid < NP1) dtab[32 + tid] = a.Dsum[tid];
  }
  const double* dsum = dtab + 32;
  // one reciprocal serves the divisions by rho; gamma/(gamma-1) and 1/Rgas come from the host
  const double irho = 1.0 / rho;
  double uv[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double t = qv[c] * irho;
    uv[c] = t + (qv[c] - t * rho) * irho;  // rounded once: the rounding of u is differentiated in div u
  }
  const double umag = uv[0] * uv[0] + uv[1] * uv[1] + uv[2] * uv[2];
  const double kk = 0.5 * umag;
  const double e_int = Et * irho - 0.5 * umag;
  const double p = rho * (g - 1.0) * e_int;
  const double Ht = TOTH ? Et + p : a.prm.g_gm1 * p * irho + kk;  // H = h + k (TOTH: G)
  const double T = p * irho * a.prm.inv_Rgas;
  // log(p / rho^gamma) as log p - gamma log rho (no pow)
  const double eta = (rho / (g - 1.0)) * (log(p) - g * log(rho));
  buf[0 * FSTRIDE + s_me] = rho;
#pragma unroll
  for (int c = 0; c < 3; ++c) buf[(1 + c) * FSTRIDE + s_me] = uv[c];
  buf[4 * FSTRIDE + s_me] = Ht;
  buf[5 * FSTRIDE + s_me] = eta;
  buf[6 * FSTRIDE + s_me] = p;
  buf[7 * FSTRIDE + s_me] = T;
  const double muf = mufac * kSuthC1 * (T * sqrt(T)) / (T + kSuthS);
  __syncthreads();

  // ---- one pass over the line points
  double gradRho[3], gradU[3][3], gradT[3];
  double Sm = 0.0, Se = 0.0, Sn = 0.0;  // sum D V^ drho; D V^ r^ dH (TOTH: D V^ dG); D V^ deta
  double Su[3] = {0.0, 0.0, 0.0};       // sum D V^ r^ du_c, + grad p below
  double sV = 0.0;                      // D's row sums times V_x
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const double hc[3] = {H[dir], H[3 + dir], H[6 + dir]};
    const double hh[3] = {0.5 * hc[0], 0.5 * hc[1], 0.5 * hc[2]};
    const double Vx = hc[0] * uv[0] + hc[1] * uv[1] + hc[2] * uv[2];
    const int x = dir == 0 ? i : (dir == 1 ? j : k);
    double w[4];
    {
      const double2 wa = *reinterpret_cast<const double2*>(dtab + 4 * x),
                    wb = *reinterpret_cast<const double2*>(dtab + 4 * x + 2);
      w[0] = wa.x; w[1] = wa.y; w[2] = wb.x; w[3] = wb.y;
    }
    const double* f = buf + (dir == 0 ? sidx(0, j, k) : (dir == 1 ? sidx(i, 0, k) : sidx(i, j, 0)));
    constexpr int stride[3] = {1, 4, PLANE};
    double gr = 0.0, gu[3] = {0.0, 0.0, 0.0}, gp = 0.0, gT = 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const double* fm = f + m * stride[dir];
      const double r_ = fm[0];
      const double du[3] = {fm[FSTRIDE] - uv[0], fm[2 * FSTRIDE] - uv[1], fm[3 * FSTRIDE] - uv[2]};
      const double H_ = fm[4 * FSTRIDE], n_ = fm[5 * FSTRIDE];
      gp += w[m] * fm[6 * FSTRIDE];
      gT += w[m] * fm[7 * FSTRIDE];
      const double dr = r_ - rho;
      gr += w[m] * dr;
#pragma unroll
      for (int c = 0; c < 3; ++c) gu[c] += w[m] * du[c];
      const double wV = w[m] * (Vx + (hh[0] * du[0] + hh[1] * du[1] + hh[2] * du[2]));  // D V^
      const double sr = wV * (rho + 0.5 * dr);
      Sm += wV * dr;
      Sn += wV * (n_ - eta);
      if constexpr (TOTH)
        Se += wV * (H_ - Ht);
      else
        Se += sr * (H_ - Ht);
#pragma unroll
      for (int c = 0; c < 3; ++c) Su[c] += sr * du[c];
    }
    sV += Vx * dsum[x];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      if (dir == 0) {
        gradRho[r] = hc[r] * gr;
        gradT[r] = hc[r] * gT;
#pragma unroll
        for (int c = 0; c < 3; ++c) gradU[c][r] = hc[r] * gu[c];
      } else {
        gradRho[r] += hc[r] * gr;
        gradT[r] += hc[r] * gT;
#pragma unroll
        for (int c = 0; c < 3; ++c) gradU[c][r] += hc[r] * gu[c];
      }
      Su[r] += hc[r] * gp;
    }
  }
  // The row sums of D are its rounding: the reference's quartets hold 1.5, 1.5 and 1.75 times sV of the
  // constant parts that the differences leave out (the diffusion's gradients none that counts).
  const double divU = gradU[0][0] + gradU[1][1] + gradU[2][2];
  const double divS = divU + 1.5 * sV;
  const double Rm = rho * divS + Sm;
  const double Rn = eta * divS + Sn;
  const double Rc = Rm + 0.25 * rho * sV;
  const double Re = TOTH ? Ht * divS + Se : Ht * Rc + Se;
  double Rmo[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) Rmo[c] = uv[c] * Rc + Su[c];

  // ---- diffusion pass 1 (elem_diffu.f90:70-140): stresses and contravariant fluxes
  {
    const double mufgp = muf + rho * musgs;
    const double mut = mufgp + mue;
    const double twoThirds = 2.0 / 3.0;
    double tau[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) tau[r][c] = mut * (gradU[r][c] + gradU[c][r]);
#pragma unroll
    for (int r = 0; r < 3; ++r) tau[r][r] = tau[r][r] - mufgp * twoThirds * divU;
    double tauU[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) tauU[r] = tau[r][0] * uv[0] + tau[r][1] * uv[1] + tau[r][2] * uv[2];
    // V-hat_dir = gpvol * sum_r He(r,dir) V_r for V in {gradRho, tauU, gradT, tau row 0,1,2}
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      const double h0 = gpv * H[dir], h1 = gpv * H[3 + dir], h2 = gpv * H[6 + dir];
      auto emit = [&](int v, double V0, double V1, double V2) {
        p2[(v * 3 + dir) * FSTRIDE + s_me] = h0 * V0 + h1 * V1 + h2 * V2;
      };
      emit(0, gradRho[0], gradRho[1], gradRho[2]);
      emit(1, tauU[0], tauU[1], tauU[2]);
      emit(2, gradT[0], gradT[1], gradT[2]);
      emit(3, tau[0][0], tau[0][1], tau[0][2]);
      emit(4, tau[1][0], tau[1][1], tau[1][2]);
      emit(5, tau[2][0], tau[2][1], tau[2][2]);
    }
  }
  __syncthreads();  // pass-1 fluxes visible

  // ---- diffusion pass 2 (elem_diffu.f90:142-194): weak divergence with D^T
  double DTx[4], DTy[4], DTz[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    DTx[m] = dtab[16 + 4 * i + m];
    DTy[m] = dtab[16 + 4 * j + m];
    DTz[m] = dtab[16 + 4 * k + m];
  }
  double dv[6];
#pragma unroll
  for (int v = 0; v < 6; ++v)
    dv[v] = divT(p2 + (v * 3 + 0) * FSTRIDE, p2 + (v * 3 + 1) * FSTRIDE, p2 + (v * 3 + 2) * FSTRIDE, i, j, k, DTx,
                 DTy, DTz);
  const double nu_e = a.prm.c_rho * mue * irho;
  const double kappa_e = muf * a.prm.CpPr + a.prm.c_ener * mue * a.prm.CpPr + a.prm.Cp09 * rho * musgs;
  if (active) {
    store_res6<double>(reinterpret_cast<double*>(a.rel), (size_t)e * NN + d, gpv * Rm + nu_e * dv[0],
                       gpv * Rmo[0] + dv[3], gpv * Rmo[1] + dv[4], gpv * Rmo[2] + dv[5],
                       gpv * Re + (dv[1] + kappa_e * dv[2]), gpv * Rn);
  }
}

// Resident 64-thread element groups per SM the register budget must allow: 8 (128 registers, no
// spill).  Measured at 64^3 with whole values of u: 8 0.986 ms, 6 (154 registers) 1.087 ms;
// 10 (96 registers) would have spilled 244 bytes.
#ifndef SOD_KR64_MIN_CTAS
#define SOD_KR64_MIN_CTAS 8
#endif
template <int EPB, bool TOTH>
__global__ void __launch_bounds__(64 * EPB, (EPB >= SOD_KR64_MIN_CTAS ? 1 : SOD_KR64_MIN_CTAS / EPB)) k_rhs_fused(const RhsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  rhs_fused_tile<EPB, TOTH>(a, blockIdx.x, smem_raw);
}

// One RK stage of the FP64 path in one cooperative launch (persistent blocks): the fused RHS
// over element tiles, then persist_stage_tail (gather / stage update; at stage 4 the entropy
// viscosity and dt).
template <int EPB, bool TOTH>
__global__ void __launch_bounds__(64 * EPB) k_stage_fused(const StageArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ntiles = (p.r.nelem + EPB - 1) / EPB;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    rhs_fused_tile<EPB, TOTH>(p.r, t, smem_raw);
    __syncthreads();  // the next tile reuses the shared memory
  }
  persist_stage_tail<double, EPB>(p, smem_raw);
}

// resident 256-thread blocks per SM the register budget must allow.  FP32 residual rows (mixed
// path): 4 blocks, 64 registers, no spill with the predicated groups of 4, 2% faster than full
// groups at 5 blocks (the predicated groups at 5 blocks spilled 76 bytes and ran 4% slower
// than that).  FP64 rows: bounded for 3 blocks the kernel takes 56-64 registers without spill, so 4
// still fit; bounded for 4 it spills 16 bytes, for 5 (48 registers) 76
#ifndef SOD_KG_MIN_BLOCKS
#define SOD_KG_MIN_BLOCKS 4
#endif
#ifndef SOD_KG_MIN_BLOCKS_F64
#define SOD_KG_MIN_BLOCKS_F64 3
#endif
template <typename R, int STAGE>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? SOD_KG_MIN_BLOCKS : SOD_KG_MIN_BLOCKS_F64) k_gather_rk(const GatherArgs a) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (STAGE == 4) {
    // the entropy viscosity that follows reduces the next time step into these (1.4e306 each)
    if (n < a.ndt) a.dt_bits[n] = __longlong_as_double(0x7f7f7f7f7f7f7f7fll);
  }
  double eta_n = 0.0;
  const bool act = gather_rk_node<R, STAGE>(a, n, eta_n);
  if constexpr (STAGE == 4) {
    if (a.member_reduce) return;  // uniform across the grid
    __shared__ double sh[3 * 8];
    gather_eta_reduce(a, act ? eta_n : 0.0, act ? eta_n : -1e300, act ? eta_n : 1e300, sh);
  }
}

#ifndef SOD_KV_MIN_BLOCKS
#define SOD_KV_MIN_BLOCKS 3  // resident 256-thread blocks per SM: 80 registers, no spill (4 blocks: 64 registers with spills, the same time)
#endif
__global__ void __launch_bounds__(32 * KV_WARPS, SOD_KV_MIN_BLOCKS) k_visc_dt(const ViscArgs a) {
  __shared__ double sm[KV_WARPS][KV_WSMEM];
  __shared__ unsigned long long lim[KV_WARPS];
  const int wb = threadIdx.x >> 5, e = blockIdx.x * KV_WARPS + wb;
  // one mesh: one dt atomic per block on the minimum of its elements' limits, instead of one per
  // element on the same address; an ensemble's elements take their member's slot each
  const bool per_elem = a.elem_member != nullptr;
  unsigned long long b = ~0ull;
  if (e < a.nelem) b = visc_dt_warp(a, e, threadIdx.x & 31, sm[wb], per_elem);
  if (!per_elem && a.dt_out) {
    if ((threadIdx.x & 31) == 0) lim[wb] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 1; q < KV_WARPS; ++q) b = min(b, lim[q]);
      if (b != ~0ull) atomicMin(reinterpret_cast<unsigned long long*>(a.dt_bits), b);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Host-side launch helpers
// ---------------------------------------------------------------------------------------------
template <int EPB>
static int set_rhs_attr() {
  SOD_CUDA(cudaFuncSetAttribute(k_rhs_fused<EPB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)rhs_smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_rhs_fused<EPB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)rhs_smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_stage_fused<EPB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)rhs_smem_bytes(EPB)));
  SOD_CUDA(cudaFuncSetAttribute(k_stage_fused<EPB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)rhs_smem_bytes(EPB)));
  return SOD_OK;
}

// Cooperative launch of one persistent FP64 stage; ctas_per_sm <= 0 asks for the most that fit.
template <int EPB>
static int launch_stage_fused_t(const StageArgs& p, int ctas_per_sm, int* grid_out, cudaStream_t st) {
  const bool toth = p.r.prm.total_enthalpy != 0;
  const void* fn = toth ? (const void*)k_stage_fused<EPB, true> : (const void*)k_stage_fused<EPB, false>;
  const size_t smem = rhs_smem_bytes(EPB);
  int occ = 0, dev = 0, nsm = 0;
  SOD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 64 * EPB, smem));
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
  cfg.dynamicSmemBytes = smem;
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

int launch_stage_mixed2(const StageArgs& p, int epb, int ctas_per_sm, int* grid_out, cudaStream_t st);
void stage_mixed2_info(int epb, bool toth, const void** fn, size_t* smem);

// the persistent stage kernel of a configuration and its dynamic shared memory
void persist_kernel_info(bool mixed, int epb, bool toth, const void** fn, size_t* smem) {
  if (mixed) {
    stage_mixed2_info(epb, toth, fn, smem);
    return;
  }
  switch (epb) {
    case 1: *fn = toth ? (const void*)k_stage_fused<1, true> : (const void*)k_stage_fused<1, false>; break;
    case 4: *fn = toth ? (const void*)k_stage_fused<4, true> : (const void*)k_stage_fused<4, false>; break;
    case 8: *fn = toth ? (const void*)k_stage_fused<8, true> : (const void*)k_stage_fused<8, false>; break;
    default: *fn = toth ? (const void*)k_stage_fused<2, true> : (const void*)k_stage_fused<2, false>; epb = 2;
  }
  *smem = rhs_smem_bytes(epb);
}

// One persistent stage launch of either precision
int launch_stage(const StageArgs& p, bool mixed, int epb, int ctas_per_sm, int* grid_out, cudaStream_t st) {
  if (mixed) return launch_stage_mixed2(p, epb, ctas_per_sm, grid_out, st);
  switch (epb) {
    case 1: return launch_stage_fused_t<1>(p, ctas_per_sm, grid_out, st);
    case 4: return launch_stage_fused_t<4>(p, ctas_per_sm, grid_out, st);
    case 8: return launch_stage_fused_t<8>(p, ctas_per_sm, grid_out, st);
    default: return launch_stage_fused_t<2>(p, ctas_per_sm, grid_out, st);
  }
}

int init_kernel_attrs() {
  static bool done = false;
  if (done) return SOD_OK;
  int rc = set_rhs_attr<1>() | set_rhs_attr<2>() | set_rhs_attr<4>() |
           set_rhs_attr<8>() |
           init_rhs_mixed2_attrs();
  if (rc) return SOD_ERR_CUDA;
  done = true;
  return SOD_OK;
}

template <int EPB>
static int launch_rhs_t(const RhsArgs& a, cudaStream_t st) {
  const size_t smem = rhs_smem_bytes(EPB);
  const int grid = (a.nelem + EPB - 1) / EPB;
  if (a.prm.total_enthalpy)
    k_rhs_fused<EPB, true><<<grid, 64 * EPB, smem, st>>>(a);
  else
    k_rhs_fused<EPB, false><<<grid, 64 * EPB, smem, st>>>(a);
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

static RhsArgs make_rhs_args(SodMesh* m, bool mixed, const double* rho, const double* q0, const double* q1,
                             const double* q2, const double* E, const double* mu_factor, const double* musgs_int) {
  RhsArgs a;
  a.nelem = m->nelem;
  a.econn = m->econn;
  a.geo = mixed ? (const void*)m->geo32 : (const void*)m->geo64;
  a.mue = mixed ? (const void*)m->mue32 : (const void*)m->mue_int;
  a.musgs = musgs_int;
  a.rho = rho; a.q0 = q0; a.q1 = q1; a.q2 = q2; a.E = E;
  a.mu_factor = mu_factor;
  a.rel = m->buf.rel;
  a.D = m->D;
  for (int r = 0; r < NP1; ++r) {
    if (!mixed) a.Dsum[r] = m->Dsum[r];
    else
      for (int c = 0; c < NP1; ++c) a.Df[r][c] = (float)m->D.d[r][c];
  }
  a.prm = m->prm;
  return a;
}

int launch_rhs(SodMesh* m, bool mixed, int epb, const double* rho, const double* q0, const double* q1,
               const double* q2, const double* E, const double* mu_factor, const double* musgs_int,
               cudaStream_t st) {
  const RhsArgs a = make_rhs_args(m, mixed, rho, q0, q1, q2, E, mu_factor, musgs_int);
  if (!mixed) {
    switch (epb) {
      case 1: return launch_rhs_t<1>(a, st);
      case 4: return launch_rhs_t<4>(a, st);
      case 8: return launch_rhs_t<8>(a, st);
      default: return launch_rhs_t<2>(a, st);
    }
  } else {
    return launch_rhs_mixed2(a, epb, st);
  }
}

static const double kA[4] = {0.0, 0.5, 0.5, 1.0};
static const double kB[4] = {1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0};

template <typename R>
static int launch_gather_t(int stage, const GatherArgs& a, cudaStream_t st) {
  const int grid = (a.npoin + 255) / 256;
  switch (stage) {
    case 0: k_gather_rk<R, 0><<<grid, 256, 0, st>>>(a); break;
    case 1: k_gather_rk<R, 1><<<grid, 256, 0, st>>>(a); break;
    case 2: k_gather_rk<R, 2><<<grid, 256, 0, st>>>(a); break;
    case 3: k_gather_rk<R, 3><<<grid, 256, 0, st>>>(a); break;
    default: k_gather_rk<R, 4><<<grid, 256, 0, st>>>(a); break;
  }
  SOD_CHECK_LAUNCH();
  return SOD_OK;
}

static void fill_gather_args(SodMesh* m, int stage, GatherArgs& a) {
  a.npoin = m->npoin;
  a.nwork = m->npoin_w;
  a.slaves = m->has_slaves ? 1 : 0;
  a.ptr = m->n2e_ptr;
  a.idx = m->n2e;
  a.rel = m->buf.rel;
  a.Ml = m->Ml;
  a.iml = m->buf.iml;
  a.gamma = m->prm.gamma;
  a.inv_Rgas = m->prm.inv_Rgas;
  a.inv_gm1 = m->prm.inv_gm1;
  a.normalise = m->prm.normalise;
  if (!a.ys) a.ys = m->buf.ys;
  a.rsum = m->buf.rsum;
  a.red = m->buf.red;
  a.counter = m->buf.counters + 0;
  a.nonfinite = m->buf.counters + kNonfiniteCounter;
  a.scal = m->buf.scal;
  a.src = m->nmember > 0 ? nullptr : m->source;
  a.wm = (m->nmember > 0 || m->wmodel.nw == 0) ? nullptr : m->wmodel.contrib;
  a.dt_bits = m->nmember > 0 ? m->member_dt_bits : m->buf.scal + 3;
  a.ndt = m->nmember > 0 ? m->nmember : 1;
  if (stage >= 1) {
    a.b_cur = kB[stage - 1];
    a.a_next = stage < 4 ? kA[stage] : 0.0;
  }
}

// The entropy normalisation from the stage-4 gather's block sums, in a fixed order.
__global__ void __launch_bounds__(1024) k_eta_combine(int nblk, int nwork, int normalise, const double* __restrict__ red,
                                                      double* __restrict__ scal) {
  __shared__ double sh[3 * 32];
  double s = 0.0, mx = -1e300, mn = 1e300;
#pragma unroll 4
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    s += red[3 * b];
    mx = fmax(mx, red[3 * b + 1]);
    mn = fmin(mn, red[3 * b + 2]);
  }
  block_reduce3(s, mx, mn, sh);
  if (threadIdx.x == 0) {
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

// Stage 4 forms the entropy normalisation too.  While its blocks are all resident at once (one wave:
// kGatherResident per SM), the last of them does it; beyond, every block would hold its SM slot for the fence and the
// atomic (~1 us of a ~4 us block), so the block sums go to a launch of their own: 64^3, 27,648 blocks,
// 458 -> 368 us mixed for 17 us more.
constexpr int kGatherResident = 4;
int launch_gather(SodMesh* m, bool mixed, int stage, GatherArgs& a, cudaStream_t st) {
  fill_gather_args(m, stage, a);
  const int nblk = (a.npoin + 255) / 256;
  const bool apart = stage == 4 && !a.member_reduce && nblk > kGatherResident * m->nsm;
  if (apart) a.counter = nullptr;
  if (int rc = mixed ? launch_gather_t<float>(stage, a, st) : launch_gather_t<double>(stage, a, st)) return rc;
  if (apart) {
    k_eta_combine<<<1, 1024, 0, st>>>(nblk, a.nwork, a.normalise, a.red, a.scal);
    SOD_CHECK_LAUNCH();
  }
  return SOD_OK;
}

// LES is on for a step when the parameters ask for it and the state carries mu_sgs
static bool les_active(const SodMesh* m, const SodState* s) {
  return m->prm.flag_les == 1 && s->mu_sgs != nullptr && m->musgs_int != nullptr;
}

// mu_sgs (nelem,64) in the reference layout -> internal layout before a step (allocates once)
int les_in(SodMesh* m, const SodState* s, cudaStream_t st) {
  if (!(m->prm.flag_les == 1 && s->mu_sgs)) return SOD_OK;
  if (!m->musgs_int) SOD_CUDA(cudaMalloc(&m->musgs_int, sizeof(double) * (size_t)m->nelem * NN));
  return mesh_ref_to_internal_elem(m, s->mu_sgs, m->musgs_int, st);
}

int les_out(SodMesh* m, const SodState* s, cudaStream_t st) {
  if (!les_active(m, s)) return SOD_OK;
  return mesh_internal_to_ref_elem(m, m->musgs_int, s->mu_sgs, st);
}

static ViscArgs make_visc_args(SodMesh* m, const SodState* s, double* dt_out, float* mue32) {
  ViscArgs v;
  v.nelem = m->nelem;
  v.econn = m->econn;
  v.Reta = s->Reta;
  v.rho = s->rho;
  v.u0 = s->u;
  v.u1 = s->u + m->npoin;
  v.u2 = s->u + 2 * (size_t)m->npoin;
  v.csound = s->csound;
  v.Tem = s->Tem;
  v.mu_fluid = s->mu_fluid;
  v.musgs = les_active(m, s) ? m->musgs_int : nullptr;
  v.helem_l = m->helem_l;
  v.helem = m->helem;
  v.jratio = m->jratio;
  v.scal = m->buf.scal;
  v.mue = m->mue_int;
  v.mue32 = mue32;
  v.dt_bits = m->nmember > 0 ? m->member_dt_bits : m->buf.scal + 3;
  v.elem_member = m->nmember > 0 ? m->elem_member : nullptr;
  v.member_scal = m->member_scal;
  v.dt_out = dt_out;
  v.prm = m->prm;
  return v;
}

// bits_set: the stage-4 gather before it has preset dt_bits
int launch_visc_dt(SodMesh* m, const SodState* s, double* dt_out, float* mue32, cudaStream_t st, bool bits_set) {
  const ViscArgs v = make_visc_args(m, s, dt_out, mue32);
  const int nm = m->nmember > 0 ? m->nmember : 1;
  if (dt_out && !bits_set) SOD_CUDA(cudaMemsetAsync(v.dt_bits, 0x7F, sizeof(double) * nm, st));  // 1.38e306 each
  const int grid = (m->nelem + KV_WARPS - 1) / KV_WARPS;
  k_visc_dt<<<grid, 32 * KV_WARPS, 0, st>>>(v);
  SOD_CHECK_LAUNCH();
  if (dt_out) SOD_CUDA(cudaMemcpyAsync(dt_out, v.dt_bits, sizeof(double) * nm, cudaMemcpyDeviceToDevice, st));
  return SOD_OK;
}

// Ensemble: per-member eta sum/max/min over its contiguous node range, kEtaChunks blocks per
// member; the last of them to finish combines the partials in chunk order (deterministic).  Bounded
// by the latency of its loads: 8 members of up to 24^3 elements 204 -> 13 us against one block per
// member, whose 512 threads walked 373,000 nodes while most SMs had no block.
__global__ void __launch_bounds__(256) k_member_eta(const int32_t* __restrict__ off, const double* __restrict__ eta,
                                                    double* scal, int normalise, double* __restrict__ red,
                                                    unsigned int* __restrict__ done) {
  const int mbr = blockIdx.x / kEtaChunks, ch = blockIdx.x % kEtaChunks;
  const int b = off[mbr], e = off[mbr + 1];
  double s = 0.0, mx = -1e300, mn = 1e300;
#pragma unroll 4
  for (int64_t t = (int64_t)b + ch * 256 + threadIdx.x; t < e; t += kEtaChunks * 256) {
    const double v = eta[t];
    s += v; mx = fmax(mx, v); mn = fmin(mn, v);
  }
  __shared__ double sh[3 * 8];
  block_reduce3(s, mx, mn, sh);
  if (threadIdx.x != 0) return;
  double* r = red + (size_t)mbr * 3 * kEtaChunks;
  r[3 * ch] = s;
  r[3 * ch + 1] = mx;
  r[3 * ch + 2] = mn;
  __threadfence();
  if (atomicAdd(done + mbr, 1u) != kEtaChunks - 1) return;
  __threadfence();
  s = 0.0; mx = -1e300; mn = 1e300;
  for (int c = 0; c < kEtaChunks; ++c) {
    s += __ldcg(r + 3 * c);
    mx = fmax(mx, __ldcg(r + 3 * c + 1));
    mn = fmin(mn, __ldcg(r + 3 * c + 2));
  }
  if (normalise) {
    const double mean = s / (double)(e - b);
    scal[2 * mbr] = mean;
    scal[2 * mbr + 1] = fmax(mx - mean, mean - mn);
  } else {
    scal[2 * mbr] = 0.0;
    scal[2 * mbr + 1] = 1.0;
  }
  done[mbr] = 0u;
}

// the first stage state of a step with boundaries or a buffer zone: (rho, q, E) as [5][N]
__global__ void __launch_bounds__(256) k_copy_state(int64_t N, const double* __restrict__ rho,
                                                    const double* __restrict__ q, const double* __restrict__ E,
                                                    double* __restrict__ y) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  y[n] = rho[n];
#pragma unroll
  for (int c = 0; c < 3; ++c) y[(1 + c) * N + n] = q[c * N + n];
  y[4 * N + n] = E[n];
}

// Reta scratch when the caller passes none
static double* reta_scratch(SodMesh* m) {
  // the FP64 rsum eta column, dead after stage 4 reads it (the mixed path's FP32 accumulators
  // end before it)
  return m->buf.rsum + 5 * (size_t)m->npoin;
}

// The periodic step (no boundaries, buffer zone, wall model, source term or LES) as four
// cooperative launches, one per RK stage: fused RHS, grid barrier, gather / stage update; the
// last one also forms the entropy viscosity and the next dt.  Same arithmetic per element and
// per node as the two-launch path; the entropy sums are blocked by the persistent grid instead,
// so the normalisation can differ from that path's in the last bits.
static int run_step_persist(SodMesh* m, SodState* s, SodState& loc, const double* dt_dev, double* dt_next,
                            bool mixed, int epb, int ctas_per_sm, cudaStream_t st) {
  NvtxRange range(mixed ? "sod rk4 step persistent (mixed)" : "sod rk4 step persistent (fp64)");
  const size_t N = m->npoin;
  StageArgs p{};
  p.g.dt = dt_dev;
  p.g.y[0] = s->rho; p.g.y[1] = s->q; p.g.y[2] = s->q + N; p.g.y[3] = s->q + 2 * N; p.g.y[4] = s->E;
  p.g.u0 = s->u; p.g.u1 = s->u + N; p.g.u2 = s->u + 2 * N;
  p.g.pr = s->pr; p.g.Tem = s->Tem; p.g.e_int = s->e_int; p.g.eta = s->eta; p.g.csound = s->csound;
  p.g.machno = s->machno; p.g.mu_fluid = s->mu_fluid; p.g.Reta = loc.Reta; p.g.mu_factor = s->mu_factor;
  p.g.node_member = m->nmember > 0 ? m->node_member : nullptr;
  p.g.member_reduce = m->nmember > 0 ? 1 : 0;
  p.nmember = m->nmember;
  p.member_node_off = m->member_node_off;
  p.member_scal = m->member_scal;
  p.v = make_visc_args(m, &loc, dt_next, mixed ? m->mue32 : nullptr);
  const int nm = m->nmember > 0 ? m->nmember : 1;
  for (int stage = 1; stage <= 4; ++stage) {
    const double* y = m->buf.ys;
    if (stage == 1)
      p.r = make_rhs_args(m, mixed, s->rho, s->q, s->q + N, s->q + 2 * N, s->E, s->mu_factor, nullptr);
    else
      p.r = make_rhs_args(m, mixed, y, y + N, y + 2 * N, y + 3 * N, y + 4 * N, s->mu_factor, nullptr);
    p.g.ys = nullptr;
    fill_gather_args(m, stage, p.g);
    p.stage = stage;
    if (stage == 4 && dt_next) SOD_CUDA(cudaMemsetAsync(p.v.dt_bits, 0x7F, sizeof(double) * nm, st));
    if (int rc = launch_stage(p, mixed, epb, ctas_per_sm, nullptr, st)) return rc;
    if (stage == 4 && dt_next)
      SOD_CUDA(cudaMemcpyAsync(dt_next, p.v.dt_bits, sizeof(double) * nm, cudaMemcpyDeviceToDevice, st));
  }
  return SOD_OK;
}

// One RK4 step on device state (mu_e already in m->mue_int / mue32).  When ev is non-null,
// ev[2*slot] / ev[2*slot+1] bracket each kernel: slots 0-3 KR stages, 4-7 KG stages, 8 KV.
// When stage_store is non-null the stage states Y2, Y3, Y4 (5 columns of npoin each) are
// written there instead of the internal stage buffer (for the adjoint's reverse sweep).
// state_done (optional) is recorded on st once the new state and its EOS fields are final, before
// the entropy viscosity and dt (and LES's sgs viscosity) that end the step.
int run_step(SodMesh* m, SodState* s, const double* dt_dev, double* dt_next, bool mixed, cudaStream_t st,
             cudaEvent_t* ev = nullptr, double* stage_store = nullptr, cudaEvent_t state_done = nullptr) {
  NvtxRange range(mixed ? "sod rk4 step (mixed)" : "sod rk4 step (fp64)");
  const size_t N = m->npoin;
  const int epb = rhs_epb(m, mixed);
  SodState loc = *s;
  const bool les = les_active(m, s);
  double* reta_tmp = nullptr;
  if (!loc.Reta) {
    // stage 4 reads rsum[5] before writing Reta, element-wise, so aliasing is safe
    reta_tmp = reta_scratch(m);
    loc.Reta = reta_tmp;
  }
  int rc;
  // non-periodic path / buffer zone: updateBuffer, then the boundary routine, on every stage
  // state and on the updated state
  const bool bc = m->bc.nb > 0;
  const bool zone = m->zone.nb > 0;
  const bool pre = bc || zone;
  const int pctas = m->persist_ctas[mixed ? 1 : 0];
  if (pctas > 0 && !pre && !les && m->wmodel.nw == 0 && !m->source && !ev && !stage_store) {
    // the one-launch stages form the entropy viscosity inside stage 4: the state is final at the end
    rc = run_step_persist(m, s, loc, dt_dev, dt_next, mixed, epb, pctas, st);
    if (!rc && state_done) SOD_CUDA(cudaEventRecord(state_done, st));
    return rc;
  }
  auto pre_stage = [&](double* ys, int stage_of) -> int {
    if (zone)
      if (int r = zone_stage(m, ys, st)) return r;
    return bc ? bc_stage(m, ys, stage_of, st) : SOD_OK;
  };
  if (bc) {
    rc = bc_snapshot_u(m, s->u, st);  // u(:,:,pos) before the update, read by slip walls
    if (rc) return rc;
  }
  for (int stage = 1; stage <= 4; ++stage) {
    double* yin = (stage_store && stage >= 2) ? stage_store + (size_t)(stage - 2) * 5 * N : m->buf.ys;
    if (pre && stage == 1) {
      // the first stage state is the state itself with the routines applied to a copy
      k_copy_state<<<(unsigned)((N + 255) / 256), 256, 0, st>>>((int64_t)N, s->rho, s->q, s->E, yin);
      SOD_CHECK_LAUNCH();
      rc = pre_stage(yin, 1);
      if (rc) return rc;
    }
    const bool from_state = stage == 1 && !pre;
    const double* src_rho = from_state ? s->rho : yin;
    const double* src_q0 = from_state ? s->q : yin + N;
    const double* src_q1 = from_state ? s->q + N : yin + 2 * N;
    const double* src_q2 = from_state ? s->q + 2 * N : yin + 3 * N;
    const double* src_E = from_state ? s->E : yin + 4 * N;
    if (m->wmodel.nw > 0) {
      rc = wall_model_stage(m, src_rho, src_q0, src_E, s->mu_factor, st);
      if (rc) return rc;
    }
    if (ev) cudaEventRecord(ev[2 * (stage - 1)], st);
    rc = launch_rhs(m, mixed, epb, src_rho, src_q0, src_q1, src_q2, src_E, s->mu_factor, les ? m->musgs_int : nullptr,
                    st);
    if (rc) return rc;
    if (ev) cudaEventRecord(ev[2 * (stage - 1) + 1], st);
    GatherArgs g{};
    g.dt = dt_dev;
    g.y[0] = s->rho; g.y[1] = s->q; g.y[2] = s->q + N; g.y[3] = s->q + 2 * N; g.y[4] = s->E;
    g.u0 = s->u; g.u1 = s->u + N; g.u2 = s->u + 2 * N;
    g.pr = s->pr; g.Tem = s->Tem; g.e_int = s->e_int; g.eta = s->eta; g.csound = s->csound;
    g.machno = s->machno; g.mu_fluid = s->mu_fluid; g.Reta = loc.Reta; g.mu_factor = s->mu_factor;
    g.node_member = m->nmember > 0 ? m->node_member : nullptr;
    // (after boundary conditions or a buffer zone the entropy sums are formed from the changed state)
    g.member_reduce = (m->nmember > 0 || pre) ? 1 : 0;
    if (stage_store && stage < 4) g.ys = stage_store + (size_t)(stage - 1) * 5 * N;
    if (ev) cudaEventRecord(ev[2 * (3 + stage)], st);
    rc = launch_gather(m, mixed, stage, g, st);
    if (rc) return rc;
    if (stage == 4 && m->nmember > 0) {
      k_member_eta<<<m->nmember * kEtaChunks, 256, 0, st>>>(m->member_node_off, s->eta, m->member_scal, m->prm.normalise,
                                                            m->member_red, m->member_done);
      SOD_CHECK_LAUNCH();
    }
    if (pre) {
      if (stage < 4) {
        double* ynext = (stage_store && stage < 4) ? stage_store + (size_t)(stage - 1) * 5 * N : m->buf.ys;
        rc = pre_stage(ynext, stage + 1);
      } else {
        rc = zone ? zone_final(m, s, st) : SOD_OK;
        if (!rc && bc) rc = bc_final(m, s, loc.Reta, st);
      }
      if (rc) return rc;
    }
    if (ev) cudaEventRecord(ev[2 * (3 + stage) + 1], st);
  }
  if (ev) cudaEventRecord(ev[16], st);
  if (state_done) SOD_CUDA(cudaEventRecord(state_done, st));
  if (les) {
    // sgs_visc after the step (time_integ.f90:498-506), before the dt of the next step uses it
    // (CFDSolverBase.f90:1592); independent of the entropy viscosity, so it may run first
    rc = launch_sgs(m, s->u, st);
    if (rc) return rc;
  }
  rc = launch_visc_dt(m, &loc, dt_next, mixed ? m->mue32 : nullptr, st, true);
  if (ev) cudaEventRecord(ev[17], st);
  return rc;
}

}  // namespace sod

using namespace sod;

static int check_state(SodMesh* m, SodState* s) {
  SOD_ARG(m && s, "mesh/state null");
  SOD_ARG(s->rho && s->q && s->E && s->u && s->pr && s->Tem && s->e_int && s->eta && s->csound && s->machno &&
              s->mu_fluid && s->mu_factor && s->mu_e,
          "state arrays must be non-null (Reta optional)");
  return SOD_OK;
}

extern "C" {

static int rk4_main_impl(SodMesh* m, SodState* s, const double* dt_dev, double* dt_next_dev, SodPrecision prec,
                         sod_stream_t stream, cudaEvent_t state_done);

int sod_rk4_main(SodMesh* m, SodState* s, const double* dt_dev, double* dt_next_dev, SodPrecision prec,
                 sod_stream_t stream) {
  return rk4_main_impl(m, s, dt_dev, dt_next_dev, prec, stream, nullptr);
}

static int rk4_main_impl(SodMesh* m, SodState* s, const double* dt_dev, double* dt_next_dev, SodPrecision prec,
                         sod_stream_t stream, cudaEvent_t state_done) {
  int rc = check_state(m, s);
  if (rc) return rc;
  SOD_ARG(dt_dev, "dt_dev null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, s->mu_e, mixed, st);
  if (rc) return rc;
  rc = les_in(m, s, st);
  if (rc) return rc;
  rc = run_step(m, s, dt_dev, dt_next_dev, mixed, st, nullptr, nullptr, state_done);
  if (rc) return rc;
  rc = les_out(m, s, st);
  if (rc) return rc;
  return mesh_internal_to_ref_elem(m, m->mue_int, s->mu_e, st);
}

int sod_rk4_main_record(SodMesh* m, SodState* s, const double* dt_dev, double* dt_next_dev, double* stages,
                        SodPrecision prec, sod_stream_t stream) {
  int rc = check_state(m, s);
  if (rc) return rc;
  SOD_ARG(dt_dev && stages, "dt_dev/stages null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, s->mu_e, mixed, st);
  if (rc) return rc;
  rc = les_in(m, s, st);
  if (rc) return rc;
  rc = run_step(m, s, dt_dev, dt_next_dev, mixed, st, nullptr, stages);
  if (rc) return rc;
  rc = les_out(m, s, st);
  if (rc) return rc;
  return mesh_internal_to_ref_elem(m, m->mue_int, s->mu_e, st);
}

int sod_rk4_steps(SodMesh* m, SodState* s, double* dt_dev, int nsteps, SodPrecision prec, sod_stream_t stream) {
  int rc = check_state(m, s);
  if (rc) return rc;
  SOD_ARG(dt_dev && nsteps >= 0, "dt_dev/nsteps");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, s->mu_e, mixed, st);
  if (rc) return rc;
  rc = les_in(m, s, st);
  if (rc) return rc;
  if (nsteps > 0) {
    // capture one step into a graph keyed by (state pointers, dt pointer, precision, epb)
    uint64_t key = (uint64_t)(uintptr_t)s->rho ^ ((uint64_t)(uintptr_t)dt_dev << 1) ^ ((uint64_t)mixed << 63) ^
                   ((uint64_t)(uintptr_t)s->Reta << 3) ^ ((uint64_t)m->tuned_epb[mixed ? 1 : 0] << 56) ^
                   ((uint64_t)(uintptr_t)(les_active(m, s) ? s->mu_sgs : nullptr) << 5);
    auto it = m->graphs.find(key);
    if (it == m->graphs.end()) {
      cudaStream_t cap;
      SOD_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
      cudaGraph_t graph;
      int64_t before = g_launches.load();
      SOD_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
      rc = run_step(m, s, dt_dev, dt_dev, mixed, cap);
      cudaError_t ce = cudaStreamEndCapture(cap, &graph);
      cudaStreamDestroy(cap);
      if (rc) return rc;
      if (ce != cudaSuccess) {
        set_error("graph capture failed: %s", cudaGetErrorString(ce));
        return SOD_ERR_CUDA;
      }
      GraphEntry ge;
      ge.nkernels = (int)(g_launches.load() - before);
      g_launches.fetch_sub(ge.nkernels);
      cudaError_t ie = cudaGraphInstantiate(&ge.exec, graph, 0);
      cudaGraphDestroy(graph);
      if (ie != cudaSuccess) {
        set_error("graph instantiate failed: %s", cudaGetErrorString(ie));
        return SOD_ERR_CUDA;
      }
      it = m->graphs.emplace(key, ge).first;
    }
    for (int t = 0; t < nsteps; ++t) {
      SOD_CUDA(cudaGraphLaunch(it->second.exec, st));
      g_launches.fetch_add(it->second.nkernels);
    }
  }
  rc = les_out(m, s, st);
  if (rc) return rc;
  return mesh_internal_to_ref_elem(m, m->mue_int, s->mu_e, st);
}

int sod_step_profile(SodMesh* m, SodState* s, double* dt_dev, int nsteps, SodPrecision prec, sod_stream_t stream,
                     float* ms_out) {
  int rc = check_state(m, s);
  if (rc) return rc;
  SOD_ARG(dt_dev && nsteps > 0 && ms_out, "dt_dev/nsteps/ms_out");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, s->mu_e, mixed, st);
  if (rc) return rc;
  rc = les_in(m, s, st);
  if (rc) return rc;
  cudaEvent_t ev[18];
  for (int q = 0; q < 18; ++q) SOD_CUDA(cudaEventCreate(&ev[q]));
  double acc[3] = {0, 0, 0};
  for (int t = 0; t < nsteps && rc == SOD_OK; ++t) {
    rc = run_step(m, s, dt_dev, dt_dev, mixed, st, ev);
    if (rc) break;
    if (cudaEventSynchronize(ev[17]) != cudaSuccess) { rc = SOD_ERR_CUDA; break; }
    for (int q = 0; q < 9; ++q) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, ev[2 * q], ev[2 * q + 1]);
      acc[q < 4 ? 0 : (q < 8 ? 1 : 2)] += ms;
    }
  }
  for (int q = 0; q < 18; ++q) cudaEventDestroy(ev[q]);
  if (rc) return rc;
  ms_out[0] = (float)(acc[0] / (4.0 * nsteps));
  ms_out[1] = (float)(acc[1] / (4.0 * nsteps));
  ms_out[2] = (float)(acc[2] / nsteps);
  rc = les_out(m, s, st);
  if (rc) return rc;
  return mesh_internal_to_ref_elem(m, m->mue_int, s->mu_e, st);
}

// Elements-per-CTA autotuner for the fused RHS kernel: times every candidate on the caller's
// state (3 warm-up + 10 timed launches each, CUDA events on the stream) and keeps the fastest
// for this mesh and precision; later steps and newly captured graphs use it.
int sod_set_rhs_config(SodMesh* m, SodPrecision prec, int config) {
  SOD_ARG(m, "mesh null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  const bool mixed = prec == SOD_MIXED;
  const bool ok = (config == 1 || config == 2 || config == 4 || config == 8);
  SOD_ARG(ok || config == 0, "unknown fused-RHS configuration");
  if (m->tuned_epb[mixed ? 1 : 0] != config) {
    for (auto& kv : m->graphs)
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    m->graphs.clear();
  }
  m->tuned_epb[mixed ? 1 : 0] = config;
  return SOD_OK;
}

int sod_set_stage_launch(SodMesh* m, SodPrecision prec, int ctas_per_sm) {
  SOD_ARG(m, "mesh null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  SOD_ARG(ctas_per_sm >= 0 && ctas_per_sm <= 32, "ctas_per_sm must be in 0..32");
  const int i = prec == SOD_MIXED ? 1 : 0;
  if (m->persist_ctas[i] != ctas_per_sm) {
    for (auto& kv : m->graphs)
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    m->graphs.clear();
  }
  m->persist_ctas[i] = ctas_per_sm;
  return SOD_OK;
}

int sod_autotune_table(SodMesh* m, SodPrecision prec, int cap, int32_t* epb, int32_t* ctas_per_sm,
                       float* ms_per_stage) {
  SOD_ARG(m, "mesh null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  const auto& t = m->tune_table[prec == SOD_MIXED ? 1 : 0];
  const int n = (int)t.size();
  for (int q = 0; q < n && q < cap; ++q) {
    if (epb) epb[q] = t[q].epb;
    if (ctas_per_sm) ctas_per_sm[q] = t[q].ctas;
    if (ms_per_stage) ms_per_stage[q] = t[q].ms;
  }
  return n;
}

int sod_autotune(SodMesh* m, SodState* s, SodPrecision prec, int* best_epb, float* best_ms, sod_stream_t stream) {
  int rc = check_state(m, s);
  if (rc) return rc;
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, s->mu_e, mixed, st);
  if (rc) return rc;
  rc = les_in(m, s, st);
  if (rc) return rc;
  const size_t N = m->npoin;
  const int cand[] = {1, 2, 4, 8};
  cudaEvent_t e0, e1;
  SOD_CUDA(cudaEventCreate(&e0));
  SOD_CUDA(cudaEventCreate(&e1));
  // One RK stage 1 per trial (fused RHS + gather / stage update into the internal stage buffers;
  // the caller's state is only read).  Two dimensions: elements per CTA, and the launch shape -
  // two launches per stage (ctas 0) or one cooperative launch of c resident CTAs per SM.
  const bool plain = m->bc.nb == 0 && m->zone.nb == 0 && m->wmodel.nw == 0 && !m->source && !les_active(m, s);
  auto& table = m->tune_table[mixed ? 1 : 0];
  table.clear();
  GatherArgs g{};
  g.dt = m->buf.scal + 4;  // any finite scalar: stage 1 scales its stage-state update by it
  SOD_CUDA(cudaMemsetAsync(m->buf.scal + 4, 0, sizeof(double), st));
  g.y[0] = s->rho; g.y[1] = s->q; g.y[2] = s->q + N; g.y[3] = s->q + 2 * N; g.y[4] = s->E;
  g.mu_factor = s->mu_factor;
  g.node_member = nullptr;  // one dt scalar for the timing (an ensemble's per-member dt is not needed)
  auto trial = [&](int epb, int ctas, float* ms_out) -> int {
    int r2 = SOD_OK;
    auto once = [&]() -> int {
      if (ctas == 0) {
        int r3 = launch_rhs(m, mixed, epb, s->rho, s->q, s->q + N, s->q + 2 * N, s->E, s->mu_factor, nullptr, st);
        if (r3) return r3;
        GatherArgs gg = g;
        return launch_gather(m, mixed, 1, gg, st);
      }
      StageArgs p{};
      p.r = make_rhs_args(m, mixed, s->rho, s->q, s->q + N, s->q + 2 * N, s->E, s->mu_factor, nullptr);
      p.g = g;
      fill_gather_args(m, 1, p.g);
      p.stage = 1;
      return launch_stage(p, mixed, epb, ctas, nullptr, st);
    };
    for (int r = 0; r < 3 && r2 == SOD_OK; ++r) r2 = once();
    cudaEventRecord(e0, st);
    for (int r = 0; r < 10 && r2 == SOD_OK; ++r) r2 = once();
    cudaEventRecord(e1, st);
    if (r2) return r2;
    if (cudaEventSynchronize(e1) != cudaSuccess) return SOD_ERR_CUDA;
    cudaEventElapsedTime(ms_out, e0, e1);
    *ms_out /= 10.f;
    return SOD_OK;
  };
  int best = 0, best_ctas = 0;
  float bms = 1e30f, bms_rhs = 1e30f;
  for (int c = 0; c < 4 && rc == SOD_OK; ++c) {
    const int epb = cand[c];
    // the fused RHS alone (reported as best_ms, as before)
    {
      for (int r = 0; r < 3 && rc == SOD_OK; ++r)
        rc = launch_rhs(m, mixed, epb, s->rho, s->q, s->q + N, s->q + 2 * N, s->E, s->mu_factor, nullptr, st);
      cudaEventRecord(e0, st);
      for (int r = 0; r < 10 && rc == SOD_OK; ++r)
        rc = launch_rhs(m, mixed, epb, s->rho, s->q, s->q + N, s->q + 2 * N, s->E, s->mu_factor, nullptr, st);
      cudaEventRecord(e1, st);
      if (rc) break;
      if (cudaEventSynchronize(e1) != cudaSuccess) { rc = SOD_ERR_CUDA; break; }
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      bms_rhs = std::min(bms_rhs, ms / 10.f);
    }
    // launch shapes: two launches, then persistent grids of occ, 3/4 occ and 1/2 occ CTAs per SM
    int shapes[4] = {0, 0, 0, 0}, ns = 1;
    if (plain) {
      const void* fn = nullptr;
      size_t smem = 0;
      persist_kernel_info(mixed, epb, m->prm.total_enthalpy != 0, &fn, &smem);
      int occ = 0;
      if (fn && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 64 * epb, smem) == cudaSuccess && occ > 0) {
        const int opts[3] = {occ, std::max(1, (3 * occ) / 4), std::max(1, occ / 2)};
        for (int o : opts) {
          bool dup = false;
          for (int q = 1; q < ns; ++q) dup |= shapes[q] == o;
          if (!dup) shapes[ns++] = o;
        }
      }
    }
    for (int q = 0; q < ns && rc == SOD_OK; ++q) {
      float ms = 0.f;
      rc = trial(epb, shapes[q], &ms);
      if (rc) break;
      table.push_back(SodMesh::TuneEntry{epb, shapes[q], ms});
      if (ms < bms) { bms = ms; best = epb; best_ctas = shapes[q]; }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  const int i = mixed ? 1 : 0;
  if (m->tuned_epb[i] != best || m->persist_ctas[i] != best_ctas) {
    for (auto& kv : m->graphs)
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    m->graphs.clear();
  }
  m->tuned_epb[i] = best;
  m->persist_ctas[i] = best_ctas;
  if (best_epb) *best_epb = best;
  if (best_ms) *best_ms = bms_rhs;
  return SOD_OK;
}

int sod_rhs(SodMesh* m, const double* rho, const double* q, const double* E, const double* mu_e,
            const double* mu_factor, double* Rmass, double* Rmom, double* Rener, double* Reta,
            SodPrecision prec, sod_stream_t stream) {
  SOD_ARG(m && rho && q && E && mu_e && mu_factor, "inputs null");
  SOD_ARG(prec == SOD_FP64 || prec == SOD_MIXED, "precision");
  cudaStream_t st = (cudaStream_t)stream;
  const bool mixed = prec == SOD_MIXED;
  int rc = ensure_step_buffers(m, mixed);
  if (rc) return rc;
  rc = mesh_mue_in(m, mu_e, mixed, st);
  if (rc) return rc;
  const size_t N = m->npoin;
  const int epb = rhs_epb(m, mixed);
  rc = launch_rhs(m, mixed, epb, rho, q, q + N, q + 2 * N, E, mu_factor, nullptr, st);
  if (rc) return rc;
  GatherArgs g{};
  g.out[0] = Rmass;
  g.out[1] = Rmom ? Rmom : nullptr;
  g.out[2] = Rmom ? Rmom + N : nullptr;
  g.out[3] = Rmom ? Rmom + 2 * N : nullptr;
  g.out[4] = Rener;
  g.out[5] = Reta;
  return launch_gather(m, mixed, 0, g, st);
}

int sod_rk4_main_host(SodMesh* m, SodState* h, double dt_host, double* dt_next_host, SodPrecision prec,
                      sod_stream_t stream) {
  SOD_ARG(m && h, "mesh/state null");
  SOD_ARG(h->rho && h->q && h->E && h->mu_e && h->mu_factor, "host state arrays null");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t N = m->npoin, EN = (size_t)m->nelem * NN;
  // persistent device mirror owned by the mesh
  auto& mv = m->host_mirror;
  const size_t sizes[] = {N, 3 * N, N, 3 * N, N, N, N, N, N, N, N, N, EN, N, 1, EN};
  if (mv.empty()) {
    for (size_t s : sizes) {
      double* p = nullptr;
      SOD_CUDA(cudaMalloc(&p, s * sizeof(double)));
      mv.push_back(p);
    }
  }
  const bool les_h = h->mu_sgs && m->prm.flag_les == 1;
  SodState d{mv[0], mv[1], mv[2], mv[3], mv[4], mv[5], mv[6], mv[7], mv[8], mv[9], mv[10], mv[11], mv[12], mv[13],
             les_h ? mv[15] : nullptr};
  double* ddt = mv[14];
  SOD_CUDA(cudaMemcpyAsync(d.rho, h->rho, N * 8, cudaMemcpyHostToDevice, st));
  SOD_CUDA(cudaMemcpyAsync(d.q, h->q, 3 * N * 8, cudaMemcpyHostToDevice, st));
  SOD_CUDA(cudaMemcpyAsync(d.E, h->E, N * 8, cudaMemcpyHostToDevice, st));
  SOD_CUDA(cudaMemcpyAsync(d.mu_e, h->mu_e, EN * 8, cudaMemcpyHostToDevice, st));
  SOD_CUDA(cudaMemcpyAsync(d.mu_factor, h->mu_factor, N * 8, cudaMemcpyHostToDevice, st));
  SOD_CUDA(cudaMemcpyAsync(ddt, &dt_host, 8, cudaMemcpyHostToDevice, st));
  if (les_h) SOD_CUDA(cudaMemcpyAsync(d.mu_sgs, h->mu_sgs, EN * 8, cudaMemcpyHostToDevice, st));
  struct Pair { double* hst; double* dev; size_t n; };
  Pair outs[] = {{h->rho, d.rho, N}, {h->q, d.q, 3 * N}, {h->E, d.E, N}, {h->u, d.u, 3 * N}, {h->pr, d.pr, N},
                 {h->Tem, d.Tem, N}, {h->e_int, d.e_int, N}, {h->eta, d.eta, N}, {h->csound, d.csound, N},
                 {h->machno, d.machno, N}, {h->mu_fluid, d.mu_fluid, N}, {h->mu_e, d.mu_e, EN},
                 {h->Reta, d.Reta, N}, {les_h ? h->mu_sgs : nullptr, d.mu_sgs, EN}};
  if (m->has_slaves)  // the step leaves slave rows as they are: bring in the rows it will copy back
    for (int i = 3; i < 11; ++i)
      if (outs[i].hst) SOD_CUDA(cudaMemcpyAsync(outs[i].dev, outs[i].hst, outs[i].n * 8, cudaMemcpyHostToDevice, st));
  if (m->has_slaves && h->Reta) SOD_CUDA(cudaMemcpyAsync(d.Reta, h->Reta, N * 8, cudaMemcpyHostToDevice, st));
  // the state fields are copied back on a second stream as soon as the step has formed them, so
  // that the read-back overlaps the entropy viscosity and dt that end the step; mu_e (and mu_sgs)
  // and dt follow on the caller's stream, which then waits for the copies
  if (!m->host_copy_stream) {
    SOD_CUDA(cudaStreamCreateWithFlags(&m->host_copy_stream, cudaStreamNonBlocking));
    SOD_CUDA(cudaEventCreateWithFlags(&m->host_ev_state, cudaEventDisableTiming));
    SOD_CUDA(cudaEventCreateWithFlags(&m->host_ev_copied, cudaEventDisableTiming));
  }
  cudaStream_t cs = m->host_copy_stream;
  int rc = rk4_main_impl(m, &d, ddt, ddt, prec, stream, m->host_ev_state);
  if (rc) return rc;
  SOD_CUDA(cudaStreamWaitEvent(cs, m->host_ev_state, 0));
  for (auto& o : outs) {
    if (!o.hst) continue;
    const bool tail = o.dev == d.mu_e || o.dev == d.mu_sgs;  // written after the state is final
    SOD_CUDA(cudaMemcpyAsync(o.hst, o.dev, o.n * 8, cudaMemcpyDeviceToHost, tail ? st : cs));
  }
  SOD_CUDA(cudaEventRecord(m->host_ev_copied, cs));
  if (dt_next_host) SOD_CUDA(cudaMemcpyAsync(dt_next_host, ddt, 8, cudaMemcpyDeviceToHost, st));
  SOD_CUDA(cudaStreamWaitEvent(st, m->host_ev_copied, 0));
  if (int rc2 = sync_stream(st)) return rc2;
  bool bad = false;
  if (int rc3 = take_nonfinite(m, st, &bad)) return rc3;
  if (bad) {
    set_error("a non-finite value (NaN/Inf) appeared in rho, q or E during the step");
    return SOD_ERR_NONFINITE;
  }
  return SOD_OK;
}

int sod_smart_visc_spectral(SodMesh* m, const double* Reta, const double* rho, const double* u,
                            const double* csound, const double* Tem, const double* eta, double* mu_e,
                            sod_stream_t stream);
int sod_adapt_dt_cfl(SodMesh* m, const double* u, const double* csound, const double* mu_fluid,
                     const double* mu_sgs, const double* rho, double* dt_dev, sod_stream_t stream);

}  // extern "C"

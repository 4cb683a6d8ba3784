// Fused stochastic LLG-Heun passes (sm_100a).
//
// The reference step (src/simulate/LLGHeun.cpp:160-282) makes two full field
// evaluations and four streaming loops over 12 SoA arrays per step; its CUDA
// backend (src/cuda/llg_heun.cu:121-208) makes 11 launches and 3 copies.
// Here a step is two launches, each one HBM pass:
//
//   predictor  s'  = n(s0 + dt * f(s0, H(s0) + H_ext))          reads s0, writes s'
//   corrector  s1  = n(s0 + dt/2 (f(s0,..) + f(s', H(s') + H_ext)))
//                                                 reads s0 and s', writes s1 over s0
//
// H(s) is the exchange gather over a sliced-ELL (SELL-32) copy of the CSR
// list (a warp = 32 consecutive atoms; bond k of lane l sits at
// slice_off + 32 k + l, so every index/coupling load of a warp is one 128-byte
// line) plus uniaxial and cubic anisotropy; H_ext is thermal noise
// regenerated in-register from Philox (no noise buffer), applied field and the
// macrocell dipole field looked up by cell id.  The predictor's
// f(s0, ...) dt is not stored: since f is perpendicular to s0 and
// s' = (s0 + f dt)/|s0 + f dt|, the corrector recovers
// f dt = s' |s0|^2 / (s'.s0) - s0 exactly from the two states it reads anyway.
#pragma once
#include <cuda_runtime.h>

#include "llg_device.cuh"

namespace vgpu {

// Predictor tail of atom i, given s0 and its total field H:
// s' = n(s0 + dt f(s0, H)) (LLGHeun.cpp:195-222).  The step tails return the
// state that they compute; llg_*_finish store it.
template <typename R>
__device__ __forceinline__ void llg_predict(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                            const R H[3], R out[3]) {
   R d[3];
   llg_rhs<R>(m.A, m.B, S0, H, d);
   if (a.ex) { a.ex[i] = d[0]; a.ey[i] = d[1]; a.ez[i] = d[2]; }
   R Sn[3] = {S0[0] + d[0] * a.dt, S0[1] + d[1] * a.dt, S0[2] + d[2] * a.dt};
   const R r = rsqrt_<R>(Sn[0] * Sn[0] + Sn[1] * Sn[1] + Sn[2] * Sn[2]);
   out[0] = Sn[0] * r; out[1] = Sn[1] * r; out[2] = Sn[2] * r;
}

template <typename R>
__device__ __forceinline__ void llg_predict_finish(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                                   const R H[3]) {
   R o[3];
   llg_predict<R>(a, i, m, S0, H, o);
   a.bx[i] = o[0]; a.by[i] = o[1]; a.bz[i] = o[2];
}

// Corrector tail of atom i, given s0, s' and the total field H' of s':
// s1 = n(s0 + dt/2 (f0 + f(s', H'))) (LLGHeun.cpp:238-279), written over s0.
template <typename R>
__device__ __forceinline__ void llg_correct(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                            const R S1[3], const R H[3], R out[3]) {
   R d[3];
   llg_rhs<R>(m.A, m.B, S1, H, d);
   R Sn[3];
   if (a.ex) {
      // stored predictor increment: s0 + dt/2 (f0 + f1) as LLGHeun.cpp:264-266
      const R e0[3] = {a.ex[i], a.ey[i], a.ez[i]};
#pragma unroll
      for (int k = 0; k < 3; ++k) Sn[k] = S0[k] + a.half_dt * (e0[k] + d[k]);
   } else {
      // recover the predictor increment f(s0) dt from s0 and s'
      const R s00 = S0[0] * S0[0] + S0[1] * S0[1] + S0[2] * S0[2];
      const R c = s00 / (S1[0] * S0[0] + S1[1] * S0[1] + S1[2] * S0[2]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
         const R e = S1[k] * c - S0[k];
         Sn[k] = S0[k] + ((R)0.5 * e + a.half_dt * d[k]);
      }
   }
   const R n2 = Sn[0] * Sn[0] + Sn[1] * Sn[1] + Sn[2] * Sn[2];
   const R r = rsqrt_<R>(n2);
   if (!(n2 > (R)0.25 && n2 < (R)4)) atomicOr(a.status, 1);  // non-finite or runaway
   out[0] = Sn[0] * r; out[1] = Sn[1] * r; out[2] = Sn[2] * r;
}

template <typename R>
__device__ __forceinline__ void llg_correct_finish(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                                   const R S1[3], const R H[3]) {
   R o[3];
   llg_correct<R>(a, i, m, S0, S1, H, o);
   a.ax[i] = o[0]; a.ay[i] = o[1]; a.az[i] = o[2];
}

// Cayley-transform rotation of sim::LLG_Midpoint (src/simulate/LLGMidpoint.cpp:
// 70-105, 117-150): F = H + alpha M x H, b2 = beta^2,
// out = (S (1 - b2 F.F) + 2 (beta F x S + F b2 F.S)) / (1 + b2 F.F).
template <typename R>
__device__ __forceinline__ void midpoint_rotate(R alpha, R beta, const R M[3], const R S[3], const R H[3],
                                                R out[3]) {
   const R beta2 = beta * beta;
   const R F[3] = {H[0] + alpha * (M[1] * H[2] - M[2] * H[1]), H[1] + alpha * (M[2] * H[0] - M[0] * H[2]),
                   H[2] + alpha * (M[0] * H[1] - M[1] * H[0])};
   const R FdotF = F[0] * F[0] + F[1] * F[1] + F[2] * F[2];
   const R beta2FdotS = beta2 * (F[0] * S[0] + F[1] * S[1] + F[2] * S[2]);
   const R c1 = (R)1 / ((R)1 + beta2 * FdotF);
   const R c2 = (R)1 - beta2 * FdotF;
   out[0] = c1 * (S[0] * c2 + (R)2 * (beta * (F[1] * S[2] - F[2] * S[1]) + F[0] * beta2FdotS));
   out[1] = c1 * (S[1] * c2 + (R)2 * (beta * (F[2] * S[0] - F[0] * S[2]) + F[1] * beta2FdotS));
   out[2] = c1 * (S[2] * c2 + (R)2 * (beta * (F[0] * S[1] - F[1] * S[0]) + F[2] * beta2FdotS));
}

// midpoint first half: M = (S0 + R(S0; F(S0, H))) / 2, not renormalised
template <typename R>
__device__ __forceinline__ void mid_predict(const MatParams<R>& m, const R S0[3], const R H[3], R out[3]) {
   R r[3];
   midpoint_rotate<R>(m.alpha, m.beta_mid, S0, S0, H, r);
   out[0] = (S0[0] + r[0]) * (R)0.5;
   out[1] = (S0[1] + r[1]) * (R)0.5;
   out[2] = (S0[2] + r[2]) * (R)0.5;
}

// midpoint second half: S1 = R(S0; F(M, H(M))), written over S0
template <typename R>
__device__ __forceinline__ void mid_correct(const LLGArgs<R>& a, const MatParams<R>& m, const R S0[3], const R M[3],
                                            const R H[3], R out[3]) {
   midpoint_rotate<R>(m.alpha, m.beta_mid, M, S0, H, out);
   const R n2 = out[0] * out[0] + out[1] * out[1] + out[2] * out[2];
   if (!(n2 > (R)0.25 && n2 < (R)4)) atomicOr(a.status, 1);  // non-finite or runaway
}

// the half-steps of a pass variant
template <typename R, int VAR>
__device__ __forceinline__ void first_half(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                           const R H[3], R out[3]) {
   if (VAR == VAR_MIDPOINT) mid_predict<R>(m, S0, H, out);
   else llg_predict<R>(a, i, m, S0, H, out);
}
template <typename R, int VAR>
__device__ __forceinline__ void second_half(const LLGArgs<R>& a, int i, const MatParams<R>& m, const R S0[3],
                                            const R S1[3], const R H[3], R out[3]) {
   if (VAR == VAR_MIDPOINT) mid_correct<R>(a, m, S0, S1, H, out);
   else llg_correct<R>(a, i, m, S0, S1, H, out);
}

// Facts of a launch that the kernels for isotropic bonds are compiled for.
// ISO_FIXED: the common case -- the Heun step, one coupling per atom (one
// material per system), Philox noise, second-order uniaxial anisotropy at most,
// no host dipole field, no field per material -- with the thermal term, a batch
// (field ramp, temperature and noise stream per system) and the macrocell field
// given by the other bits.  The branches on those facts and the parameter loads
// behind them are gone (406 warp instructions per 32 atoms in the predictor of a
// thermal batch).
constexpr int kIsoBlock = 256;
enum IsoFeat : int { ISO_FIXED = 1, ISO_THERMAL = 2, ISO_BATCH = 4, ISO_CELL = 8 };
#define VGPU_ISO_FEATURES(F) F(1) F(3) F(5) F(7) F(9) F(11)

// the bits that hold for a (0 when a is not the ISO_FIXED case)
template <typename R> inline int iso_features(const LLGArgs<R>& a, int fmt, int var) {
   const bool batch = a.sys_off != nullptr;
   const bool one_j = a.M == 1 || (batch && a.m_per_sys == 1);
   if (fmt != FMT_ISO_TAB || var != VAR_HEUN || !one_j || a.hd_atom || a.cubic || a.aniso_ext || a.bq_off ||
       a.noise_mode != VGPU_NOISE_PHILOX || (sizeof(R) == 4 && a.ex) || (batch && a.cell))
      return 0;
   if (!batch && (a.ramp_n || a.local_field)) return 0;
   return ISO_FIXED | (a.thermal ? ISO_THERMAL : 0) | (batch ? ISO_BATCH : 0) | (a.cell ? ISO_CELL : 0);
}

// a with the facts of RF written in (equal to what a holds whenever
// iso_features names RF)
template <typename R, int RF> __device__ __forceinline__ LLGArgs<R> fold_iso(const LLGArgs<R>& in) {
   LLGArgs<R> a = in;
   if (RF & ISO_FIXED) {
      a.hd_atom = nullptr;
      a.cubic = 0;
      a.aniso_ext = 0;
      a.bq_off = nullptr;
      a.noise_mode = VGPU_NOISE_PHILOX;
      a.integrator = INTEG_HEUN;
      a.thermal = (RF & ISO_THERMAL) ? 1 : 0;
      if (sizeof(R) == 4) a.ex = a.ey = a.ez = nullptr;
      if (!(RF & ISO_CELL)) a.cell = nullptr;
      if (RF & ISO_BATCH) a.m_per_sys = 1;
      if (!(RF & ISO_BATCH)) {
         a.sys_off = nullptr;
         a.ramp_n = 0;
         a.local_field = 0;
         a.mat = nullptr;
      }
   }
   return a;
}

// The bonds of one atom, as the upload left them (read before pdl_begin), and
// its exchange field over isotropic bonds of one coupling J.  Rows of six keep
// their words in registers and have every neighbour's load in flight.  Same
// products in the same order as exchange_gather_w and exchange_gather_row.
struct IsoRow {
   int base, w, j[6];
};

template <typename R> __device__ __forceinline__ IsoRow iso_row(const LLGArgs<R>& a, int i) {
   IsoRow r;
   const int off = __ldg(a.slice_off + (i >> 5));
   r.w = (__ldg(a.slice_off + (i >> 5) + 1) - off) >> 5;
   r.base = off + (i & 31);
#pragma unroll
   for (int k = 0; k < 6; ++k) r.j[k] = r.w == 6 ? __ldg(a.col + r.base + 32 * k) & a.idx_mask : 0;
   return r;
}

template <typename R>
__device__ __forceinline__ void iso_field(const LLGArgs<R>& a, const IsoRow& r, R J, const R* sx, const R* sy,
                                          const R* sz, R& hx, R& hy, R& hz) {
   auto add = [&](R x, R y, R z) { hx += J * x; hy += J * y; hz += J * z; };
   if (r.w == 6) {
      R x[6], y[6], z[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) { x[k] = sx[r.j[k]]; y[k] = sy[r.j[k]]; z[k] = sz[r.j[k]]; }
#pragma unroll
      for (int k = 0; k < 6; ++k) add(x[k], y[k], z[k]);
   } else {
#pragma unroll 4
      for (int k = 0; k < r.w; ++k) {
         const int j = __ldg(a.col + r.base + 32 * k) & a.idx_mask;
         add(sx[j], sy[j], sz[j]);
      }
   }
}

// One pass over isotropic bonds with the facts of RF (launch_fmt).  With a.gx
// the predictor keeps the step's external field for the corrector, which then
// neither draws the noise again nor recomputes the field (nothing it depends on
// changes between the two passes of a step).
template <typename R, int MODE, int RF>
__global__ void __launch_bounds__(kIsoBlock) llg_iso_pass_kernel(const LLGArgs<R> in) {
   const LLGArgs<R> a = fold_iso<R, RF>(in);
   const int i = 32 * a.slice_first + blockIdx.x * blockDim.x + threadIdx.x;
   const bool on = i < a.n_upd;
   IsoRow r;
   int mi = 0;
   if (on) {
      r = iso_row<R>(a, i);
      mi = a.mat ? __ldg(a.mat + i) : 0;
   }
   pdl_begin();
   asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
   if (!on) return;
   const MatParams<R>& m = a.mp[mi];
   const R J = __ldg(a.jtab + mi * a.M + mi);
   const R S0[3] = {a.ax[i], a.ay[i], a.az[i]};
   R E[3], H[3], hx = 0, hy = 0, hz = 0, o[3];
   if (MODE == PASS_PREDICTOR) {
      iso_field<R>(a, r, J, a.ax, a.ay, a.az, hx, hy, hz);
      external_field<R>(a, i, m, true, E);
      if (a.gx) { a.gx[i] = E[0]; a.gy[i] = E[1]; a.gz[i] = E[2]; }
      site_field<R, 0, false>(a, i, m, a.ax, a.ay, a.az, S0, hx, hy, hz, H);
      H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
      llg_predict<R>(a, i, m, S0, H, o);
      a.bx[i] = o[0]; a.by[i] = o[1]; a.bz[i] = o[2];
   } else {
      const R S1[3] = {a.bx[i], a.by[i], a.bz[i]};
      if (a.gx) { E[0] = a.gx[i]; E[1] = a.gy[i]; E[2] = a.gz[i]; }
      iso_field<R>(a, r, J, a.bx, a.by, a.bz, hx, hy, hz);
      if (!a.gx) external_field<R>(a, i, m, true, E);
      site_field<R, 0, false>(a, i, m, a.bx, a.by, a.bz, S1, hx, hy, hz, H);
      H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
      llg_correct<R>(a, i, m, S0, S1, H, o);
      a.ax[i] = o[0]; a.ay[i] = o[1]; a.az[i] = o[2];
   }
}

// Predictor of atom i: s' = n(s0 + dt f(s0, H)) (Heun) or the midpoint M.
// LOAD = 1 reads neighbour spins through L2 (they may have been written
// earlier in the same launch).
template <typename R, int FMT, int LOAD, int VAR = VAR_HEUN_EXT>
__device__ __forceinline__ void llg_predict_atom(const LLGArgs<R>& a, int i) {
   const int mi = a.mat ? __ldg(a.mat + i) : 0;
   const MatParams<R> m = a.mp[mi];
   const R S0[3] = {a.ax[i], a.ay[i], a.az[i]};
   R H[3], E[3];
   spin_field<R, FMT, LOAD, false, VAR != VAR_HEUN>(a, i, mi, m, a.ax, a.ay, a.az, S0, H);
   external_field<R>(a, i, m, true, E);
   if (a.gx) { a.gx[i] = E[0]; a.gy[i] = E[1]; a.gz[i] = E[2]; }  // kept for the corrector
   H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
   R o[3];
   first_half<R, VAR>(a, i, m, S0, H, o);
   a.bx[i] = o[0]; a.by[i] = o[1]; a.bz[i] = o[2];
}

// Corrector of atom i: s1 = n(s0 + dt/2 (f0 + f(s', H'))) (Heun) or the
// midpoint's second half, written over s0.
template <typename R, int FMT, int LOAD, int VAR = VAR_HEUN_EXT>
__device__ __forceinline__ void llg_correct_atom(const LLGArgs<R>& a, int i) {
   const int mi = a.mat ? __ldg(a.mat + i) : 0;
   const MatParams<R> m = a.mp[mi];
   const R S0[3] = {a.ax[i], a.ay[i], a.az[i]};
   const R S1[3] = {a.bx[i], a.by[i], a.bz[i]};
   R H[3], E[3];
   if (a.gx) { E[0] = a.gx[i]; E[1] = a.gy[i]; E[2] = a.gz[i]; }
   spin_field<R, FMT, LOAD, false, VAR != VAR_HEUN>(a, i, mi, m, a.bx, a.by, a.bz, S1, H);
   if (!a.gx) external_field<R>(a, i, m, true, E);
   H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
   R o[3];
   second_half<R, VAR>(a, i, m, S0, S1, H, o);
   a.ax[i] = o[0]; a.ay[i] = o[1]; a.az[i] = o[2];
}

template <typename R, int FMT, int MODE, int VAR>
__global__ void __launch_bounds__(256) llg_pass_kernel(const LLGArgs<R> a) {
   // launched with programmatic stream serialisation (launch_pdl): the
   // previous kernel of the stream has completed and its writes are visible
   pdl_begin();
   const int i = (MODE == PASS_FIELD ? 0 : 32 * a.slice_first) + blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= (MODE == PASS_FIELD ? a.n : a.n_upd)) return;
   if (MODE == PASS_PREDICTOR) {
      llg_predict_atom<R, FMT, 0, VAR>(a, i);
   } else if (MODE == PASS_CORRECTOR) {
      llg_correct_atom<R, FMT, 0, VAR>(a, i);
   } else {
      // field of s0: exchange, anisotropy, applied and dipole terms (no thermal term)
      const int mi = a.mat ? __ldg(a.mat + i) : 0;
      const MatParams<R> m = a.mp[mi];
      const R S0[3] = {a.ax[i], a.ay[i], a.az[i]};
      R H[3], E[3];
      spin_field<R, FMT, 0, false, VAR != VAR_HEUN>(a, i, mi, m, a.ax, a.ay, a.az, S0, H);
      external_field<R>(a, i, m, false, E);
      a.fx[i] = H[0] + E[0]; a.fy[i] = H[1] + E[1]; a.fz[i] = H[2] + E[2];
   }
}

template <typename R, int FMT, int VAR>
inline cudaError_t launch_mode(const LLGArgs<R>& a, int mode, int grid, int bs, cudaStream_t st) {
   const dim3 g(grid), b(bs);
   if (mode == PASS_PREDICTOR) return launch_pdl(llg_pass_kernel<R, FMT, PASS_PREDICTOR, VAR>, g, b, 0, st, a);
   if (mode == PASS_CORRECTOR) return launch_pdl(llg_pass_kernel<R, FMT, PASS_CORRECTOR, VAR>, g, b, 0, st, a);
   return launch_pdl(llg_pass_kernel<R, FMT, PASS_FIELD, VAR>, g, b, 0, st, a);
}

template <typename R, int FMT>
inline cudaError_t launch_fmt(const LLGArgs<R>& a, int mode, cudaStream_t st) {
   const int bs = 256;
   const int grid = ((mode == PASS_FIELD ? a.n : a.n_upd - 32 * a.slice_first) + bs - 1) / bs;
   if (grid <= 0) return cudaSuccess;
   if constexpr (FMT == FMT_ISO_TAB) {
      const int var = a.integrator == INTEG_MIDPOINT ? VAR_MIDPOINT : VAR_HEUN;
      switch (mode == PASS_FIELD ? 0 : iso_features<R>(a, FMT, var)) {
#define VGPU_F(k)                                                                                             \
   case k:                                                                                                    \
      return launch_pdl(mode == PASS_PREDICTOR ? llg_iso_pass_kernel<R, PASS_PREDICTOR, k>                    \
                                               : llg_iso_pass_kernel<R, PASS_CORRECTOR, k>,                   \
                        dim3((a.n_upd - 32 * a.slice_first + kIsoBlock - 1) / kIsoBlock), dim3(kIsoBlock), 0, st, a);
         VGPU_ISO_FEATURES(VGPU_F)
#undef VGPU_F
      }
   }
   if (a.integrator == INTEG_MIDPOINT && mode != PASS_FIELD) return launch_mode<R, FMT, VAR_MIDPOINT>(a, mode, grid, bs, st);
   if (a.aniso_ext || a.bq_off) return launch_mode<R, FMT, VAR_HEUN_EXT>(a, mode, grid, bs, st);
   return launch_mode<R, FMT, VAR_HEUN>(a, mode, grid, bs, st);
}

template <typename R>
cudaError_t launch_llg_pass(const LLGArgs<R>& a, int fmt, int mode, int nslices, cudaStream_t st) {
   (void)nslices;
   switch (fmt) {
      case FMT_ISO_TAB: return launch_fmt<R, FMT_ISO_TAB>(a, mode, st);
      case FMT_ISO_BOND: return launch_fmt<R, FMT_ISO_BOND>(a, mode, st);
      case FMT_VEC_TAB: return launch_fmt<R, FMT_VEC_TAB>(a, mode, st);
      case FMT_VEC_BOND: return launch_fmt<R, FMT_VEC_BOND>(a, mode, st);
      case FMT_DMI_TAB: return launch_fmt<R, FMT_DMI_TAB>(a, mode, st);
      default: return launch_fmt<R, FMT_TENSOR_BOND>(a, mode, st);
   }
}

template <typename R>
__global__ void thermal_noise_kernel(const LLGArgs<R> a) {
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= a.n) return;
   R gx, gy, gz;
   thermal_xi(a, i, gx, gy, gz);
   a.fx[i] = gx; a.fy[i] = gy; a.fz[i] = gz;
}

template <typename R>
cudaError_t launch_thermal_noise(const LLGArgs<R>& a, cudaStream_t st) {
   thermal_noise_kernel<R><<<(a.n + 255) / 256, 256, 0, st>>>(a);
   return cudaGetLastError();
}
}  // namespace vgpu

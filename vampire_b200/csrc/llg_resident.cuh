// Many LLG steps in one launch, for systems whose atoms fit the resident
// threads of the GPU.
//
// A step is two dependent passes over the atoms.  As two launches each pass of
// a small system costs what its launch costs the host, about 3 us, whatever its
// size below some 50,000 atoms; above that every launch starts its loads cold
// and draws the thermal noise again.  Here one cooperative launch runs all
// steps: a thread owns K atoms, whose spins, predictor state and external field
// stay in its registers and whose bond words stay in shared memory; only the
// neighbours' spins travel.
//
// They travel with their time: a spin is stored as one 16-byte word {x, y, z,
// half-step} (FP64: two words, the half-step in both), written and read whole,
// and a reader that finds an older half-step reads again.  No barrier, no
// flag and no fence is needed, so a half-step costs one store and one load
// through L2 and its arithmetic.  (With a flag per block behind
// release/acquire fences a half-step took 2.9 us, no better than a launch.)
// Microseconds a step of a long launch, simple cubic, 300 K: 2.15 at 8,000 and
// 1.98 at 32,768 atoms (5.0 in two launches), FP64 2.95 and 3.08; 151,951 atoms
// 5.5 (11.0); a 37,044-atom FCC alloy with DMI 5.0 (8.6).  What bounds it is the
// wait for the words, the largest share of the cycles between two instructions of
// a warp at every size, with 14 % of the issue slots in use at 8,000 atoms, 49 %
// (566 instructions per 32 atoms and step, polls included) and half of the L1
// data pipe at 151,951.
//
// The two states keep apart what a reader may still need: an atom overwrites
// its spin of the last step only after reading every neighbour's predictor
// state, which those neighbours formed after reading that spin; and its
// predictor state only after reading every neighbour's new spin.  That needs
// neighbours to be mutual (res_mutual_kernel checks it at upload; a system with
// one-sided bonds runs pass by pass).
//
// The thermal noise of the next step needs no neighbour and is drawn while the
// stores travel.  Waits are bounded (1 s): a warp that gives up sets status bit
// 2 (VGPU_ERR_TIMEOUT on the host) and leaves, and the others then give up too.
// Half-steps are numbered through from launch to launch, so what an earlier
// launch left is never taken for the present.  a.wait_test marks the first words
// with the number before, which no wait asks for.
//
// The arithmetic is that of the passes (the same functions in the same order),
// so the states are the same bit for bit.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "llg_kernels.cuh"

namespace vgpu {

constexpr int kResBlock = kResidentBlock;       // small blocks: a small system spreads over more SMs
constexpr int kResSlices = kResBlock / 32;
constexpr uint64_t kResWaitNs = 1000000000ull;  // 1 s
constexpr int kResMaxMat = 32;                  // material rows kept in shared memory

__device__ __forceinline__ uint64_t res_now() {
   uint64_t t;
   asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
   return t;
}

// 16-byte words that are written and read whole (one access, so a reader sees
// a value and its half-step together)
__device__ __forceinline__ void res_store(void* p, uint64_t lo, uint64_t hi) {
   asm volatile("{\n .reg .b128 v;\n mov.b128 v, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], v;\n}" ::"l"(p), "l"(lo),
                "l"(hi)
                : "memory");
}
__device__ __forceinline__ void res_load(const void* p, uint64_t& lo, uint64_t& hi) {
   asm volatile("{\n .reg .b128 v;\n ld.relaxed.gpu.global.b128 v, [%2];\n mov.b128 {%0, %1}, v;\n}"
                : "=l"(lo), "=l"(hi)
                : "l"(p)
                : "memory");
}

// the spin of one atom and its half-step: FP32 one word {x, y, z, t}, FP64 two
// words {x, low y, t}, {high y, z, t} (32-bit parts), `plane` bytes apart; p: the
// atom's byte offset
template <typename R> struct ResSpin;
template <> struct ResSpin<float> {
   static constexpr int kWords = 1;
   uint64_t lo, hi;
   __device__ __forceinline__ void load(const char* X, uint32_t, uint32_t p) { res_load(X + p, lo, hi); }
   __device__ __forceinline__ uint32_t late(uint32_t t) const { return (uint32_t)(hi >> 32) ^ t; }
   __device__ __forceinline__ float x() const { return __uint_as_float((uint32_t)lo); }
   __device__ __forceinline__ float y() const { return __uint_as_float((uint32_t)(lo >> 32)); }
   __device__ __forceinline__ float z() const { return __uint_as_float((uint32_t)hi); }
   static __device__ __forceinline__ void store(char* X, uint32_t, uint32_t p, const float S[3], uint32_t t) {
      res_store(X + p, (uint64_t)__float_as_uint(S[0]) | ((uint64_t)__float_as_uint(S[1]) << 32),
                (uint64_t)__float_as_uint(S[2]) | ((uint64_t)t << 32));
   }
};
template <> struct ResSpin<double> {
   static constexpr int kWords = 2;
   uint64_t a0, a1, b0, b1;
   __device__ __forceinline__ void load(const char* X, uint32_t plane, uint32_t p) {
      res_load(X + p, a0, a1);
      res_load(X + plane + p, b0, b1);
   }
   __device__ __forceinline__ uint32_t late(uint32_t t) const {
      return ((uint32_t)(a1 >> 32) ^ t) | ((uint32_t)(b1 >> 32) ^ t);
   }
   __device__ __forceinline__ double x() const { return __longlong_as_double((long long)a0); }
   __device__ __forceinline__ double y() const { return __hiloint2double((int)(uint32_t)b1, (int)(uint32_t)a1); }
   __device__ __forceinline__ double z() const { return __longlong_as_double((long long)b0); }
   static __device__ __forceinline__ void store(char* X, uint32_t plane, uint32_t p, const double S[3], uint32_t t) {
      const uint64_t y = (uint64_t)__double_as_longlong(S[1]), tt = (uint64_t)t << 32;
      res_store(X + p, (uint64_t)__double_as_longlong(S[0]), (y & 0xffffffffull) | tt);
      res_store(X + plane + p, (uint64_t)__double_as_longlong(S[2]), (y >> 32) | tt);
   }
};

// The spins at byte offsets p[0..W-1] at half-step t, all their loads in flight;
// while one of a warp's is late, all are read again.  All lanes of a warp call
// together; false in every lane when one of them waited beyond the limit.
template <typename R, int W>
__device__ __forceinline__ bool res_read(const char* X, uint32_t plane, const uint32_t p[W], uint32_t t,
                                         ResSpin<R> s[W]) {
   uint32_t late = 0;
#pragma unroll
   for (int k = 0; k < W; ++k) s[k].load(X, plane, p[k]);
#pragma unroll
   for (int k = 0; k < W; ++k) late |= s[k].late(t);
   if (!__any_sync(0xffffffffu, late != 0)) return true;
   const uint64_t t0 = res_now();
   for (int polls = 1;; ++polls) {
      late = 0;
#pragma unroll
      for (int k = 0; k < W; ++k) s[k].load(X, plane, p[k]);
#pragma unroll
      for (int k = 0; k < W; ++k) late |= s[k].late(t);
      if (!__any_sync(0xffffffffu, late != 0)) return true;
      if ((polls & 255) == 0 && __any_sync(0xffffffffu, res_now() - t0 > kResWaitNs)) return false;
   }
}

// bond words of a format kept in shared memory: neighbour | material bits
// (FMT_ISO_TAB), neighbour | coupling index (FP32 FMT_DMI_TAB compact records)
template <typename R, int FMT> constexpr bool res_words() {
   return FMT == FMT_ISO_TAB || (FMT == FMT_DMI_TAB && sizeof(R) == 4);
}

// what one atom's gather needs besides the spins
template <typename R> struct ResRow {
   int base, w;          // SELL entry of the first bond, bonds
   const uint32_t* w0;   // words in shared memory (res_words formats), stride 32
   int mi;
   bool one_j;           // one coupling for every bond of the atom: j0
   R j0;
   const float4* dict;
};

// coupling index or material of a bond word
template <typename R, int FMT> __device__ __forceinline__ uint32_t res_coupling(const LLGArgs<R>& a, uint32_t c) {
   if (FMT == FMT_DMI_TAB && sizeof(R) == 4) return c >> a.crec_shift;
   return a.mat_shift ? c >> a.mat_shift : 0u;
}

// one bond of the exchange field, as in exchange_gather and its fixed-width and
// compact-record forms
// (q: coupling index of compact records, else the neighbour's material)
template <typename R, int FMT>
__device__ __forceinline__ void res_bond(const LLGArgs<R>& a, const ResRow<R>& r, int k, uint32_t q, R x, R y, R z,
                                         R& hx, R& hy, R& hz) {
   const int e = r.base + 32 * k;
   if constexpr (FMT == FMT_DMI_TAB && sizeof(R) == 4) {
      const float4 d = r.dict[q];
      if (a.tab_scalar) {
         dmi_bond<R>((R)d.x, (R)d.x, (R)d.x, (R)d.y, (R)d.z, (R)d.w, x, y, z, hx, hy, hz);
      } else {
         const float4 d2 = r.dict[a.cdict_n + q];
         dmi_bond<R>((R)d.x, (R)d2.x, (R)d2.y, (R)d.y, (R)d.z, (R)d.w, x, y, z, hx, hy, hz);
      }
   } else if constexpr (FMT == FMT_ISO_TAB) {
      const R J = r.one_j ? r.j0 : __ldg(a.jtab + r.mi * a.M + (int)q);
      hx += J * x; hy += J * y; hz += J * z;
   } else if constexpr (FMT == FMT_ISO_BOND) {
      const R J = __ldg(a.jb[0] + e);
      hx += J * x; hy += J * y; hz += J * z;
   } else if constexpr (FMT == FMT_VEC_TAB || FMT == FMT_DMI_TAB) {
      const R* t = a.jtab + 3 * (r.mi * a.M + (int)q);
      if constexpr (FMT == FMT_VEC_TAB) {
         hx += __ldg(t) * x; hy += __ldg(t + 1) * y; hz += __ldg(t + 2) * z;
      } else {
         const R dx = __ldg(a.jb[0] + e), dy = __ldg(a.jb[1] + e), dz = __ldg(a.jb[2] + e);
         dmi_bond<R>(__ldg(t), __ldg(t + 1), __ldg(t + 2), dx, dy, dz, x, y, z, hx, hy, hz);
      }
   } else if constexpr (FMT == FMT_VEC_BOND) {
      hx += __ldg(a.jb[0] + e) * x; hy += __ldg(a.jb[1] + e) * y; hz += __ldg(a.jb[2] + e) * z;
   } else {
      const R t0 = __ldg(a.jb[0] + e), t1 = __ldg(a.jb[1] + e), t2 = __ldg(a.jb[2] + e);
      const R t3 = __ldg(a.jb[3] + e), t4 = __ldg(a.jb[4] + e), t5 = __ldg(a.jb[5] + e);
      const R t6 = __ldg(a.jb[6] + e), t7 = __ldg(a.jb[7] + e), t8 = __ldg(a.jb[8] + e);
      hx += (t0 * x + t1 * y + t2 * z);
      hy += (t3 * x + t4 * y + t5 * z);
      hz += (t6 * x + t7 * y + t8 * z);
   }
}

// Exchange field of one atom at half-step t, W bonds at a time with all their
// loads in flight.  The row width is the same for all lanes of a warp (a slice);
// padded bonds read the atom's own spin (self, always in time) and add nothing.
template <typename R, int FMT, int W>
__device__ __forceinline__ bool res_gather(const LLGArgs<R>& a, const ResRow<R>& r, const char* X, uint32_t plane,
                                           uint32_t self, uint32_t t, R& hx, R& hy, R& hz) {
   constexpr bool COMPACT = FMT == FMT_DMI_TAB && sizeof(R) == 4;
   const uint32_t mask = COMPACT ? (1u << a.crec_shift) - 1u : (uint32_t)a.idx_mask;
   for (int k0 = 0; k0 < r.w; k0 += W) {
      uint32_t c[W], p[W];
      unsigned real = 0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
         c[k] = 0;
         p[k] = self;
         if (k0 + k < r.w) {  // the same for the whole warp
            if constexpr (res_words<R, FMT>()) c[k] = r.w0[32 * (k0 + k)];
            else c[k] = (uint32_t)__ldg(a.col + r.base + 32 * (k0 + k));
            const uint32_t j = c[k] & mask;
            if (j < (uint32_t)a.n) {
               real |= 1u << k;
               p[k] = 16u * j;
            }
         }
      }
      ResSpin<R> s[W];
      if (!res_read<R, W>(X, plane, p, t, s)) return false;
#pragma unroll
      for (int k = 0; k < W; ++k)
         if ((real >> k) & 1u)
            res_bond<R, FMT>(a, r, k0 + k, res_coupling<R, FMT>(a, c[k]), s[k].x(), s[k].y(), s[k].z(), hx, hy, hz);
   }
   return true;
}

// shared memory: slice offsets, materials, dictionary, words
struct ResLayout {
   int mats, dict, words, bytes;
};
template <typename R>
__host__ __device__ inline ResLayout res_layout(int K, int M, int dict_bytes, int word_bytes) {
   ResLayout l;
   l.mats = ((kResSlices * K + 1 + 3) & ~3) * 4;
   l.dict = (l.mats + (M <= kResMaxMat ? M * (int)sizeof(MatParams<R>) : 0) + 15) & ~15;
   l.words = l.dict + dict_bytes;
   l.bytes = l.words + word_bytes;
   return l;
}

// blocks per SM that the registers are capped for: as many resident atoms as
// the gather's loads in flight allow without spilling much
template <typename R, int FMT, int VAR, int K> constexpr int res_min_blocks() {
   if (sizeof(R) == 8) return 3;
   if (FMT == FMT_DMI_TAB) return 4;
   if (FMT == FMT_ISO_TAB && VAR == VAR_HEUN) return K == 1 ? 6 : K == 2 ? 5 : 4;
   return 6;
}

// What a block of kResBlock threads with one atom each keeps in shared memory,
// filled by the constructor (ends with a block barrier).
template <typename R, int FMT> struct ResBlockData {
   int o0;
   bool one_j;
   const int* off;
   const MatParams<R>* mats;
   const float4* dict;
   const uint32_t* words;
   __device__ ResBlockData(const LLGArgs<R>& a, unsigned char* smem, int nslices, int word_bytes) {
      constexpr bool WORDS = res_words<R, FMT>();
      const int dict_bytes = WORDS && FMT == FMT_DMI_TAB ? 16 * (a.tab_scalar ? a.cdict_n : 2 * a.cdict_n) : 0;
      const ResLayout lay = res_layout<R>(1, a.M, dict_bytes, word_bytes);
      int* s_off = reinterpret_cast<int*>(smem);
      MatParams<R>* s_mat = reinterpret_cast<MatParams<R>*>(smem + lay.mats);
      float4* s_dict = reinterpret_cast<float4*>(smem + lay.dict);
      uint32_t* s_words = reinterpret_cast<uint32_t*>(smem + lay.words);
      const int tid = threadIdx.x, s0 = blockIdx.x * kResSlices, ns = min(kResSlices, nslices - s0);
      o0 = __ldg(a.slice_off + s0);
      one_j = a.M == 1 || (a.sys_off && a.m_per_sys == 1);
      if (WORDS) {
         const int nw = __ldg(a.slice_off + s0 + ns) - o0;
         const uint32_t* src = FMT == FMT_ISO_TAB ? reinterpret_cast<const uint32_t*>(a.col) : a.crec;
         for (int q = tid; q < nw; q += kResBlock) s_words[q] = __ldg(src + o0 + q);
         for (int q = tid; q < dict_bytes / 16; q += kResBlock) s_dict[q] = __ldg(a.cdict + q);
      }
      for (int q = tid; q <= kResSlices; q += kResBlock) s_off[q] = __ldg(a.slice_off + s0 + min(q, ns)) - o0;
      if (a.M <= kResMaxMat) {
         const int nw = a.M * (int)(sizeof(MatParams<R>) / 4);
         for (int q = tid; q < nw; q += kResBlock)
            reinterpret_cast<uint32_t*>(s_mat)[q] = __ldg(reinterpret_cast<const uint32_t*>(a.mp) + q);
      }
      off = s_off;
      mats = a.M <= kResMaxMat ? s_mat : a.mp;
      dict = s_dict;
      words = s_words;
      __syncthreads();
   }
   __device__ const MatParams<R>& mat(const LLGArgs<R>&, int mi) const { return mats[mi]; }
   // the row of this thread's atom (i: the atom, 0 for a thread past the last)
   __device__ ResRow<R> row(const LLGArgs<R>& a, int i) const {
      const int sl = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int mi = a.mat ? __ldg(a.mat + i) : 0;
      return ResRow<R>{o0 + off[sl] + lane, (off[sl + 1] - off[sl]) >> 5, words + off[sl] + lane, mi, one_j,
                       FMT == FMT_ISO_TAB ? __ldg(a.jtab + mi * a.M + mi) : (R)0, dict};
   }
};

// RF for formats other than FMT_ISO_TAB: the common facts written in -- thermal
// noise from Philox, one system, no field per material, no host dipole field, a
// scalar coupling table in the dictionary (FP32 DMI)
constexpr int kResCommon = 1;
template <typename R> inline int common_features(const LLGArgs<R>& a, int fmt, int var) {
   const bool ok = var == VAR_HEUN && a.thermal && a.noise_mode == VGPU_NOISE_PHILOX && !a.sys_off && !a.ramp_n &&
                   !a.local_field && !a.hd_atom && !(sizeof(R) == 4 && a.ex) &&
                   !(fmt == FMT_DMI_TAB && sizeof(R) == 4 && !a.tab_scalar);
   return ok ? kResCommon : 0;
}
template <typename R, int FMT, int RF> __device__ __forceinline__ LLGArgs<R> res_fold(const LLGArgs<R>& in) {
   if (FMT == FMT_ISO_TAB) return fold_iso<R, RF>(in);
   LLGArgs<R> a = in;
   if (RF == kResCommon) {
      a.thermal = 1;
      a.noise_mode = VGPU_NOISE_PHILOX;
      a.sys_off = nullptr;
      a.ramp_n = 0;
      a.local_field = 0;
      a.hd_atom = nullptr;
      if (sizeof(R) == 4) a.ex = a.ey = a.ez = nullptr;
      if (FMT == FMT_DMI_TAB && sizeof(R) == 4) a.tab_scalar = 1;
   }
   return a;
}

// XA, XB: the tagged spins and predictor states of all threads' atoms (`plane`
// bytes per word of a spin)
template <typename R, int FMT, int VAR, int K, int RF>
__global__ void __launch_bounds__(kResBlock, (res_min_blocks<R, FMT, VAR, K>()))
    llg_resident_kernel(const LLGArgs<R> in, int nsteps, char* XA, char* XB, uint32_t plane, uint32_t epoch0,
                        int nslices, int word_bytes) {
   LLGArgs<R> a = res_fold<R, FMT, RF>(in);
   constexpr bool WORDS = res_words<R, FMT>();
   constexpr bool FIXED = FMT == FMT_ISO_TAB && (RF & ISO_FIXED) != 0;
   extern __shared__ __align__(16) unsigned char res_smem[];
   const int dict_bytes = WORDS && FMT == FMT_DMI_TAB ? 16 * (a.tab_scalar ? a.cdict_n : 2 * a.cdict_n) : 0;
   const ResLayout lay = res_layout<R>(K, a.M, dict_bytes, word_bytes);
   int* s_off = reinterpret_cast<int*>(res_smem);
   MatParams<R>* s_mat = reinterpret_cast<MatParams<R>*>(res_smem + lay.mats);
   float4* s_dict = reinterpret_cast<float4*>(res_smem + lay.dict);
   uint32_t* s_words = reinterpret_cast<uint32_t*>(res_smem + lay.words);
   const int tid = threadIdx.x, blk = blockIdx.x;
   // one coupling per atom: one material, or batched systems of one material
   const bool one_j = FIXED || a.M == 1 || (a.sys_off && a.m_per_sys == 1);
   R S0[K][3], P[K][3], E[K][3], j0[K];
   int mi[K];
#pragma unroll
   for (int k = 0; k < K; ++k) {
      const int i = (blk * K + k) * kResBlock + tid;
      mi[k] = 0;
      j0[k] = 0;
      S0[k][0] = 1; S0[k][1] = 0; S0[k][2] = 0;  // threads past the last atom: a spin nobody reads
      if (i < a.n_upd) {
         mi[k] = a.mat ? __ldg(a.mat + i) : 0;
         if (FMT == FMT_ISO_TAB) j0[k] = __ldg(a.jtab + mi[k] * a.M + mi[k]);
         S0[k][0] = a.ax[i]; S0[k][1] = a.ay[i]; S0[k][2] = a.az[i];
      }
      P[k][0] = S0[k][0]; P[k][1] = S0[k][1]; P[k][2] = S0[k][2];
      ResSpin<R>::store(XA, plane, 16u * (uint32_t)i, S0[k], a.wait_test ? epoch0 - 1 : epoch0);
   }
   const int s0 = blk * kResSlices * K, ns = min(kResSlices * K, nslices - s0);
   const int o0 = __ldg(a.slice_off + s0);
   if constexpr (WORDS) {
      const int nw = __ldg(a.slice_off + s0 + ns) - o0;
      const uint32_t* src = FMT == FMT_ISO_TAB ? reinterpret_cast<const uint32_t*>(a.col) : a.crec;
      for (int q = tid; q < nw; q += kResBlock) s_words[q] = __ldg(src + o0 + q);
      for (int q = tid; q < dict_bytes / 16; q += kResBlock) s_dict[q] = __ldg(a.cdict + q);
   }
   for (int q = tid; q <= kResSlices * K; q += kResBlock) s_off[q] = __ldg(a.slice_off + s0 + min(q, ns)) - o0;
   if (a.M <= kResMaxMat) {
      const int nw = a.M * (int)(sizeof(MatParams<R>) / 4);
      for (int q = tid; q < nw; q += kResBlock)
         reinterpret_cast<uint32_t*>(s_mat)[q] = __ldg(reinterpret_cast<const uint32_t*>(a.mp) + q);
   }
   const MatParams<R>* mpt = a.M <= kResMaxMat ? s_mat : a.mp;
   __syncthreads();  // the last one: the steps order themselves by the tags
   // FIXED, one atom per thread: the offsets of its six neighbours
   constexpr bool REGS = FIXED && K <= 2;
   uint32_t nb[REGS ? K : 1][6];
   unsigned real[REGS ? K : 1];
   bool six = false;
   if constexpr (REGS) {
      six = true;
#pragma unroll
      for (int k = 0; k < K; ++k) {
         const int sl = kResSlices * k + (tid >> 5), i = (blk * K + k) * kResBlock + tid;
         const int off = s_off[sl], w = (s_off[sl + 1] - off) >> 5;
         real[k] = 0;
         six = six && w <= 6;
#pragma unroll
         for (int q = 0; q < 6; ++q) {
            nb[k][q] = 16u * (uint32_t)i;
            if (q < w) {
               const uint32_t j = s_words[off + (tid & 31) + 32 * q] & (uint32_t)a.idx_mask;
               if (j < (uint32_t)a.n) {
                  real[k] |= 1u << q;
                  nb[k][q] = 16u * j;
               }
            }
         }
      }
   }
   const uint64_t step0 = a.step;
   auto field = [&](int k, int i, bool on, const char* X, uint32_t t, const R S[3], R H[3]) -> bool {
      R hx = 0, hy = 0, hz = 0;
      bool ok;
      if (REGS && six) {
         const int kk = REGS ? k : 0;
         ResSpin<R> s[6];
         ok = res_read<R, 6>(X, plane, nb[kk], t, s);
#pragma unroll
         for (int q = 0; q < 6; ++q)
            if ((real[kk] >> q) & 1u) { hx += j0[k] * s[q].x(); hy += j0[k] * s[q].y(); hz += j0[k] * s[q].z(); }
      } else {
         const int sl = kResSlices * k + (tid >> 5);
         const int off = s_off[sl];
         const ResRow<R> r{o0 + off + (tid & 31), (s_off[sl + 1] - off) >> 5, s_words + off + (tid & 31), mi[k], one_j,
                           j0[k], s_dict};
         const uint32_t self = 16u * (uint32_t)i;
         if constexpr (FMT == FMT_DMI_TAB && sizeof(R) == 4) {
            // FCC rows: one round trip for all 12 neighbours
            if (r.w == 12) ok = res_gather<R, FMT, 12>(a, r, X, plane, self, t, hx, hy, hz);
            else ok = res_gather<R, FMT, 6>(a, r, X, plane, self, t, hx, hy, hz);
         } else {
            ok = res_gather<R, FMT, 6>(a, r, X, plane, self, t, hx, hy, hz);
         }
      }
      if (ok && on) {
         site_field<R, 0, VAR != VAR_HEUN>(a, i, mpt[mi[k]], nullptr, nullptr, nullptr, S, hx, hy, hz, H);
         H[0] += E[k][0]; H[1] += E[k][1]; H[2] += E[k][2];
      }
      return ok;
   };
   bool ok = true;
   for (int s = 0; s < nsteps && ok; ++s) {
      a.step = step0 + (uint64_t)s;
      set_ramp(a);
      const uint32_t e = epoch0 + 2 * (uint32_t)s;
#pragma unroll
      for (int k = 0; k < K; ++k) {
         const int i = (blk * K + k) * kResBlock + tid;
         if (i < a.n_upd) external_field<R>(a, i, mpt[mi[k]], true, E[k]);
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
         const int i = (blk * K + k) * kResBlock + tid;
         const bool on = i < a.n_upd;
         R H[3];
         ok = ok && field(k, i, on, XA, e, S0[k], H);
         if (ok) {
            if (on) first_half<R, VAR>(a, i, mpt[mi[k]], S0[k], H, P[k]);
            ResSpin<R>::store(XB, plane, 16u * (uint32_t)i, P[k], e + 1);
         }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
         const int i = (blk * K + k) * kResBlock + tid;
         const bool on = i < a.n_upd;
         R H[3], o[3];
         ok = ok && field(k, i, on, XB, e + 1, P[k], H);
         if (ok) {
            if (on) {
               second_half<R, VAR>(a, i, mpt[mi[k]], S0[k], P[k], H, o);
               S0[k][0] = o[0]; S0[k][1] = o[1]; S0[k][2] = o[2];
            }
            ResSpin<R>::store(XA, plane, 16u * (uint32_t)i, S0[k], e + 2);
         }
      }
   }
   if (!ok) {
      if ((tid & 31) == 0) atomicOr(a.status, 2);
      return;
   }
#pragma unroll
   for (int k = 0; k < K; ++k) {
      const int i = (blk * K + k) * kResBlock + tid;
      if (i < a.n_upd) {
         a.ax[i] = S0[k][0]; a.ay[i] = S0[k][1]; a.az[i] = S0[k][2];
         a.bx[i] = P[k][0]; a.by[i] = P[k][1]; a.bz[i] = P[k][2];
      }
   }
}

// Deterministic Heun steps that also leave a trace, for the adjoint: the state
// after each step (traj, 3 stride values a step) or each warp's sum of mu s_z
// (mz, [nsteps][warps]), in FP64.  Starts from, and ends in, the state x of 3
// stride values; inc (3 stride) takes the predictor increments.  The step is
// llg_resident_kernel's with one atom per thread.
template <typename R, int FMT>
__global__ void __launch_bounds__(kResBlock, (res_min_blocks<R, FMT, VAR_HEUN_EXT, 1>()))
    llg_path_kernel(const LLGArgs<R> in, int nsteps, char* XA, char* XB, uint32_t plane, uint32_t epoch0, int nslices,
                    int word_bytes, R* x, R* inc, int stride, R* traj, double* mz) {
   LLGArgs<R> a = in;
   a.thermal = 0;
   a.ex = inc; a.ey = inc + stride; a.ez = inc + 2 * stride;
   extern __shared__ __align__(16) unsigned char res_smem[];
   const ResBlockData<R, FMT> d(a, res_smem, nslices, word_bytes);
   const int i = blockIdx.x * kResBlock + threadIdx.x;
   const bool on = i < a.n;
   const uint32_t self = 16u * (uint32_t)i;
   R S0[3] = {1, 0, 0}, P[3] = {1, 0, 0}, E[3] = {0, 0, 0};
   const ResRow<R> r = d.row(a, on ? i : 0);
   if (on) {
      for (int c = 0; c < 3; ++c) S0[c] = x[(size_t)c * stride + i];
      external_field<R>(a, i, d.mat(a, r.mi), false, E);
   }
   ResSpin<R>::store(XA, plane, self, S0, a.wait_test ? epoch0 - 1 : epoch0);
   auto field = [&](const char* X, uint32_t t, const R S[3], R H[3]) -> bool {
      R hx = 0, hy = 0, hz = 0;
      if (!res_gather<R, FMT, 6>(a, r, X, plane, self, t, hx, hy, hz)) return false;
      site_field<R, 0, false>(a, i, d.mat(a, r.mi), nullptr, nullptr, nullptr, S, hx, hy, hz, H);
      H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
      return true;
   };
   bool ok = true;
   for (int s = 0; s < nsteps && ok; ++s) {
      const uint32_t e = epoch0 + 2 * (uint32_t)s;
      R H[3], o[3];
      ok = field(XA, e, S0, H);
      if (!ok) break;
      if (on) llg_predict<R>(a, i, d.mat(a, r.mi), S0, H, P);
      ResSpin<R>::store(XB, plane, self, P, e + 1);
      ok = field(XB, e + 1, P, H);
      if (!ok) break;
      if (on) {
         llg_correct<R>(a, i, d.mat(a, r.mi), S0, P, H, o);
         S0[0] = o[0]; S0[1] = o[1]; S0[2] = o[2];
      }
      ResSpin<R>::store(XA, plane, self, S0, e + 2);
      if (traj && on)
         for (int c = 0; c < 3; ++c) traj[(3 * (size_t)s + c) * stride + i] = S0[c];
      if (mz) {
         double v = on ? (double)S0[2] * (double)d.mat(a, r.mi).mu_s_muB : 0.0;
         for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
         const int warps = gridDim.x * (kResBlock / 32);
         if ((threadIdx.x & 31) == 0) mz[(size_t)s * warps + (i >> 5)] = v;
      }
   }
   if (!ok) {
      if ((threadIdx.x & 31) == 0) atomicOr(a.status, 2);
      return;
   }
   if (on)
      for (int c = 0; c < 3; ++c) x[(size_t)c * stride + i] = S0[c];
}

// every bond i -> j has a bond j -> i (*bad set otherwise)
template <typename R>
__global__ void res_mutual_kernel(const LLGArgs<R> a, int* bad) {
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= a.n) return;
   const int off = a.slice_off[i >> 5], w = (a.slice_off[(i >> 5) + 1] - off) >> 5;
   for (int k = 0; k < w; ++k) {
      const int j = a.col[off + (i & 31) + 32 * k] & a.idx_mask;
      if (j >= a.n) continue;  // padding entry
      const int offj = a.slice_off[j >> 5], wj = (a.slice_off[(j >> 5) + 1] - offj) >> 5;
      bool found = false;
      for (int q = 0; q < wj && !found; ++q) found = (a.col[offj + (j & 31) + 32 * q] & a.idx_mask) == i;
      if (!found) *bad = 1;
   }
}

// dynamic shared memory beyond what every kernel may take (few kernels' static
// kilobyte counts against it: asked for from 40 KB)
template <typename F> inline cudaError_t allow_smem(F* f, int smem) {
   if (smem <= 40 * 1024) return cudaSuccess;
   return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kStageSmemLimit);
}

template <typename R> using ResidentFn = void (*)(LLGArgs<R>, int, char*, char*, uint32_t, uint32_t, int, int);

// the kernel of a format, variant, number of atoms per thread and feature set
// (nullptr: none; several atoms per thread are compiled for the two common
// formats)
template <typename R, int FMT, int K>
inline ResidentFn<R> resident_heun(int feat) {
   if constexpr (FMT == FMT_ISO_TAB) {
      switch (feat) {
#define VGPU_F(k) \
   case k: return llg_resident_kernel<R, FMT, VAR_HEUN, K, k>;
         VGPU_ISO_FEATURES(VGPU_F)
#undef VGPU_F
      }
   } else if (feat == kResCommon) {
      return llg_resident_kernel<R, FMT, VAR_HEUN, K, kResCommon>;
   }
   return llg_resident_kernel<R, FMT, VAR_HEUN, K, 0>;
}

// the feature set of a launch
template <typename R> inline int resident_features(const LLGArgs<R>& a, int fmt, int var) {
   return fmt == FMT_ISO_TAB ? iso_features<R>(a, fmt, var) : common_features<R>(a, fmt, var);
}

template <typename R, int FMT>
inline ResidentFn<R> resident_fmt(int var, int K, int feat) {
   if (var == VAR_HEUN) {
      if (K == 1) return resident_heun<R, FMT, 1>(feat);
      if constexpr (res_words<R, FMT>()) {
         if (K == 2) return resident_heun<R, FMT, 2>(feat);
         if (K == 4) return resident_heun<R, FMT, 4>(feat);
      }
      return nullptr;
   }
   if (K != 1) return nullptr;
   if (var == VAR_HEUN_EXT) return llg_resident_kernel<R, FMT, VAR_HEUN_EXT, 1, 0>;
   return llg_resident_kernel<R, FMT, VAR_MIDPOINT, 1, 0>;
}

template <typename R>
inline ResidentFn<R> resident_fn(int fmt, int var, int K, int feat) {
   switch (fmt) {
      case FMT_ISO_TAB: return resident_fmt<R, FMT_ISO_TAB>(var, K, feat);
      case FMT_ISO_BOND: return resident_fmt<R, FMT_ISO_BOND>(var, K, feat);
      case FMT_VEC_TAB: return resident_fmt<R, FMT_VEC_TAB>(var, K, feat);
      case FMT_VEC_BOND: return resident_fmt<R, FMT_VEC_BOND>(var, K, feat);
      case FMT_DMI_TAB: return resident_fmt<R, FMT_DMI_TAB>(var, K, feat);
      default: return resident_fmt<R, FMT_TENSOR_BOND>(var, K, feat);
   }
}

// dynamic shared memory of a plan
template <typename R>
static int resident_smem(const LLGArgs<R>& a, int fmt, const ResidentPlan& p) {
   const bool words = fmt == FMT_ISO_TAB || (fmt == FMT_DMI_TAB && sizeof(R) == 4);
   const int dict = words && fmt == FMT_DMI_TAB ? 16 * (a.tab_scalar ? a.cdict_n : 2 * a.cdict_n) : 0;
   return res_layout<R>(p.K, a.M, dict, words ? p.word_bytes : 0).bytes;
}

template <typename R>
cudaError_t resident_capacity(const LLGArgs<R>& a, int fmt, int var, const ResidentPlan& p, int sms, int* blocks) {
   *blocks = 0;
   const int smem = resident_smem<R>(a, fmt, p);
   if (!resident_fn<R>(fmt, var, p.K, 0) || smem > kStageSmemLimit) return cudaSuccess;
   std::vector<int> feats{0};  // whatever the parameters turn out to be: the least over the compiled features
   if (fmt == FMT_ISO_TAB && var == VAR_HEUN) {
#define VGPU_F(k) feats.push_back(k);
      VGPU_ISO_FEATURES(VGPU_F)
#undef VGPU_F
   } else if (var == VAR_HEUN) {
      feats.push_back(kResCommon);
   }
   int least = 1 << 30;
   for (int feat : feats) {
      const ResidentFn<R> f = resident_fn<R>(fmt, var, p.K, feat);
      cudaError_t e = allow_smem(f, smem);
      int per_sm = 0;
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kResBlock, smem);
      if (e != cudaSuccess) return e;
      least = std::min(least, per_sm * sms);
   }
   *blocks = least;
   return cudaSuccess;
}

// cooperative launch of a kernel of one atom per thread (p.K == 1)
template <typename R, typename... Args>
inline cudaError_t launch_one_atom(void (*f)(Args...), const LLGArgs<R>& a, int fmt, const ResidentPlan& p,
                                   cudaStream_t st, Args... args) {
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(p.grid);
   cfg.blockDim = dim3(kResBlock);
   cfg.dynamicSmemBytes = (size_t)resident_smem<R>(a, fmt, p);
   cfg.stream = st;
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeCooperative;
   attr[0].val.cooperative = 1;
   cfg.attrs = attr;
   cfg.numAttrs = 1;
   return cudaLaunchKernelEx(&cfg, f, args...);
}

// whether a kernel of one atom per thread is resident with the plan's grid
template <typename R, typename F>
inline cudaError_t one_atom_fits(F* f, const LLGArgs<R>& a, int fmt, const ResidentPlan& p, int device, bool* fits) {
   *fits = false;
   const int smem = resident_smem<R>(a, fmt, p);
   int sms = 0, per_sm = 0;
   cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
   if (e == cudaSuccess) e = allow_smem(f, smem);
   if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kResBlock, smem);
   *fits = per_sm * sms >= p.grid;
   return e;
}

template <typename R> using PathFn = void (*)(LLGArgs<R>, int, char*, char*, uint32_t, uint32_t, int, int, R*, R*, int,
                                             R*, double*);
template <typename R> inline PathFn<R> path_fn(int fmt) {
   switch (fmt) {
      case FMT_ISO_TAB: return llg_path_kernel<R, FMT_ISO_TAB>;
      case FMT_ISO_BOND: return llg_path_kernel<R, FMT_ISO_BOND>;
      case FMT_VEC_TAB: return llg_path_kernel<R, FMT_VEC_TAB>;
      case FMT_VEC_BOND: return llg_path_kernel<R, FMT_VEC_BOND>;
      case FMT_DMI_TAB: return llg_path_kernel<R, FMT_DMI_TAB>;
      default: return llg_path_kernel<R, FMT_TENSOR_BOND>;
   }
}

template <typename R>
cudaError_t path_fits(const LLGArgs<R>& a, int fmt, const ResidentPlan& p, int device, bool* fits) {
   return one_atom_fits<R>(path_fn<R>(fmt), a, fmt, p, device, fits);
}

template <typename R>
cudaError_t launch_llg_path(const LLGArgs<R>& a, int fmt, int nsteps, const ResidentPlan& p, int nslices, R* x, R* inc,
                            int stride, R* traj, double* mz, cudaStream_t st) {
   char* X = static_cast<char*>(p.spins);
   const uint32_t plane = 16u * (uint32_t)(p.grid * kResBlock);
   return launch_one_atom<R>(path_fn<R>(fmt), a, fmt, p, st, LLGArgs<R>(a), nsteps, X,
                             X + (size_t)ResSpin<R>::kWords * plane, plane, p.epoch, nslices, p.word_bytes, x, inc,
                             stride, traj, mz);
}

template <typename R>
cudaError_t launch_resident_check(const LLGArgs<R>& a, int* bad, cudaStream_t st) {
   res_mutual_kernel<R><<<(a.n + 255) / 256, 256, 0, st>>>(a, bad);
   return cudaGetLastError();
}

template <typename R>
cudaError_t launch_llg_resident(const LLGArgs<R>& a, int fmt, int var, int nsteps, const ResidentPlan& p, int nslices,
                                cudaStream_t st) {
   const ResidentFn<R> f = resident_fn<R>(fmt, var, p.K, resident_features<R>(a, fmt, var));
   if (!f) return cudaErrorInvalidValue;
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(p.grid);
   cfg.blockDim = dim3(kResBlock);
   cfg.dynamicSmemBytes = (size_t)resident_smem<R>(a, fmt, p);
   cfg.stream = st;
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeCooperative;  // every block resident: threads wait on one another's spins
   attr[0].val.cooperative = 1;
   cfg.attrs = attr;
   cfg.numAttrs = 1;
   char* X = static_cast<char*>(p.spins);
   const uint32_t plane = 16u * (uint32_t)(p.grid * p.K * kResBlock);
   return cudaLaunchKernelEx(&cfg, f, a, nsteps, X, X + (size_t)ResSpin<R>::kWords * plane, plane, p.epoch, nslices,
                             p.word_bytes);
}

}  // namespace vgpu

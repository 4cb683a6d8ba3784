// Many LLG steps of a small system in one launch: FP32 systems of isotropic bonds
// with at most 2,048 atoms, on one thread-block cluster, the states in its
// distributed shared memory.
//
// A small system lives on a few SMs of one GPC, so its spins need not travel
// through L2 (llg_resident.cuh): each block keeps its atoms' spins and predictor
// states in shared memory, neighbours are read from the block that has them, and
// the half-steps are separated by the cluster's hardware barrier (arrive after the
// store, the next noise drawn, then wait).  Microseconds a step against the tagged
// spins in L2: 125 atoms 1.05 and 1.51, 990 atoms 1.49 and 2.02, 2,016 atoms 1.83
// and 2.03; from 4,096 atoms the reads between SMs cost more than L2 (2.24 and
// 1.97; 8,000 atoms 3.41 and 2.15), and FP64 gains nothing (990 atoms 3.4 and
// 2.8), so those run there.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "llg_resident.cuh"

namespace vgpu {

namespace {

__device__ __forceinline__ unsigned cluster_rank() {
   unsigned r;
   asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
   return r;
}
__device__ __forceinline__ void cluster_arrive() {
   asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// address of `slot` of the spin array at shared address `arr` in block `rank`
// of the cluster, and the spin at such an address
__device__ __forceinline__ uint32_t spin_address(uint32_t arr, uint32_t rank, uint32_t slot) {
   uint32_t p;
   asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(arr), "r"(rank));
   return p + (uint32_t)sizeof(float4) * slot;
}
__device__ __forceinline__ float4 spin_at(uint32_t p) {
   float4 v;
   asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p));
   return v;
}

// the spin at p, in this block's own shared memory (`own`: a plain shared-memory
// address) or in another block's.  The path between SMs is the narrow one, and
// own neighbours are most.
__device__ __forceinline__ float4 spin_near(uint32_t p, bool own) {
   float4 v;
   asm volatile(
       "{\n .reg .pred o;\n setp.ne.u32 o, %5, 0;\n"
       " @o ld.shared::cta.v4.f32 {%0, %1, %2, %3}, [%4];\n"
       " @!o ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
       : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
       : "r"(p), "r"((uint32_t)own));
   return v;
}

// bond words: block << 12 | slot (the slot after the last thread's: the zero spin
// that padded bonds read), the neighbour's material << 16
constexpr int kClusterBlock = kClusterAtoms / 16;
constexpr uint32_t kSlotBits = 12, kSlotMask = (1u << kSlotBits) - 1u;
constexpr int kClusterWidth = 6;  // loads in flight

// shared memory: spins, predictor states, materials, words
struct ClusterLayout {
   int mats, words, bytes;
};
__host__ __device__ inline ClusterLayout cluster_layout(int threads, int zmax, int M) {
   ClusterLayout l;
   l.mats = 2 * (threads + 1) * (int)sizeof(float4);
   l.words = (l.mats + (M <= kResMaxMat ? M * (int)sizeof(MatParams<float>) : 0) + 15) & ~15;
   l.bytes = l.words + 4 * threads * zmax;
   return l;
}

// nsteps steps of all atoms, one per thread, in order over the blocks of one
// cluster.  zmax: bonds of the widest row.
template <int VAR, int RF>
__global__ void __launch_bounds__(kClusterBlock) llg_cluster_kernel(const LLGArgs<float> in, int nsteps, int zmax) {
   LLGArgs<float> a = fold_iso<float, RF>(in);
   extern __shared__ __align__(16) unsigned char res_smem[];
   const int T = blockDim.x, tid = threadIdx.x;
   const ClusterLayout lay = cluster_layout(T, zmax, a.M);
   float4* sA = reinterpret_cast<float4*>(res_smem);
   float4* sB = sA + T + 1;
   MatParams<float>* s_mat = reinterpret_cast<MatParams<float>*>(res_smem + lay.mats);
   uint32_t* s_words = reinterpret_cast<uint32_t*>(res_smem + lay.words);
   const uint32_t rank = cluster_rank();
   const int i = (int)rank * T + tid;
   const bool on = i < a.n_upd;
   const bool one_j = (RF & ISO_FIXED) != 0 || a.M == 1 || (a.sys_off && a.m_per_sys == 1);
   ResRow<float> row{0, 0, nullptr, 0, one_j, 0.f, nullptr};
   float S0[3] = {0, 0, 0}, P[3] = {0, 0, 0}, E[3] = {0, 0, 0};
   const uint32_t zero_word = (rank << kSlotBits) | (uint32_t)T;
   if (on) {
      const int off = __ldg(a.slice_off + (i >> 5));
      row.base = off + (i & 31);
      row.w = (__ldg(a.slice_off + (i >> 5) + 1) - off) >> 5;
      row.mi = a.mat ? __ldg(a.mat + i) : 0;
      row.j0 = __ldg(a.jtab + row.mi * a.M + row.mi);
      for (int k = 0; k < row.w; ++k) {
         const uint32_t c = (uint32_t)__ldg(a.col + row.base + 32 * k);
         const int j = (int)(c & (uint32_t)a.idx_mask);
         const uint32_t q = one_j ? 0u : res_coupling<float, FMT_ISO_TAB>(a, c);
         uint32_t wd = zero_word;
         if (j < a.n) wd = ((uint32_t)(j / T) << kSlotBits) | (uint32_t)(j % T);
         s_words[k * T + tid] = wd | (q << 16);
      }
   }
   if (tid == 0) sA[T] = sB[T] = make_float4(0.f, 0.f, 0.f, 0.f);
   if (a.M <= kResMaxMat) {
      const int nw = a.M * (int)(sizeof(MatParams<float>) / 4);
      for (int q = tid; q < nw; q += T)
         reinterpret_cast<uint32_t*>(s_mat)[q] = __ldg(reinterpret_cast<const uint32_t*>(a.mp) + q);
   }
   const uint32_t arrA = (uint32_t)__cvta_generic_to_shared(sA), dB = (uint32_t)((T + 1) * (int)sizeof(float4));
   __syncthreads();  // materials in place
   const MatParams<float> m = a.M <= kResMaxMat ? s_mat[row.mi] : a.mp[row.mi];
   if (a.sys_off && on) {
      // the stream and atom numbering of this system (thermal_xi), once
      const int k = row.mi / a.m_per_sys;
      const uint64_t seed = (((uint64_t)a.seed_hi << 32) | a.seed_lo) + (uint64_t)k;
      a.noise_base = 0u - (uint32_t)__ldg(a.sys_off + k);
      a.seed_lo = (uint32_t)seed;
      a.seed_hi = (uint32_t)(seed >> 32);
   }
   a.sys_off = nullptr;
   // ISO_FIXED: the addresses of the six neighbours (rows of fewer: the zero slot)
   uint32_t nb[6], own = 0;
   if constexpr ((RF & ISO_FIXED) != 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
         const uint32_t c = k < row.w ? s_words[k * T + tid] : zero_word;
         const uint32_t r = (c >> kSlotBits) & 15u;
         if (r == rank) own |= 1u << k;
         nb[k] = r == rank ? arrA + (uint32_t)sizeof(float4) * (c & kSlotMask) : spin_address(arrA, r, c & kSlotMask);
      }
   }
   // everything above is as the upload or a copy on the stream left it; the spins
   // and the dipole field are the previous kernel's
   pdl_begin();
   asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
   if (on) { S0[0] = a.ax[i]; S0[1] = a.ay[i]; S0[2] = a.az[i]; }
   sA[tid] = make_float4(S0[0], S0[1], S0[2], 0.f);
   cluster_arrive();
   const uint64_t step0 = a.step;
   // d: 0 for the spins, dB for the predictor states
   auto field = [&](uint32_t d, const float S[3], float H[3]) {
      float hx = 0, hy = 0, hz = 0;
      if constexpr ((RF & ISO_FIXED) != 0) {
         float4 s[6];
#pragma unroll
         for (int k = 0; k < 6; ++k) s[k] = spin_near(nb[k] + d, (own >> k) & 1u);
#pragma unroll
         for (int k = 0; k < 6; ++k) { hx += row.j0 * s[k].x; hy += row.j0 * s[k].y; hz += row.j0 * s[k].z; }
      } else {
         constexpr int W = kClusterWidth;
         for (int k0 = 0; k0 < row.w; k0 += W) {
            uint32_t c[W];
            float4 s[W];
#pragma unroll
            for (int k = 0; k < W; ++k) c[k] = k0 + k < row.w ? s_words[(k0 + k) * T + tid] : zero_word;
#pragma unroll
            for (int k = 0; k < W; ++k) s[k] = spin_at(spin_address(arrA, (c[k] >> kSlotBits) & 15u, c[k] & kSlotMask) + d);
#pragma unroll
            for (int k = 0; k < W; ++k)
               if (k0 + k < row.w)
                  res_bond<float, FMT_ISO_TAB>(a, row, k0 + k, c[k] >> 16, s[k].x, s[k].y, s[k].z, hx, hy, hz);
         }
      }
      site_field<float, 0, VAR != VAR_HEUN>(a, i, m, nullptr, nullptr, nullptr, S, hx, hy, hz, H);
      H[0] += E[0]; H[1] += E[1]; H[2] += E[2];
   };
   for (int s = 0; s < nsteps; ++s) {
      a.step = step0 + (uint64_t)s;
      set_ramp(a);
      if (on) external_field<float>(a, i, m, true, E);
      cluster_wait();  // every block's spins of this step in place
      if (on) {
         float H[3];
         field(0, S0, H);
         first_half<float, VAR>(a, i, m, S0, H, P);
         sB[tid] = make_float4(P[0], P[1], P[2], 0.f);
      }
      cluster_arrive();
      cluster_wait();  // every predictor state in place, every read of the spins done
      if (on) {
         float H[3], o[3];
         field(dB, P, H);
         second_half<float, VAR>(a, i, m, S0, P, H, o);
         S0[0] = o[0]; S0[1] = o[1]; S0[2] = o[2];
         sA[tid] = make_float4(o[0], o[1], o[2], 0.f);
      }
      cluster_arrive();
   }
   if (on) {
      a.ax[i] = S0[0]; a.ay[i] = S0[1]; a.az[i] = S0[2];
      a.bx[i] = P[0]; a.by[i] = P[1]; a.bz[i] = P[2];
   }
   cluster_wait();  // no block leaves while its shared memory is read
}

// the kernel of a variant and feature set
using ClusterFn = void (*)(LLGArgs<float>, int, int);
ClusterFn cluster_fn(int var, int feat) {
   switch (feat) {
#define VGPU_F(k) \
   case k: return llg_cluster_kernel<VAR_HEUN, k>;
      VGPU_ISO_FEATURES(VGPU_F)
#undef VGPU_F
   }
   if (var == VAR_HEUN) return llg_cluster_kernel<VAR_HEUN, 0>;
   if (var == VAR_HEUN_EXT) return llg_cluster_kernel<VAR_HEUN_EXT, 0>;
   return llg_cluster_kernel<VAR_MIDPOINT, 0>;
}

void cluster_config(const LLGArgs<float>& a, const ClusterShape& c, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
   *cfg = cudaLaunchConfig_t{};
   cfg->gridDim = dim3(c.size);
   cfg->blockDim = dim3(c.threads);
   cfg->dynamicSmemBytes = (size_t)cluster_layout(c.threads, c.zmax, a.M).bytes;
   attr[0].id = cudaLaunchAttributeClusterDimension;
   attr[0].val.clusterDim.x = c.size;
   attr[0].val.clusterDim.y = 1;
   attr[0].val.clusterDim.z = 1;
   attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[1].val.programmaticStreamSerializationAllowed = 1;
   cfg->attrs = attr;
   cfg->numAttrs = 2;
}

}  // namespace

// clusters of a shape that the GPU holds at once, whatever the parameters turn
// out to be (0: it cannot run): the least over the generic kernel and the
// compiled features
cudaError_t cluster_capacity(const LLGArgs<float>& a, int var, const ClusterShape& c, int* clusters) {
   *clusters = 0;
   cudaLaunchConfig_t cfg;
   cudaLaunchAttribute attr[2];
   cluster_config(a, c, &cfg, attr);
   if (cfg.dynamicSmemBytes > kStageSmemLimit) return cudaSuccess;
   std::vector<int> feats{0};
   if (var == VAR_HEUN && c.zmax <= 6) {
#define VGPU_F(k) feats.push_back(k);
      VGPU_ISO_FEATURES(VGPU_F)
#undef VGPU_F
   }
   int least = 1 << 30;
   for (int feat : feats) {
      const ClusterFn f = cluster_fn(var, feat);
      cudaError_t e = cudaSuccess;
      if (c.size > 8) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e == cudaSuccess) e = allow_smem(f, (int)cfg.dynamicSmemBytes);
      int n = 0;
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, f, &cfg);
      if (e != cudaSuccess) return e;
      least = std::min(least, n);
   }
   *clusters = least;
   return cudaSuccess;
}

cudaError_t launch_llg_cluster(const LLGArgs<float>& a, int var, int nsteps, const ClusterShape& c, cudaStream_t st) {
   cudaLaunchConfig_t cfg;
   cudaLaunchAttribute attr[2];
   cluster_config(a, c, &cfg, attr);
   cfg.stream = st;
   return cudaLaunchKernelEx(&cfg, cluster_fn(var, c.zmax <= 6 ? iso_features<float>(a, FMT_ISO_TAB, var) : 0), a, nsteps,
                             c.zmax);
}

}  // namespace vgpu

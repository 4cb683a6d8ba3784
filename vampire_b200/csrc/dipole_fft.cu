// Far-field macrocell dipole sum by FFT convolution.
//
// The far field of every cell is H_i = sum_{j != i} T(r_j - r_i) m_j with the
// bare point-dipole tensor T(r) = (3 e e - 1)/|r|^3 (src/dipole/inter.cpp:66-80
// for cells beyond the cutoff; src/dipole/macrocell.cpp for all pairs).  When
// the occupied cells sit on one regular grid (every full cell of a lattice
// does: its magnetic centre is the cell origin plus a fixed offset), T depends
// only on the grid offset, so the sum is a linear convolution of the moment
// grid with T.  It is evaluated as a circular convolution on a grid padded to
// P >= 2G - 1 points per axis (G = occupied extent), with P a power of two:
//
//   x    forward transform of the real lines of the G-box, two lines as the
//        real and imaginary parts of one; the moments (mu_B) are read straight
//        from the cells, and the P/2 + 1 points that determine the spectrum of
//        a real line are written
//   y    forward transform in place, planes z < G
//   z    per z column: forward transform, H(k) = T(k) M(k), inverse transform
//        in one kernel, the spectra in registers
//   y    inverse transform in place, points y < G kept
//   x    inverse transform of line pairs, written to the cells' field
//
// T is real and even under r -> -r, so its spectrum is real; each component is
// even or odd in every single axis, so one octant of it (kx, ky, kz <= P/2,
// the rest by sign) is all that is kept: 6 (P/2+1)^3 reals, 6.6 MB in FP32 at
// P = 128, resident in L2, where the full complex spectra were 100 MB read on
// every update.
//
// The line transforms keep 8 points per thread in registers and go through
// shared memory once between radix-8 passes (radix 2 or 4 last), ceil(log2 P
// / 3) passes in all.  Blocks are bound by latency and L2 traffic, not by
// arithmetic: with lines of 128 points the grids are 3 x 3.3 MB.  At 125,000
// cells (50^3, P = 128) the five launches measured take the place of radix-2
// passes through shared memory over complex lines (two barriers and integer
// divisions per point and stage): 376 us then, 46 now (x 7, y 5, z 24, y 5,
// x 4); see fft_z_kernel for the split.
//
// Precision follows the handle: in the FP64 build every step is FP64, so the
// result equals the direct FP64 sum to rounding (~1e-15 of the field); the
// FP32 production handles transform FP32 grids where an axis has more than 8
// cells (the tensor spectra computed in FP64 once and rounded, twiddles rounded
// from FP64, moments and fields FP64 at the ends), a few 1e-7 of the field.  Cost O(P^3 log P) instead of
// O(Nc^2).
#include "dipole_fft.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "vgpu_internal.cuh"

namespace vgpu {

struct FFTField {
   int nc = 0;
   int p[3] = {0, 0, 0};       // padded points per axis (powers of two, at least 8)
   int logp[3] = {0, 0, 0};
   int g[3] = {0, 0, 0};       // occupied extent in cells
   int hx = 0;                 // stored points of an x spectrum: p[0] / 2 + 1
   size_t np = 0;              // p[0] * p[1] * p[2]
   bool fp32 = false;          // precision of grid, tspec and tw
   void* tspec = nullptr;      // [6][p[2]/2+1][p[1]/2+1][hx] real spectra of Txx, Txy, Txz, Tyy, Tyz, Tzz
   void* grid = nullptr;       // [3][g[2]][p[1]][hx] complex, transformed in place
   void* tw[3] = {nullptr, nullptr, nullptr};  // [p] exp(-2 pi i k / p) per axis
   int* box_cell = nullptr;    // [gx*gy*gz] cell at each box point (x fastest), or -1
};

namespace {

template <typename C> struct RealOf;
template <> struct RealOf<float2> { using type = float; };
template <> struct RealOf<double2> { using type = double; };

template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
   return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return {a.x + b.x, a.y + b.y}; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return {a.x - b.x, a.y - b.y}; }
// times -i (forward) or +i (inverse)
template <typename C, bool INV> __device__ __forceinline__ C crot(C a) {
   if (INV) return {-a.y, a.x};
   return {a.y, -a.x};
}

// discrete Fourier transforms of 2, 4 and 8 points in registers, natural order
template <typename C, bool INV> __device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d) {
   const C t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = crot<C, INV>(csub(b, d));
   a = cadd(t0, t2); b = cadd(t1, t3); c = csub(t0, t2); d = csub(t1, t3);
}
template <typename C, bool INV, int R> __device__ __forceinline__ void dft(C u[R]) {
   if constexpr (R == 2) {
      const C t = u[0];
      u[0] = cadd(t, u[1]);
      u[1] = csub(t, u[1]);
   } else if constexpr (R == 4) {
      dft4<C, INV>(u[0], u[1], u[2], u[3]);
   } else {
      using R1 = typename RealOf<C>::type;
      C e0 = u[0], e1 = u[2], e2 = u[4], e3 = u[6], o0 = u[1], o1 = u[3], o2 = u[5], o3 = u[7];
      dft4<C, INV>(e0, e1, e2, e3);
      dft4<C, INV>(o0, o1, o2, o3);
      const R1 h = (R1)0.70710678118654752440;
      const C r1 = crot<C, INV>(o1), r3 = crot<C, INV>(o3);
      o1 = {h * (o1.x + r1.x), h * (o1.y + r1.y)};  // (1 -+ i)/sqrt 2 times
      o2 = crot<C, INV>(o2);
      o3 = {h * (r3.x - o3.x), h * (r3.y - o3.y)};  // (-1 -+ i)/sqrt 2 times
      u[0] = cadd(e0, o0); u[4] = csub(e0, o0);
      u[1] = cadd(e1, o1); u[5] = csub(e1, o1);
      u[2] = cadd(e2, o2); u[6] = csub(e2, o2);
      u[3] = cadd(e3, o3); u[7] = csub(e3, o3);
   }
}

// Transforms of NC lines of N = 2^LOGN points, each held by the same N/8
// threads: thread j has points j + i N/8 (i = 0..7) of line c in v[c], before
// and after (natural order both times).  Passes of radix 8, the last one of
// the radix that is left; between passes the points go through shared memory
// at idx(c, point), the NC lines between the same two barriers.  Every thread
// of the block takes part.  NSLOG: log2 of the points already combined.
template <typename C, int LOGN, bool INV, int NSLOG, int NC, typename Idx>
__device__ __forceinline__ void fft_lines(C (&v)[NC][8], int j, C* s, Idx idx, const C* __restrict__ tw) {
   constexpr int RL = LOGN - NSLOG >= 3 ? 3 : LOGN - NSLOG;
   constexpr int R = 1 << RL, NB = 8 / R, NS = 1 << NSLOG, T = (1 << LOGN) / 8;
   constexpr bool LAST = NSLOG + RL == LOGN;
#pragma unroll
   for (int q = 0; q < NB; ++q) {
      const int bb = j + q * T, k = bb & (NS - 1);
      C w[R];
      if (NSLOG > 0) {
#pragma unroll
         for (int r = 1; r < R; ++r) {
            w[r] = __ldg(tw + ((k * r) << (LOGN - NSLOG - RL)));
            if (INV) w[r].y = -w[r].y;
         }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
         C u[R];
#pragma unroll
         for (int r = 0; r < R; ++r) u[r] = v[c][q + r * NB];
         if (NSLOG > 0) {
#pragma unroll
            for (int r = 1; r < R; ++r) u[r] = cmul(w[r], u[r]);
         }
         dft<C, INV, R>(u);
         if (LAST) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[c][q + r * NB] = u[r];
         } else {
            const int o = ((bb >> NSLOG) << (NSLOG + RL)) + k;
#pragma unroll
            for (int r = 0; r < R; ++r) s[idx(c, o + r * NS)] = u[r];
         }
      }
   }
   if constexpr (!LAST) {
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
         for (int i = 0; i < 8; ++i) v[c][i] = s[idx(c, j + i * T)];
      __syncthreads();  // s may be written again
      fft_lines<C, LOGN, INV, NSLOG + RL>(v, j, s, idx, tw);
   }
}

// lines per block of the strided transforms: 2,048 points (256 threads) and
// at most 64 lines.  16 adjacent columns at 128 points: a 128-byte segment per
// point in FP32.
constexpr int lines_of(int logn) { return (2048 >> logn) < 64 ? (2048 >> logn) : 64; }
constexpr int threads_of(int logn) { return lines_of(logn) << (logn - 3); }

// lines along y or z, in place: line l starts at (l / inner) * outer + l %
// inner, its points are `ps` apart; points p >= ld read as zero, points p < st
// are stored.  blockIdx.y: component (cs apart).
template <typename C, int LOGN, bool INV>
__global__ void __launch_bounds__(threads_of(LOGN)) fft_strided_kernel(C* __restrict__ data, size_t cs, int nlines,
                                                                       int inner, size_t outer, size_t ps,
                                                                       const C* __restrict__ tw, int ld, int st) {
   constexpr int W = lines_of(LOGN), T = (1 << LOGN) / 8;
   __shared__ C s[W << LOGN];
   pdl_begin();
   const int w = threadIdx.x % W, j = threadIdx.x / W;
   const int l = blockIdx.x * W + w;
   const bool on = l < nlines;
   C* base = data + (size_t)blockIdx.y * cs + (size_t)(l / inner) * outer + (size_t)(l % inner);
   C v[1][8];
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int p = j + i * T;
      v[0][i] = on && p < ld ? base[(size_t)p * ps] : C{0, 0};
   }
   fft_lines<C, LOGN, INV, 0>(v, j, s, [&](int, int p) { return p * W + w; }, tw);
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int p = j + i * T;
      if (on && p < st) base[(size_t)p * ps] = v[0][i];
   }
}

// sources of the real x lines: row r of component c, point x
struct MomentRows {  // the G-box, x fastest; zero at its empty cells
   const int* box_cell;
   const double* mag;
   int nc, gx;
   __device__ double operator()(int c, int r, int x) const {
      if (x >= gx) return 0.0;
      const int cell = __ldg(box_cell + (size_t)r * gx + x);
      return cell >= 0 ? __ldg(mag + (size_t)c * nc + cell) * (1.0 / 9.27400915e-24) : 0.0;
   }
};

struct TensorRows {  // bare tensor on the padded grid, zero at the origin and beyond the occupied extent
   int px, py, pz, gx, gy, gz;
   double size;
   __device__ double operator()(int c, int r, int x) const {
      const int y = r % py, z = r / py;
      const int dx = x < px / 2 ? x : x - px, dy = y < py / 2 ? y : y - py, dz = z < pz / 2 ? z : z - pz;
      if (!(abs(dx) < gx && abs(dy) < gy && abs(dz) < gz && (dx | dy | dz) != 0)) return 0.0;
      const double rx = dx * size, ry = dy * size, rz = dz * size;
      const double rij = 1.0 / sqrt(rx * rx + ry * ry + rz * rz);
      const double e[3] = {rx * rij, ry * rij, rz * rij};
      const double r3 = rij * rij * rij;
      const int a = c < 3 ? 0 : c < 5 ? 1 : 2, b = c < 3 ? c : c < 5 ? c - 2 : 2;
      return (3.0 * e[a] * e[b] - (a == b ? 1.0 : 0.0)) * r3;
   }
};

// Row r of the box or grid starts at row_start(r): rows per plane `rpp`, the
// planes hold `py` rows of hx points.
__device__ __forceinline__ size_t row_start(int r, int rpp, int py, int hx) {
   return ((size_t)(r / rpp) * py + (size_t)(r % rpp)) * hx;
}

// lines of a block of the x transforms: 1,024 points, at least one line
constexpr int xlines_of(int logn) { return logn >= 10 ? 1 : 1024 >> logn; }

// forward x: rows 2t and 2t + 1 as real and imaginary part of complex line t;
// the spectra are taken apart by their symmetry (Z(N - k) from shared memory)
template <typename C, int LOGN, typename Rows>
__global__ void __launch_bounds__(128) fft_x_forward_kernel(const Rows rows, C* __restrict__ out, size_t cs, int nrows,
                                                            int rpp, int py, const C* __restrict__ tw) {
   constexpr int N = 1 << LOGN, T = N / 8, L = xlines_of(LOGN), NP = N + N / 8, HX = N / 2 + 1;
   using R = typename RealOf<C>::type;
   __shared__ C s[L * NP];
   pdl_begin();
   const int j = threadIdx.x % T, line = threadIdx.x / T;
   const int ra = 2 * (blockIdx.x * L + line), rb = ra + 1;
   const int c = blockIdx.y;
   auto idx = [&](int, int p) { return line * NP + p + (p >> 3); };  // padded: points 8 apart in different banks
   C v[1][8];
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int x = j + i * T;
      v[0][i] = {(R)(ra < nrows ? rows(c, ra, x) : 0.0), (R)(rb < nrows ? rows(c, rb, x) : 0.0)};
   }
   fft_lines<C, LOGN, false, 0>(v, j, s, idx, tw);
#pragma unroll
   for (int i = 0; i < 8; ++i) s[idx(0, j + i * T)] = v[0][i];
   __syncthreads();
   C* oa = out + (size_t)c * cs + row_start(ra, rpp, py, HX);
   C* ob = out + (size_t)c * cs + row_start(rb, rpp, py, HX);
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int k = j + i * T;
      if (k <= N / 2) {
         const C z = v[0][i], n = s[idx(0, (N - k) & (N - 1))];
         const R h = (R)0.5;
         if (ra < nrows) oa[k] = {h * (z.x + n.x), h * (z.y - n.y)};
         if (rb < nrows) ob[k] = {h * (z.y + n.y), h * (n.x - z.x)};
      }
   }
}

// inverse x of the G-box rows, two at a time, written to the cells' field
template <typename C, int LOGN>
__global__ void __launch_bounds__(128) fft_x_inverse_kernel(const C* __restrict__ in, size_t cs, int nrows, int rpp,
                                                            int py, const C* __restrict__ tw,
                                                            const int* __restrict__ box_cell, int gx, int nc,
                                                            double scale, double* __restrict__ field) {
   constexpr int N = 1 << LOGN, T = N / 8, L = xlines_of(LOGN), NP = N + N / 8, HX = N / 2 + 1;
   __shared__ C s[L * NP];
   pdl_begin();
   const int j = threadIdx.x % T, line = threadIdx.x / T;
   const int ra = 2 * (blockIdx.x * L + line), rb = ra + 1;
   const int c = blockIdx.y;
   const C* ia = in + (size_t)c * cs + row_start(ra, rpp, py, HX);
   const C* ib = in + (size_t)c * cs + row_start(rb, rpp, py, HX);
   C v[1][8];
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int k = j + i * T, m = k <= N / 2 ? k : N - k;
      C a = ra < nrows ? ia[m] : C{0, 0}, b = rb < nrows ? ib[m] : C{0, 0};
      if (m == 0 || m == N / 2) a.y = b.y = 0;  // real by symmetry
      if (k > N / 2) { a.y = -a.y; b.y = -b.y; }
      v[0][i] = {a.x - b.y, a.y + b.x};
   }
   fft_lines<C, LOGN, true, 0>(v, j, s, [&](int, int p) { return line * NP + p + (p >> 3); }, tw);
#pragma unroll
   for (int i = 0; i < 8; ++i) {
      const int x = j + i * T;
      if (x < gx) {
         const int a = ra < nrows ? __ldg(box_cell + (size_t)ra * gx + x) : -1;
         const int b = rb < nrows ? __ldg(box_cell + (size_t)rb * gx + x) : -1;
         if (a >= 0) field[(size_t)c * nc + a] = (double)v[0][i].x * scale;
         if (b >= 0) field[(size_t)c * nc + b] = (double)v[0][i].y * scale;
      }
   }
}

// The middle of the convolution: for W adjacent (y, x) columns the three
// moment components' forward z transforms (points z >= gz are zero), H(k) =
// T(k) M(k), and the inverse transforms, of which z < gz is stored.  The three
// spectra stay in registers (24 complex points a thread) and share the
// barriers of the exchanges.
template <typename C, int LOGN>
__global__ void __launch_bounds__(threads_of(LOGN)) fft_z_kernel(C* __restrict__ data, size_t cs,
                                                                 const typename RealOf<C>::type* __restrict__ t, int hx,
                                                                 int py, int gz, const C* __restrict__ tw) {
   constexpr int N = 1 << LOGN, W = lines_of(LOGN), T = N / 8;
   using R = typename RealOf<C>::type;
   extern __shared__ __align__(16) unsigned char fft_smem[];
   C* s = reinterpret_cast<C*>(fft_smem);
   pdl_begin();
   const int w = threadIdx.x % W, j = threadIdx.x / W;
   const int nlines = hx * py;
   const int l = blockIdx.x * W + w;
   const bool on = l < nlines;
   C v[3][8];
#pragma unroll
   for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
         const int p = j + i * T;
         v[c][i] = on && p < gz ? data[(size_t)c * cs + (size_t)p * nlines + l] : C{0, 0};
      }
   auto idx = [&](int c, int p) { return c * (W << LOGN) + p * W + w; };
   fft_lines<C, LOGN, false, 0>(v, j, s, idx, tw);
   {
      const int ky = on ? l / hx : 0, kx = on ? l % hx : 0;
      const int hy = py / 2 + 1;
      const bool fy = ky > py / 2;  // the mirrored half: odd components change sign
      const size_t ts = (size_t)hx * hy * (N / 2 + 1);
      const R* row = t + (size_t)(fy ? py - ky : ky) * hx + kx;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
         const int k = j + i * T;
         const bool fz = k > N / 2;
         const R* q = row + (size_t)(fz ? N - k : k) * hx * hy;
         const R xx = __ldg(q), yy = __ldg(q + 3 * ts), zz = __ldg(q + 5 * ts);
         R xy = __ldg(q + ts), xz = __ldg(q + 2 * ts), yz = __ldg(q + 4 * ts);
         if (fy) { xy = -xy; yz = -yz; }
         if (fz) { xz = -xz; yz = -yz; }
         const C mx = v[0][i], my = v[1][i], mz = v[2][i];
         v[0][i] = {xx * mx.x + xy * my.x + xz * mz.x, xx * mx.y + xy * my.y + xz * mz.y};
         v[1][i] = {xy * mx.x + yy * my.x + yz * mz.x, xy * mx.y + yy * my.y + yz * mz.y};
         v[2][i] = {xz * mx.x + yz * my.x + zz * mz.x, xz * mx.y + yz * my.y + zz * mz.y};
      }
   }
   fft_lines<C, LOGN, true, 0>(v, j, s, idx, tw);
#pragma unroll
   for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
         const int p = j + i * T;
         if (on && p < gz) data[(size_t)c * cs + (size_t)p * nlines + l] = v[c][i];
      }
}

// the octant of the (real) tensor spectra from the full transforms, rounded to R
template <typename R>
__global__ void spectrum_octant_kernel(const double2* __restrict__ full, size_t cs, int hx, int py, int hy, int hz,
                                       R* __restrict__ out) {
   const size_t n = (size_t)hx * hy * hz;
   for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
      const size_t x = q % hx, y = (q / hx) % hy, z = q / ((size_t)hx * hy);
      out[(size_t)blockIdx.y * n + q] = (R)full[(size_t)blockIdx.y * cs + (z * py + y) * hx + x].x;
   }
}

int ilog2(int v) {
   int l = 0;
   while ((1 << l) < v) ++l;
   return l;
}

// CALL with the constant LN = logn, for logn = 3..10 (the planner's range)
#define VGPU_FFT_DISPATCH(logn, CALL)                                       \
   switch (logn) {                                                          \
      case 3: { constexpr int LN = 3; CALL; } break;                        \
      case 4: { constexpr int LN = 4; CALL; } break;                        \
      case 5: { constexpr int LN = 5; CALL; } break;                        \
      case 6: { constexpr int LN = 6; CALL; } break;                        \
      case 7: { constexpr int LN = 7; CALL; } break;                        \
      case 8: { constexpr int LN = 8; CALL; } break;                        \
      case 9: { constexpr int LN = 9; CALL; } break;                        \
      case 10: { constexpr int LN = 10; CALL; } break;                      \
      default: e = cudaErrorInvalidValue;                                   \
   }

template <typename C, typename Rows>
cudaError_t x_forward(const Rows& rows, C* out, size_t cs, int logn, int ncomp, int nrows, int rpp, int py, const C* tw,
                      cudaStream_t st) {
   cudaError_t e = cudaSuccess;
   VGPU_FFT_DISPATCH(logn, {
      constexpr int L = xlines_of(LN);
      const int npairs = (nrows + 1) / 2;
      e = launch_pdl(fft_x_forward_kernel<C, LN, Rows>, dim3((npairs + L - 1) / L, ncomp), dim3(L << (LN - 3)), 0, st,
                     rows, out, cs, nrows, rpp, py, tw);
   })
   return e;
}

template <typename C, bool INV>
cudaError_t strided(C* data, size_t cs, int logn, int ncomp, int nlines, int inner, size_t outer, size_t ps,
                    const C* tw, int ld, int stp, cudaStream_t st) {
   cudaError_t e = cudaSuccess;
   VGPU_FFT_DISPATCH(logn, {
      constexpr int W = lines_of(LN);
      e = launch_pdl(fft_strided_kernel<C, LN, INV>, dim3((nlines + W - 1) / W, ncomp), dim3(threads_of(LN)), 0, st,
                     data, cs, nlines, inner, outer, ps, tw, ld, stp);
   })
   return e;
}

template <typename C> constexpr int z_smem(int logn) { return 3 * (int)sizeof(C) * (lines_of(logn) << logn); }

// the z kernel's shared memory above the default limit (FP64): asked for once per field
template <typename C>
cudaError_t z_prepare(int logn) {
   cudaError_t e = cudaSuccess;
   VGPU_FFT_DISPATCH(logn, {
      e = cudaFuncSetAttribute(fft_z_kernel<C, LN>, cudaFuncAttributeMaxDynamicSharedMemorySize, z_smem<C>(LN));
   })
   return e;
}

template <typename C>
cudaError_t field_apply(FFTField* f, const double* mag, double* field, cudaStream_t st, int* launches) {
   using R = typename RealOf<C>::type;
   const int py = f->p[1];
   const int gx = f->g[0], gy = f->g[1], gz = f->g[2], hx = f->hx;
   C* grid = static_cast<C*>(f->grid);
   const C* tw[3] = {static_cast<const C*>(f->tw[0]), static_cast<const C*>(f->tw[1]), static_cast<const C*>(f->tw[2])};
   const size_t cs = (size_t)gz * py * hx;
   const size_t plane = (size_t)py * hx;
   cudaError_t e = x_forward<C>(MomentRows{f->box_cell, mag, f->nc, gx}, grid, cs, f->logp[0], 3, gy * gz, gy, py,
                                tw[0], st);
   if (e == cudaSuccess) e = strided<C, false>(grid, cs, f->logp[1], 3, gz * hx, hx, plane, hx, tw[1], gy, py, st);
   if (e == cudaSuccess) {
      VGPU_FFT_DISPATCH(f->logp[2], {
         constexpr int W = lines_of(LN);
         e = launch_pdl(fft_z_kernel<C, LN>, dim3((hx * py + W - 1) / W), dim3(threads_of(LN)), z_smem<C>(LN), st,
                        grid, cs, static_cast<const R*>(f->tspec), hx, py, gz, tw[2]);
      })
   }
   if (e == cudaSuccess) e = strided<C, true>(grid, cs, f->logp[1], 3, gz * hx, hx, plane, hx, tw[1], py, gy, st);
   if (e == cudaSuccess) {
      VGPU_FFT_DISPATCH(f->logp[0], {
         constexpr int L = xlines_of(LN);
         const int npairs = (gy * gz + 1) / 2;
         e = launch_pdl(fft_x_inverse_kernel<C, LN>, dim3((npairs + L - 1) / L, 3), dim3(L << (LN - 3)), 0, st,
                        (const C*)grid, cs, gy * gz, gy, py, tw[0], (const int*)f->box_cell, gx, f->nc,
                        1.0 / (double)f->np, field);
      })
   }
   if (launches) *launches += 5;
   return e;
}

// the tensor spectra: FP64 transforms of the six components on the whole grid,
// then their octant in the field's precision
template <typename C>
cudaError_t make_spectra(FFTField* f, double size, double2* const* tw, cudaStream_t st) {
   using R = typename RealOf<C>::type;
   const int px = f->p[0], py = f->p[1], pz = f->p[2], hx = f->hx, hy = py / 2 + 1, hz = pz / 2 + 1;
   const size_t cs = (size_t)pz * py * hx;
   double2* full = nullptr;
   cudaError_t e = cudaMalloc(&full, sizeof(double2) * 6 * cs);
   if (e != cudaSuccess) return e;
   e = cudaMalloc(&f->tspec, sizeof(R) * 6 * (size_t)hx * hy * hz);
   if (e == cudaSuccess)
      e = x_forward<double2>(TensorRows{px, py, pz, f->g[0], f->g[1], f->g[2], size}, full, cs, f->logp[0], 6, py * pz,
                             py, py, (const double2*)tw[0], st);
   if (e == cudaSuccess)
      e = strided<double2, false>(full, cs, f->logp[1], 6, pz * hx, hx, (size_t)py * hx, hx, tw[1], py, py, st);
   if (e == cudaSuccess)
      e = strided<double2, false>(full, cs, f->logp[2], 6, py * hx, py * hx, 0, (size_t)py * hx, tw[2], pz, pz, st);
   if (e == cudaSuccess) {
      const size_t n = (size_t)hx * hy * hz;
      spectrum_octant_kernel<R><<<dim3((unsigned)std::min<size_t>((n + 255) / 256, 148 * 8), 6), 256, 0, st>>>(
          full, cs, hx, py, hy, hz, static_cast<R*>(f->tspec));
      e = cudaGetLastError();
   }
   if (e == cudaSuccess) e = cudaStreamSynchronize(st);
   cudaFree(full);
   return e;
}

}  // namespace

FFTField* fft_field_create(int nc, const double* cpos, const int* natoms, double size, bool fp32, cudaStream_t st,
                           cudaError_t* err, std::string* why) {
   *err = cudaSuccess;
   int first = -1;
   for (int c = 0; c < nc && first < 0; ++c)
      if (natoms[c] > 0) first = c;
   if (first < 0 || !(size > 0.0)) {
      *why = "no occupied cells";
      return nullptr;
   }
   // grid coordinates of every occupied cell relative to the first one
   std::vector<long long> gi(3 * (size_t)nc, 0);
   long long lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
   for (int c = 0; c < nc; ++c) {
      if (natoms[c] <= 0) continue;
      for (int a = 0; a < 3; ++a) {
         const double u = (cpos[4 * c + a] - cpos[4 * first + a]) / size;
         const double r = std::nearbyint(u);
         if (std::fabs(u - r) > 1e-9) {
            *why = "cell centres are not on one regular grid";
            return nullptr;
         }
         gi[3 * (size_t)c + a] = (long long)r;
         lo[a] = std::min(lo[a], (long long)r);
         hi[a] = std::max(hi[a], (long long)r);
      }
   }
   FFTField* f = new FFTField();
   f->nc = nc;
   size_t np = 1;
   for (int a = 0; a < 3; ++a) {
      const long long G = hi[a] - lo[a] + 1;
      int P = 8;  // the line transforms hold 8 points per thread
      while (P < 2 * G - 1 && P <= 1024) P <<= 1;
      if (P > 1024) {
         *why = "cell grid too large for the FFT solver";
         delete f;
         return nullptr;
      }
      f->g[a] = (int)G;
      f->p[a] = P;
      f->logp[a] = ilog2(P);
      np *= (size_t)P;
   }
   if (np > ((size_t)1 << 25)) {
      *why = "padded cell grid above 2^25 points";
      delete f;
      return nullptr;
   }
   f->np = np;
   f->hx = f->p[0] / 2 + 1;
   // Grids of at most 8 cells per axis stay in FP64: with so few passes the two
   // roundings of packing real lines in pairs weigh more than the passes they
   // save (2-norm error of B against FP64 on FP32 handles: 4^3 cells 1.76e-7 with
   // complex radix-2 lines, 1.81e-7 with packed FP32 lines; 8^3 2.24e-7 and
   // 2.35e-7; from 9 cells on packed lines are the more exact, 10^3 2.50e-7 and
   // 2.21e-7), and such a grid costs its launches whatever its type.
   fp32 = fp32 && std::max(f->p[0], std::max(f->p[1], f->p[2])) > 16;
   f->fp32 = fp32;
   // cell at each point of the G-box; two cells on one grid point are not a grid
   const size_t nbox = (size_t)f->g[0] * f->g[1] * f->g[2];
   std::vector<int> boxc(nbox, -1);
   for (int c = 0; c < nc; ++c) {
      if (natoms[c] <= 0) continue;
      const size_t x = (size_t)(gi[3 * (size_t)c] - lo[0]), y = (size_t)(gi[3 * (size_t)c + 1] - lo[1]),
                   z = (size_t)(gi[3 * (size_t)c + 2] - lo[2]);
      int& at = boxc[(z * f->g[1] + y) * f->g[0] + x];
      if (at >= 0) {
         *why = "two cells share a grid point";
         delete f;
         return nullptr;
      }
      at = c;
   }
   const size_t cw = fp32 ? sizeof(float2) : sizeof(double2);
   cudaError_t e = cudaMalloc(&f->grid, cw * 3 * (size_t)f->g[2] * f->p[1] * f->hx);
   if (e == cudaSuccess) e = cudaMalloc(&f->box_cell, sizeof(int) * nbox);
   if (e == cudaSuccess) e = cudaMemcpyAsync(f->box_cell, boxc.data(), sizeof(int) * nbox, cudaMemcpyHostToDevice, st);
   // twiddles in FP64 for the spectra, and rounded to the field's precision
   std::vector<std::vector<double2>> tw(3);
   std::vector<std::vector<float2>> twf(3);
   double2* tw64[3] = {nullptr, nullptr, nullptr};
   for (int a = 0; a < 3 && e == cudaSuccess; ++a) {
      const int P = f->p[a];
      tw[a].resize(P);
      twf[a].resize(P);
      for (int k = 0; k < P; ++k) {
         const double ang = -2.0 * M_PI * (double)k / (double)P;
         tw[a][k] = make_double2(std::cos(ang), std::sin(ang));
         twf[a][k] = make_float2((float)tw[a][k].x, (float)tw[a][k].y);
      }
      e = cudaMalloc(&tw64[a], sizeof(double2) * P);
      if (e == cudaSuccess)
         e = cudaMemcpyAsync(tw64[a], tw[a].data(), sizeof(double2) * P, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess && fp32) {
         e = cudaMalloc(&f->tw[a], sizeof(float2) * P);
         if (e == cudaSuccess)
            e = cudaMemcpyAsync(f->tw[a], twf[a].data(), sizeof(float2) * P, cudaMemcpyHostToDevice, st);
      }
   }
   if (e == cudaSuccess) e = fp32 ? make_spectra<float2>(f, size, tw64, st) : make_spectra<double2>(f, size, tw64, st);
   if (e == cudaSuccess) e = fp32 ? z_prepare<float2>(f->logp[2]) : z_prepare<double2>(f->logp[2]);
   if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // host tables above leave scope
   for (int a = 0; a < 3; ++a) {
      if (e == cudaSuccess && !fp32) f->tw[a] = tw64[a];
      else cudaFree(tw64[a]);
   }
   if (e != cudaSuccess) {
      *err = e;
      fft_field_destroy(f);
      return nullptr;
   }
   return f;
}

cudaError_t fft_field_apply(FFTField* f, const double* mag, double* field, cudaStream_t st, int* launches) {
   if (f->fp32) return field_apply<float2>(f, mag, field, st, launches);
   return field_apply<double2>(f, mag, field, st, launches);
}

void fft_field_destroy(FFTField* f) {
   if (!f) return;
   cudaFree(f->tspec);
   cudaFree(f->grid);
   cudaFree(f->box_cell);
   for (int a = 0; a < 3; ++a) cudaFree(f->tw[a]);
   delete f;
}

void fft_field_shape(const FFTField* f, int p[3]) {
   for (int a = 0; a < 3; ++a) p[a] = f ? f->p[a] : 0;
}

}  // namespace vgpu

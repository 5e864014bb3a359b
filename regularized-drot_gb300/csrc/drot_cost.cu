// drot_cost.cu -- squared-Euclidean cost matrices of point clouds on the
// 5th-generation tensor cores (tcgen05.mma kind::tf32, accumulator in TMEM).
//
// No counterpart in the reference, whose callers build C on the host
// (benchmark/utils/compute_w2_dist.py:68-94) and hand it to the solver.  For
// point clouds x (m x d) and y (n x d), row-major:
//     C[j*ld + i] = scale * max(||x_i||^2 + ||y_j||^2 - 2 <x_i, y_j>, 0)
// i.e. the column-major m x n cost the solver reads (the reference's PyTorch
// layout [n, m]).  The Gram term is one GEMM with K = d, done in "3xTF32":
// x = x_hi + x_lo with x_hi = RN_tf32(x), x_lo = RN_tf32(x - x_hi) (same
// for y), <x, y> ~ x_hi.y_hi + x_hi.y_lo + x_lo.y_hi accumulated in FP32 --
// the split-precision scheme that gives FP32-level accuracy on TF32 tensor
// cores (the dropped x_lo.y_lo term is below 2^-22 relative).  Norms are
// FP32 FMA sums in k order.
//
// Persistent kernel (at most two CTAs per SM, each walking the tiles of all
// instances with stride grid): per 128 x 128 tile, 256 threads stage the
// hi / lo operand tiles in shared memory (K-major, no swizzle: 8-row x
// 16-byte core matrices), one thread issues 3 * d/8 MMAs into a 128-lane x
// 128-column TMEM accumulator and a tcgen05.commit arrives on an mbarrier;
// then each warp reads its TMEM lane quadrant for half of the columns
// (tcgen05.ld 32x32b) and writes those rows of each column (128 bytes per
// warp store).  Operands and accumulators are double-buffered, so tile n+1's
// loads and MMAs run while tile n's C is stored.  The kernel is bound by the
// C stores (4 bytes per element).
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "drot_gb300.h"
#include "drot_kernels.cuh"

namespace drot {

constexpr int kCostM = 128;        // tile rows (x points) = TMEM lanes
constexpr int kCostN = 128;        // tile columns (y points) = TMEM columns
constexpr int kCostMaxInst = 256;  // instances per launch (descriptors travel in the parameters)
constexpr int kCostThreads = 256;  // 8 warps: x / y rows staged one per thread

struct CostInst {
  long long x_off, y_off, c_off;  // element offsets: x (m x d), y (n x d), C (ld x n)
  int m, n, ld, tiles_m, tiles;
  int tile0;  // tiles of the earlier instances
};

struct CostParams {
  const float* x;
  const float* y;
  float* c;
  int* err;
  long long timeout_ns;
  int dim, n_inst, clamp, total_tiles;
  float scale, pad2;
  CostInst inst[kCostMaxInst];
};

// Instruction descriptor of the tile's MMAs (M = 128 x points, N = 128 y points).
constexpr uint32_t kCostIdesc = tf32_idesc(kCostM, kCostN);

// Stage tile (i0, j0) of instance I into one operand buffer: x rows by
// threads 0..127, y rows by threads 128..255 (one row each): hi / lo TF32
// parts in the K-major layout, FP32 norms in k order.
__device__ __forceinline__ void cost_stage(const CostParams& P, const CostInst& I, int i0, int j0,
                                           unsigned char* buf, uint32_t op_bytes, float* norms) {
  const int d = P.dim, kc = d >> 2, tid = threadIdx.x;
  const bool is_y = tid >= kCostM;
  const int r = is_y ? tid - kCostM : tid;
  const int row = (is_y ? j0 : i0) + r;
  const bool in = row < (is_y ? I.n : I.m);
  const float4* src = reinterpret_cast<const float4*>(
      (is_y ? P.y + I.y_off : P.x + I.x_off) + (long long)(in ? row : 0) * d);
  unsigned char* hi_t = buf + (is_y ? 2 * op_bytes : 0);
  unsigned char* lo_t = hi_t + op_bytes;
  float nrm = 0.0f;
  for (int c4 = 0; c4 < kc; ++c4) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in) v = __ldg(src + c4);
    const float e[4] = {v.x, v.y, v.z, v.w};
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      hi[q] = to_tf32(e[q]);
      lo[q] = to_tf32(e[q] - __uint_as_float(hi[q]));
      nrm = fmaf(e[q], e[q], nrm);
    }
    const uint32_t off = kmaj_off(r, c4 * 4, kc);
    *reinterpret_cast<uint4*>(hi_t + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(lo_t + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  norms[tid] = nrm;  // x norms [0, 128), y norms [128, 256)
}

// The 3 x d/8 MMAs of one tile into a 128-column TMEM accumulator, then a
// commit arriving on `bar` (one thread).
__device__ __forceinline__ void cost_issue(unsigned char* buf, uint32_t op_bytes, int d,
                                           uint32_t tmem, uint64_t* bar) {
  const uint32_t ah = smem_u32(buf), al = ah + op_bytes;
  const uint32_t bh = al + op_bytes, bl = bh + op_bytes;
  gram_tf32x3(ah, al, bh, bl, d, tmem, kCostIdesc);
  tc_commit(bar);
}

// Instance and tile coordinates of global tile g (k advances monotonically).
__device__ __forceinline__ void cost_locate(const CostParams& P, int g, int& k, int& i0, int& j0) {
  while (g >= P.inst[k].tile0 + P.inst[k].tiles) ++k;
  const int t = g - P.inst[k].tile0;
  i0 = (t % P.inst[k].tiles_m) * kCostM;
  j0 = (t / P.inst[k].tiles_m) * kCostN;
}

// Persistent: CTA b takes tiles b, b + grid, ... of all instances in order.
// Operand buffers and TMEM accumulators are double-buffered, so while the
// eight warps stage tile n+1 and then store tile n's C, the tensor core
// computes tile n+1: the MMA and the operand loads hide behind the stores.
__global__ void __launch_bounds__(kCostThreads, 1) cost_sqeuclid_kernel(const __grid_constant__ CostParams P) {
  const int d = P.dim;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t op_bytes = (uint32_t)kCostM * d * 4;  // one hi or lo tile (x or y: 128 rows)
  const uint32_t buf_bytes = 4 * op_bytes;
  // norms of tile n in slot n % 3: staging writes tile n+1's while slower
  // warps may still read tile n-1's
  float* norms = reinterpret_cast<float*>(smem + 2 * buf_bytes);  // [3][256]
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ uint32_t s_tmem;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&s_tmem)), "r"((uint32_t)(2 * kCostN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    fence_mbar_init();
  }
  int g = blockIdx.x, kk = 0, i0 = 0, j0 = 0;
  if (g < P.total_tiles) {
    cost_locate(P, g, kk, i0, j0);
    cost_stage(P, P.inst[kk], i0, j0, smem, op_bytes, norms);
  }
  fence_proxy_async_shared();  // generic-proxy smem writes -> visible to the tensor core
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  if (tid == 0 && g < P.total_tiles) cost_issue(smem, op_bytes, d, tmem, &mbar[0]);

  // Epilogue split: warp w reads TMEM lanes 32 (w % 4) .. + 31 (its lane
  // quadrant) and columns 64 (w / 4) .. + 63 of the accumulator.
  const int quad = warp & 3, half = warp >> 2;
  for (int n = 0; g < P.total_tiles; ++n, g += gridDim.x) {
    const int b = n & 1;
    const int g_next = g + (int)gridDim.x;
    int kn = kk, in0 = 0, jn0 = 0;
    if (g_next < P.total_tiles) {
      cost_locate(P, g_next, kn, in0, jn0);
      cost_stage(P, P.inst[kn], in0, jn0, smem + (b ^ 1) * buf_bytes, op_bytes,
                 norms + ((n + 1) % 3) * 256);
    }
    fence_proxy_async_shared();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0 && g_next < P.total_tiles)
      cost_issue(smem + (b ^ 1) * buf_bytes, op_bytes, d, tmem + (uint32_t)((b ^ 1) * kCostN),
                 &mbar[b ^ 1]);
    // tile n's accumulator: use n >> 1 of buffer b
    bool got = mbar_wait(&mbar[b], (uint32_t)((n >> 1) & 1), P.timeout_ns);
    if (!__syncthreads_and(got ? 1 : 0)) {
      // An MMA that never completed: report it, give the MMAs in flight a
      // second bounded chance to land, and stop without storing.
      if (tid == 0) atomicExch(P.err, 1);
      mbar_wait(&mbar[b], (uint32_t)((n >> 1) & 1), P.timeout_ns);
      if (g_next < P.total_tiles) mbar_wait(&mbar[b ^ 1], (uint32_t)(((n + 1) >> 1) & 1), P.timeout_ns);
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const CostInst& I = P.inst[kk];
    const int i = i0 + quad * 32 + lane;
    const float* nb = norms + (n % 3) * 256;
    const float xi = nb[quad * 32 + lane];
    float* crow = P.c + I.c_off + (long long)(j0 + half * 64) * I.ld + i;
    const bool full = i0 + kCostM <= I.m && j0 + kCostN <= I.n;
    const bool row_in = i < I.m;
#pragma unroll
    for (int cb = 0; cb < 64; cb += 32) {
      uint32_t r[32];
      const uint32_t taddr = tmem + (uint32_t)(b * kCostN) + ((uint32_t)(quad * 32) << 16) +
                             (uint32_t)(half * 64 + cb);
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
          "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
          "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
            "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
            "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
            "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
            "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
            "=r"(r[31])
          : "r"(taddr) : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const float* yn = nb + kCostM + half * 64 + cb;
      float* cp = crow + (long long)cb * I.ld;
      if (full) {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float v = fmaf(-2.0f, __uint_as_float(r[e]), xi + yn[e]);
          if (P.clamp) v = fmaxf(v, 0.0f);
          cp[(long long)e * I.ld] = v * P.scale;
        }
      } else if (row_in) {
        const int jb = j0 + half * 64 + cb;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (jb + e < I.n) {
            float v = fmaf(-2.0f, __uint_as_float(r[e]), xi + yn[e]);
            if (P.clamp) v = fmaxf(v, 0.0f);
            cp[(long long)e * I.ld] = v * P.scale;
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    kk = kn;
    i0 = in0;
    j0 = jn0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(tmem), "r"((uint32_t)(2 * kCostN)) : "memory");
}

static size_t cost_smem_bytes(int dim) {
  // two operand buffers (x hi / lo, y hi / lo: 4 x 128 rows x dim floats) + [3][256] norms
  return (size_t)2 * 4 * kCostM * dim * 4 + sizeof(float) * 3 * 256;
}

// ---------------------------------------------------------------------------
// chain rule of the cost to the points (autograd backward of the cost)
// ---------------------------------------------------------------------------
//
// For G = dL/dC of one instance (column-major m x n, the layout of C),
//     dL/dx_i = 2 scale (x_i sum_j G_ij - sum_j G_ij y_j)
//     dL/dy_j = 2 scale (y_j sum_i G_ij - sum_i G_ij x_i)
// (G zeroed where C = 0 when the cost was clamped).  A CTA takes a block of
// 256 rows (band) by a few 32-column tiles (chunk) of one instance; thread t loads 4 rows (t % 64) of the 8 columns t / 64 + 4 p of a
// tile into registers (128-bit loads, 8 of G and 8 of C in flight).
//   rows: from the registers, 4 rows x (d + 1) sums per thread with y of the
//     column broadcast from shared memory (d / 4 loads for 4 (d + 1) FMAs);
//     the four column groups' sums are added at the end -> the chunk's partial
//     of dL/dx.
//   columns: the tile goes to shared memory column by column (pitch 260
//     floats: conflict-free 128-bit accesses both ways); a thread sums 8 of
//     the d components of two columns over its share of the band's rows (x
//     broadcast), the shares are added -> the band's partial of dL/dy.
// A second kernel adds the partials in order.  No atomics: deterministic.
// Bound at d = 16 by issue slots and shared memory, about half busy each (2 (d +
// 1) FMAs per element; 90 M elements: 51 % and 43 %, DRAM at 0.43 of the copy
// bandwidth), and by the latency of a tile's loads between its barriers.  One CTA
// per band walking all columns, which this replaces, kept 16 CTAs busy on a 4000
// x 3000 matrix: 900 us against 47 us here.

constexpr int kGradRows = 256;   // rows per band (= threads)
constexpr int kGradCols = 32;    // columns per tile
constexpr int kGradPitch = kGradRows + 4;

struct GradInst {
  long long x_off, y_off, c_off;  // element offsets: x (m x d), y (n x d), G / C (ld x n)
  long long py_off, px_off;       // float offsets of its partials: [bands][n][d + 1] of dL/dy,
                                  // [chunks][m][d + 1] of dL/dx
  int m, n, ld, bands, chunks, aligned;
};

struct GradParams {
  const float* x;
  const float* y;
  const float* g;
  const float* c;  // null: no clamp mask
  float* gx;
  float* gy;
  float* part;
  int n_inst;
  int chunk_cols;  // columns of a chunk (whole tiles)
  float scale2;  // 2 * scale
  GradInst inst[kCostMaxInst];
};

// Shared memory of the kernel (floats): the tile, x of the band, y of the
// tile, the column shares; the row groups' sums reuse the tile.
template <int DIM>
struct GradShape {
  static constexpr int KS = DIM / 8;          // component slices of a column pair
  static constexpr int RG = KS == 3 ? 4 : 16 / KS;  // row shares of 16 column pairs x KS
  static constexpr int TILE = kGradCols * kGradPitch;
  static constexpr int XS = kGradRows * DIM, YS = kGradCols * DIM;
  static constexpr int SHARE = RG * kGradCols * (DIM + 1);
  static constexpr int GROUP = kGradRows * (DIM + 1);  // one column group's row sums
  static constexpr int FLOATS = (TILE > GROUP ? TILE : GROUP) + XS + YS + SHARE;
};

template <int DIM>
__global__ void __launch_bounds__(kGradRows, DIM <= 16 ? 2 : 1)
cost_grad_kernel(const __grid_constant__ GradParams P) {
  using S = GradShape<DIM>;
  extern __shared__ __align__(16) float gsm[];
  float* const gt = gsm;  // [kGradCols][kGradPitch]
  float* const xs = gsm + (S::TILE > S::GROUP ? S::TILE : S::GROUP);  // [kGradRows][DIM]
  float* const ys = xs + S::XS;                                       // [kGradCols][DIM]
  float* const sh = ys + S::YS;                                       // [RG][kGradCols][DIM + 1]
  const GradInst& I = P.inst[blockIdx.z];
  const int band = blockIdx.x;
  if (band >= I.bands || (int)blockIdx.y >= I.chunks) return;
  const int t = threadIdx.x;
  const int m = I.m, n = I.n;
  const long long ld = I.ld;
  const int r0 = band * kGradRows;
  for (int e = t; e < kGradRows * DIM; e += kGradRows)
    xs[e] = r0 + e / DIM < m ? __ldg(P.x + I.x_off + (long long)r0 * DIM + e) : 0.0f;
  const int rr = 4 * (t % 64), cg = t / 64, i = r0 + rr;
  const float* const gcol = P.g + I.c_off + i;
  const float* const ccol = P.c ? P.c + I.c_off + i : nullptr;
  const bool vec = I.aligned && i + 4 <= m;
  // column phase: pair cp, slice ks, row share rg
  const int cp = t % 16, ks = (t / 16) % S::KS, rg = t / (16 * S::KS);
  for (int chunk = blockIdx.y; chunk < I.chunks; chunk += gridDim.y) {
    const int cb = chunk * P.chunk_cols, ce = min(cb + P.chunk_cols, n);
    float ax[4][DIM], rs[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      rs[e] = 0.0f;
#pragma unroll
      for (int k = 0; k < DIM; ++k) ax[e][k] = 0.0f;
    }
    for (int c0 = cb; c0 < ce; c0 += kGradCols) {
      float v[8][4];
      {
        // the next tile's lines into L2: this tile's loads then wait for L2,
        // not for DRAM (32 columns of 8 lines each, of G and of C)
        const int jn = c0 + kGradCols + t / 8, ln = r0 + 32 * (t % 8);
        if (jn < n && ln < m) {
          prefetch_l2(P.g + I.c_off + (long long)jn * ld + ln);
          if (P.c) prefetch_l2(P.c + I.c_off + (long long)jn * ld + ln);
        }
      }
#pragma unroll
      for (int hb = 0; hb < 8; hb += 4) {
        float cv[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            v[hb + q][e] = 0.0f;
            cv[q][e] = 1.0f;
          }
        }
        if (vec) {
          // all loads of the half tile before the first use
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = c0 + cg + 4 * (hb + q);
            if (j < ce) load_vec_nc<4>(gcol + (long long)j * ld, v[hb + q]);
          }
          if (ccol) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int j = c0 + cg + 4 * (hb + q);
              if (j < ce) load_vec_nc<4>(ccol + (long long)j * ld, cv[q]);
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = c0 + cg + 4 * (hb + q);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (j < ce && i + e < m) {
                v[hb + q][e] = __ldg(gcol + (long long)j * ld + e);
                if (ccol) cv[q][e] = __ldg(ccol + (long long)j * ld + e);
              }
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e) v[hb + q][e] = cv[q][e] > 0.0f ? v[hb + q][e] : 0.0f;
      }
      __syncthreads();  // the previous tile's readers are done
#pragma unroll
      for (int p = 0; p < 8; ++p)
        store_vec<4>(gt + (cg + 4 * p) * kGradPitch + rr, v[p]);
      for (int e = t; e < kGradCols * DIM; e += kGradRows)
        ys[e] = c0 + e / DIM < ce ? __ldg(P.y + I.y_off + (long long)c0 * DIM + e) : 0.0f;
      __syncthreads();
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float* const yp = ys + (cg + 4 * p) * DIM;
#pragma unroll
        for (int e = 0; e < 4; ++e) rs[e] += v[p][e];
#pragma unroll
        for (int k = 0; k < DIM; k += 4) {
          const float4 y4 = *reinterpret_cast<const float4*>(yp + k);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ax[e][k] = fmaf(v[p][e], y4.x, ax[e][k]);
            ax[e][k + 1] = fmaf(v[p][e], y4.y, ax[e][k + 1]);
            ax[e][k + 2] = fmaf(v[p][e], y4.z, ax[e][k + 2]);
            ax[e][k + 3] = fmaf(v[p][e], y4.w, ax[e][k + 3]);
          }
        }
      }
      if (rg < S::RG) {
        float ay[2][8], cs[2] = {0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < 8; ++k) ay[0][k] = ay[1][k] = 0.0f;
        constexpr int SPAN = kGradRows / S::RG;
#pragma unroll 2
        for (int r = rg * SPAN; r < (rg + 1) * SPAN; r += 4) {
          const float4 ga = *reinterpret_cast<const float4*>(gt + cp * kGradPitch + r);
          const float4 gb = *reinterpret_cast<const float4*>(gt + (cp + 16) * kGradPitch + r);
          const float a4[4] = {ga.x, ga.y, ga.z, ga.w}, b4[4] = {gb.x, gb.y, gb.z, gb.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float* const xp = xs + (r + e) * DIM + ks * 8;
            const float4 u = *reinterpret_cast<const float4*>(xp);
            const float4 w = *reinterpret_cast<const float4*>(xp + 4);
            const float x8[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
            cs[0] += a4[e];
            cs[1] += b4[e];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              ay[0][k] = fmaf(a4[e], x8[k], ay[0][k]);
              ay[1][k] = fmaf(b4[e], x8[k], ay[1][k]);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float* const s = sh + (rg * kGradCols + cp + 16 * q) * (DIM + 1);
#pragma unroll
          for (int k = 0; k < 8; ++k) s[ks * 8 + k] = ay[q][k];
          if (ks == 0) s[DIM] = cs[q];
        }
      }
      __syncthreads();
      {
        // the band's partials of the tile's columns (contiguous in memory)
        const int live = min(kGradCols, ce - c0) * (DIM + 1);
        float* const pp = P.part + I.py_off + ((long long)band * n + c0) * (DIM + 1);
        for (int e = t; e < live; e += kGradRows) {
          float s = sh[e];
#pragma unroll
          for (int q = 1; q < S::RG; ++q) s += sh[q * kGradCols * (DIM + 1) + e];
          pp[e] = s;
        }
      }
    }
    // the column groups' row sums, one group after the other
    float* const acc = gsm;  // [kGradRows][DIM + 1]
    for (int q = 0; q < 4; ++q) {
      __syncthreads();
      if (cg == q) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float* const a = acc + (rr + e) * (DIM + 1);
#pragma unroll
          for (int k = 0; k < DIM; ++k) a[k] = q ? a[k] + ax[e][k] : ax[e][k];
          a[DIM] = q ? a[DIM] + rs[e] : rs[e];
        }
      }
    }
    __syncthreads();
    const int live = min(kGradRows, m - r0) * (DIM + 1);
    float* const pp = P.part + I.px_off + ((long long)chunk * m + r0) * (DIM + 1);
    for (int e = t; e < live; e += kGradRows) pp[e] = acc[e];
    __syncthreads();  // before the next chunk's tiles
  }
}

// dL/dx_i from the chunks' partials and dL/dy_j from the bands', added in
// order; a thread per component.
template <int DIM>
__global__ void cost_grad_reduce_kernel(const __grid_constant__ GradParams P) {
  const GradInst& I = P.inst[blockIdx.y];
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
       e < (long long)(I.m + I.n) * DIM; e += step) {
    const bool is_x = e < (long long)I.m * DIM;
    const long long o = is_x ? e : e - (long long)I.m * DIM;
    const long long pt = o / DIM;
    const int k = (int)(o - pt * DIM);
    const int parts = is_x ? I.chunks : I.bands, count = is_x ? I.m : I.n;
    const float* pp = P.part + (is_x ? I.px_off : I.py_off) + pt * (DIM + 1);
    float a = 0.0f, s = 0.0f;
#pragma unroll 4
    for (int b = 0; b < parts; ++b, pp += (long long)count * (DIM + 1)) {
      a += __ldcg(pp + k);
      s += __ldcg(pp + DIM);
    }
    const float v = __ldg((is_x ? P.x + I.x_off : P.y + I.y_off) + o);
    (is_x ? P.gx + I.x_off : P.gy + I.y_off)[o] = P.scale2 * fmaf(v, s, -a);
  }
}

static size_t grad_smem_bytes(int dim) {
  return sizeof(float) * (size_t)(dim == 8 ? GradShape<8>::FLOATS
                                  : dim == 16 ? GradShape<16>::FLOATS
                                  : dim == 24 ? GradShape<24>::FLOATS : GradShape<32>::FLOATS);
}

// Tiles per chunk: the CTAs fill whole waves as nearly as they can (every tile
// costs about the same; a chunk's start about 0.7 of one).  4000 x 3000, d =
// 16: 5 tiles, 304 CTAs in one wave.
static int grad_chunk_tiles(int n_inst, const drot_cost_instance* inst, int dim) {
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    sms = 152;
  }
  const long long slots = (dim <= 16 ? 2LL : 1LL) * sms;
  int best = 1;
  double best_cost = 0.0;
  for (int k = 1; k <= 64; ++k) {
    long long ctas = 0;
    for (int q = 0; q < n_inst; ++q) {
      const long long tiles = ((long long)inst[q].n + kGradCols - 1) / kGradCols;
      ctas += ((long long)inst[q].m + kGradRows - 1) / kGradRows * ((tiles + k - 1) / k);
    }
    const double cost = (double)((ctas + slots - 1) / slots) * (k + 0.7);
    if (k == 1 || cost < best_cost) {
      best = k;
      best_cost = cost;
    }
  }
  return best;
}

// Partials layout; returns the floats they need (0: invalid descriptors).
static long long grad_layout(int n_inst, const drot_cost_instance* inst, int dim, GradParams* P) {
  long long part = 0;
  for (int k = 0; k < n_inst; ++k) {
    const drot_cost_instance& a = inst[k];
    if (a.m <= 0 || a.n <= 0 || a.ld < a.m || a.x_offset < 0 || a.y_offset < 0 || a.c_offset < 0)
      return 0;
  }
  const int chunk_cols = kGradCols * grad_chunk_tiles(n_inst, inst, dim);
  if (P) P->chunk_cols = chunk_cols;
  for (int k = 0; k < n_inst; ++k) {
    const drot_cost_instance& a = inst[k];
    const int bands = (a.m + kGradRows - 1) / kGradRows;
    const int chunks = (a.n + chunk_cols - 1) / chunk_cols;
    if (P) {
      GradInst& I = P->inst[k];
      I.x_off = a.x_offset * dim;
      I.y_off = a.y_offset * dim;
      I.c_off = a.c_offset;
      I.py_off = part;
      I.px_off = part + (long long)bands * a.n * (dim + 1);
      I.m = a.m;
      I.n = a.n;
      I.ld = a.ld;
      I.bands = bands;
      I.chunks = chunks;
      I.aligned = (a.ld % 4 == 0) && (a.c_offset % 4 == 0);
    }
    part += ((long long)bands * a.n + (long long)chunks * a.m) * (dim + 1);
  }
  return part;
}

}  // namespace drot

using namespace drot;

extern "C" {

size_t drot_sqeuclidean_cost_grad_workspace_bytes(int n_inst, const drot_cost_instance* inst,
                                                  int dim) {
  if (n_inst <= 0 || n_inst > kCostMaxInst || !inst || dim <= 0 || dim > 32 || (dim & 7))
    return 0;
  const long long f = grad_layout(n_inst, inst, dim, nullptr);
  return f > 0 ? (size_t)f * sizeof(float) : 0;
}

int drot_sqeuclidean_cost_grad(int n_inst, const drot_cost_instance* inst, const float* x,
                               const float* y, int dim, float scale, const float* c,
                               const float* grad_c, float* grad_x, float* grad_y,
                               void* workspace, size_t workspace_bytes, drot_stream_t stream) {
  if (n_inst <= 0 || n_inst > kCostMaxInst || !inst || !x || !y || !grad_c || !grad_x ||
      !grad_y || !workspace)
    return DROT_ERR_INVALID_ARG;
  if (dim <= 0 || dim > 32 || (dim & 7) != 0) return DROT_ERR_UNSUPPORTED;
  if (((uintptr_t)grad_c & 15u) || (c && ((uintptr_t)c & 15u))) return DROT_ERR_INVALID_ARG;
  static GradParams P;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  memset(&P, 0, sizeof(P));
  const long long nf = grad_layout(n_inst, inst, dim, &P);
  if (nf <= 0) return DROT_ERR_INVALID_ARG;
  if (workspace_bytes < (size_t)nf * sizeof(float)) return DROT_ERR_WORKSPACE;
  int max_bands = 0, max_chunks = 0;
  long long max_points = 0;
  for (int k = 0; k < n_inst; ++k) {
    max_bands = std::max(max_bands, P.inst[k].bands);
    max_chunks = std::max(max_chunks, P.inst[k].chunks);
    max_points = std::max(max_points, (long long)P.inst[k].m + P.inst[k].n);
  }
  P.x = x;
  P.y = y;
  P.g = grad_c;
  P.c = c;
  P.gx = grad_x;
  P.gy = grad_y;
  P.part = (float*)workspace;
  P.n_inst = n_inst;
  P.scale2 = 2.0f * scale;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = grad_smem_bytes(dim);
  const void* k1 = dim == 8 ? (const void*)cost_grad_kernel<8>
                 : dim == 16 ? (const void*)cost_grad_kernel<16>
                 : dim == 24 ? (const void*)cost_grad_kernel<24>
                             : (const void*)cost_grad_kernel<32>;
  const void* k2 = dim == 8 ? (const void*)cost_grad_reduce_kernel<8>
                 : dim == 16 ? (const void*)cost_grad_reduce_kernel<16>
                 : dim == 24 ? (const void*)cost_grad_reduce_kernel<24>
                             : (const void*)cost_grad_reduce_kernel<32>;
  if (cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return DROT_ERR_CUDA;
  void* args[] = {(void*)&P};
  if (cudaLaunchKernel(k1, dim3(max_bands, std::min(max_chunks, 65535), n_inst), dim3(kGradRows), args, smem, st) !=
          cudaSuccess ||
      cudaLaunchKernel(k2, dim3((unsigned)std::min<long long>((max_points * dim + 255) / 256, 608),
                                n_inst), dim3(256),
                       args, 0, st) != cudaSuccess) {
    cudaGetLastError();
    return DROT_ERR_CUDA;
  }
  return DROT_OK;
}


int drot_sqeuclidean_cost(int n_inst, const drot_cost_instance* inst, const float* x,
                          const float* y, int dim, float scale, int clamp, float* c,
                          drot_stream_t stream) {
  if (n_inst <= 0 || n_inst > kCostMaxInst || !inst || !x || !y || !c) return DROT_ERR_INVALID_ARG;
  if (dim <= 0 || dim > 32 || (dim & 7) != 0) return DROT_ERR_UNSUPPORTED;
  if (((uintptr_t)x & 15u) || ((uintptr_t)y & 15u)) return DROT_ERR_INVALID_ARG;
  // The parameter block (descriptors included) is about 12 KB: kept off the
  // stack, filled and launched under a lock (launch copies it).
  static CostParams P;
  static int* err_flag[64] = {};
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return DROT_ERR_CUDA;
  if (!err_flag[dev] && cudaMalloc(&err_flag[dev], sizeof(int)) != cudaSuccess) return DROT_ERR_CUDA;
  int* err = err_flag[dev];
  memset(&P, 0, sizeof(P));
  long long total_tiles = 0;
  for (int k = 0; k < n_inst; ++k) {
    const drot_cost_instance& a = inst[k];
    if (a.m <= 0 || a.n <= 0 || a.ld < a.m || a.x_offset < 0 || a.y_offset < 0 ||
        a.c_offset < 0 || ((a.x_offset * dim) & 3) || ((a.y_offset * dim) & 3))
      return DROT_ERR_INVALID_ARG;
    CostInst& I = P.inst[k];
    I.x_off = a.x_offset * dim;
    I.y_off = a.y_offset * dim;
    I.c_off = a.c_offset;
    I.m = a.m;
    I.n = a.n;
    I.ld = a.ld;
    I.tiles_m = (a.m + kCostM - 1) / kCostM;
    const long long tiles = (long long)I.tiles_m * ((a.n + kCostN - 1) / kCostN);
    if (tiles > 65535LL * 1024) return DROT_ERR_UNSUPPORTED;
    I.tiles = (int)tiles;
    I.tile0 = (int)total_tiles;
    total_tiles += tiles;
    if (total_tiles > (1LL << 30)) return DROT_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  P.x = x;
  P.y = y;
  P.c = c;
  P.err = err;
  P.timeout_ns = 2000000000LL;
  P.dim = dim;
  P.n_inst = n_inst;
  P.clamp = clamp ? 1 : 0;
  P.scale = scale;
  P.total_tiles = (int)total_tiles;
  const size_t smem = cost_smem_bytes(dim);
  if (cudaFuncSetAttribute((const void*)cost_sqeuclid_kernel,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute((const void*)cost_sqeuclid_kernel,
                           cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return DROT_ERR_CUDA;
  // Persistent grid of two CTAs per SM: each holds 256 of the SM's 512 TMEM
  // columns, and the registers (under 128 per thread, 256 threads) and
  // shared memory (under 100 KB at d <= 24) of two fit an SM.  CTAs that do
  // not fit (d = 32) start when one finishes; the tile stride keeps every
  // tile covered either way.
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return DROT_ERR_CUDA;
  const int grid = (int)std::min<long long>(total_tiles, 2LL * sms);
  if (cudaMemsetAsync(err, 0, sizeof(int), st) != cudaSuccess) return DROT_ERR_CUDA;
  cost_sqeuclid_kernel<<<grid, kCostThreads, smem, st>>>(P);
  if (cudaGetLastError() != cudaSuccess) return DROT_ERR_CUDA;
  int h_err = 0;
  if (cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return DROT_ERR_CUDA;
  return h_err ? DROT_ERR_BARRIER_TIMEOUT : DROT_OK;
}

}  // extern "C"

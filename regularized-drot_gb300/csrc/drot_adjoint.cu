// drot_adjoint.cu -- implicit adjoint of the quadratic-regularised DROT plan.
//
// No counterpart in the reference (its operators return plans without
// autograd, pytorch/src/drot_cuda.cpp:26-44).  At the solution of
//     min <C, X> + (lambda / 2) ||X||_F^2  s.t.  X 1 = p, X^T 1 = q, X >= 0
// (the fixed point of the QR iteration, lambda = (kappa - 1) / s), the plan on
// its support S is X_ij = (u_i + v_j - C_ij) / lambda.  Differentiating the
// marginal constraints on a fixed support gives, for an upstream gradient
// G = dL/dX, the adjoint system
//     [ D_r  M  ] [a]   [ rowsum(G o M) ]
//     [ M^T  D_c] [b] = [ colsum(G o M) ]
// with M the 0/1 support mask and D_r, D_c its row / column counts; then
// dL/dC = (a_i + b_j - G_ij) / lambda on S (0 elsewhere), dL/dp = a,
// dL/dq = b.  The matrix is a graph Laplacian (of the bipartite support
// graph, after b -> -b): singular but the right-hand side is consistent, so
// conjugate gradients converge; a and b are determined up to a + t, b - t.
//
// The support is read off the duals, not off X: at the fixed point of
// X = max(X + phi1 + phi2 - sC, 0) / kappa the plan is positive exactly where
// D_ij = phi1_i + phi2_j - s C_ij > 0, while a finite solve still carries
// entries of X that decay geometrically towards 0 off the support (tiny but
// positive); counting those would add wrong equations to the system.
//
// Kernels here:
//   adj_mask_kernel  -- the support bitmasks of D > 0 in both layouts
//                       (column words: 32 rows of a column; row words: 32
//                       columns of a row) and a byte mask in the layout of C,
//                       one warp per 32 x 32 block.
//   adj_pcg_kernel   -- Jacobi-preconditioned CG for a batch of instances in
//                       one persistent cooperative launch.  The matvec
//                       multiplies the bit masks with the digits of the
//                       search direction on the tensor cores, exactly.
//                       Two grid barriers per iteration; each instance
//                       stops on its own relative residual.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <queue>
#include <utility>
#include <vector>

#include "drot_gb300.h"
#include "drot_kernels.cuh"
#include "drot_launch.h"

namespace drot {

struct AdjInst {
  long long c_off;   // element offset of C (column-major, leading dimension ld)
  long long f1_off, f2_off;  // offsets of the instance's phi1 / phi2
  long long mc_off;  // word offset of the column-word mask [nc][nwr]
  long long mr_off;  // word offset of the row-word mask [nr][nwc]
  int nr, nc, ld, nwr, nwc;
  int v_off;         // offset of [a; b] in the packed vectors (nr + nc entries)
  int seg0, nseg;    // its segments (contiguous)
  int owner;         // CTA that counts its convergence
  float s;           // step size of the solve
  float lam;         // regularisation weight lambda = (kappa - 1) / s
};

struct AdjSeg {
  int inst, l0, l1, cta;  // lines [l0, l1) of instance inst, processed by CTA cta
};

struct AdjParams {
  const void* c;
  int c_bf16;
  const float *phi1, *phi2;
  unsigned char* mask;  // byte mask, layout of C (may be null)
  const float* g;       // upstream gradient dL/dX, layout of C
  double* z;            // solution [a; b]
  double *r, *d0, *d1, *q, *invdiag, *deg, *y;  // y = M^-1 r
  unsigned *mcol, *mrow;
  const AdjInst* inst;
  const AdjSeg* seg;
  const int* cta_seg0;  // [grid + 1]: the segments of CTA c are cta_seg0[c] .. cta_seg0[c+1]
  double* slot_dq;      // per segment: d.q
  double* slot_ry;      // [2][n_seg]: r.y (y = M^-1 r), by iteration parity
  double* slot_rr;      // [2][n_seg]: r.r, by iteration parity
  double* slot_rr0;     // per segment: initial r.r
  int* iters;           // per instance: CG iterations run
  int* conv;            // per instance: converged flag (owner CTA only)
  double* relres;       // per instance: final relative residual ||r|| / ||r0||
  unsigned* conv_count;
  unsigned* bar;
  int* abort_flag;
  long long timeout_ns;
  int n_inst, n_seg, max_iters;
  int chunk;            // entries staged as digits at a time, a multiple of 32
  int max_lines;        // lines of the largest instance
  double tol;
};

// ---------------------------------------------------------------------------
// support masks
// ---------------------------------------------------------------------------

// grid: (blocks, n_inst); a warp per 32 x 32 block (row word w, column word v).
__global__ void adj_mask_kernel(const AdjParams A) {
  const int k = blockIdx.y;
  const AdjInst I = A.inst[k];
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const long long nblk = (long long)I.nwr * I.nwc;
  for (long long blk = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); blk < nblk;
       blk += (long long)gridDim.x * wpb) {
    const int w = (int)(blk % I.nwr);  // row word
    const int v = (int)(blk / I.nwr);  // column word
    const int i = w * 32 + lane;
    const float f1 = i < I.nr ? __ldg(A.phi1 + I.f1_off + i) : 0.0f;
    unsigned mine = 0u, rowword = 0u;
    for (int c = 0; c < 32; ++c) {
      const int j = v * 32 + c;
      bool on = false;
      if (i < I.nr && j < I.nc) {
        const long long e = I.c_off + (long long)j * I.ld + i;
        const float cv = A.c_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(A.c)[e])
                                  : __ldg(reinterpret_cast<const float*>(A.c) + e);
        const float f2 = __ldg(A.phi2 + I.f2_off + j);
        on = fmaf(-I.s, cv, f1 + f2) > 0.0f;
        if (A.mask) A.mask[e] = on ? 1 : 0;
      }
      const unsigned word = __ballot_sync(0xffffffffu, on);
      if (lane == c) mine = word;
      rowword |= ((word >> lane) & 1u) << c;
    }
    const int j = v * 32 + lane;
    if (j < I.nc) A.mcol[I.mc_off + (long long)j * I.nwr + w] = mine;
    if (i < I.nr) A.mrow[I.mr_off + (long long)i * I.nwc + v] = rowword;
  }
}

// ---------------------------------------------------------------------------
// batched PCG (FP64 vectors)
// ---------------------------------------------------------------------------

// The matvec: for every line, the sum of the direction's entries over the set
// bits of the line's mask words.  FP64 adds are slow on this part (a warp's add
// takes 16 clocks of an SM), and adding set bit by set bit cost 110 us per CG
// iteration at 11 M elements.  Here the sums are integer sums on the tensor
// cores: the entries are written as 88-bit fixed-point numbers on the scale of
// the instance's largest one, cut into 8 digits of 11 bits, and the product of
// the 0 / 1 mask (A: 16 lines x 16 entries) with the digits (B: 16 entries x 8
// digits) is an FP16 MMA with FP32 accumulation whose every partial sum is an
// integer below 2^23 times 2^-24, so nothing is rounded.  The digit sums are
// added up as 64-bit integers and rounded to FP64 (three times at most), and do
// not depend on their order.
//   Entries down to 2^-35 of the largest (its power of two, 2^E) are exact in
// that, smaller ones cut below 2^(E-87).  The cut of a line's k entries, k
// 2^(E-87) at most, is below one rounding of an FP64 sum of them unless they all
// are small.  Those lines -- the line's own entry below 2^(E-34) and its sum
// below k 2^(E-34): in a component of the support graph whose right-hand side is
// small beside the others' -- are added entry by entry in FP64 instead
// (line_walk), where an instance has entries that are cut at all: every line has
// the accuracy of an FP64 sum of its own entries.
//
// One mask word (32 entries of a line) is two MMAs.  Their k indices are dealt
// out so that a lane's operand is one AND: register r (0..3: the two halves of
// the first MMA's k, then the second's) of thread-in-group t holds bits 4 t + r
// and 4 t + r + 16, as the FP16 numbers 2^(r - 24); the digits carry 2^-r.
//
// us per CG iteration (a solve's time over its iterations), bits walked -> here: 8
// instances of 512..2048 rows and columns with 0.5 % of the entries on the support
// 89 -> 19, with 0.15 % 101 -> 18; one of 200 x 200 35 -> 18; 64 of 512..4096 with
// 1 % 257 -> 133.
constexpr int kAdjThreads = 512;
constexpr int kAdjChunk = 4096;     // entries whose digits are staged at a time, at most
constexpr int kAdjBlock = 512;      // lines whose sums are held at a time
constexpr int kAdjDigitBytes = 16;  // of a staged entry

__device__ __forceinline__ void mma_mask(float (&c)[4], unsigned a0, unsigned a1, unsigned a2,
                                         unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
               "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// |v| on the scale of exponent field emax as 88 bits in two halves of 44.
__device__ __forceinline__ void to_fixed88(double v, int emax, unsigned long long& hi,
                                           unsigned long long& lo) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int e = (int)((bits >> 52) & 0x7ffu);
  const unsigned long long m = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
  const int sh = emax - e;
  const unsigned long long mask = (1ull << 44) - 1ull;
  hi = sh < 44 ? m >> (9 + sh) : 0ull;
  lo = (sh <= 35 ? m << (35 - sh) : (sh < 88 ? m >> (sh - 35) : 0ull)) & mask;
  if (e == 0) hi = lo = 0ull;  // zero (and subnormal)
}

// Digits of the entries v[0 .. n), n <= kAdjChunk, zero up to whole words, as
// B operands: word w, lane (digit g, t), register r at [w][4 g + t][r].
__device__ __forceinline__ void stage_digits(const double* v, int n, int emax, unsigned* B) {
  const int pairs = (n + 31) / 32 * 16;
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
    const int w = i >> 4, k = i & 15;  // entries 32 w + k and + 16
    const int j0 = 32 * w + k, j1 = j0 + 16;
    const double v0 = j0 < n ? v[j0] : 0.0, v1 = j1 < n ? v[j1] : 0.0;
    unsigned long long h0, l0, h1, l1;
    to_fixed88(v0, emax, h0, l0);
    to_fixed88(v1, emax, h1, l1);
    // +- 2^-r, in both halves
    const unsigned r = k & 3, one = 0x3c00u - (r << 10);
    const unsigned sc = (one | (v0 < 0.0 ? 0x8000u : 0u)) |
                        ((one | (v1 < 0.0 ? 0x8000u : 0u)) << 16);
    const __half2 scale = *reinterpret_cast<const __half2*>(&sc);
    unsigned* const to = B + w * 128 + (k >> 2) * 4 + r;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int s = 33 - 11 * (g & 3);
      const unsigned d0 = (unsigned)((g < 4 ? h0 : l0) >> s) & 0x7ffu;
      const unsigned d1 = (unsigned)((g < 4 ? h1 : l1) >> s) & 0x7ffu;
      // 1024 + the digit's low 10 bits has those as its low bits; less 1024 where
      // the digit's top bit is clear
      const unsigned u = 0x64006400u | (d0 & 0x3ffu) | (d1 & 0x3ffu) << 16;
      const unsigned t = ((d0 >> 10) ^ 1u) * 0x6400u | ((d1 >> 10) ^ 1u) * 0x64000000u;
      const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&u),
                                *reinterpret_cast<const __half2*>(&t));
      const __half2 y = __hmul2(x, scale);
      to[g * 16] = *reinterpret_cast<const unsigned*>(&y);
    }
  }
}

// Adds the digit sums of `n` lines (n <= kAdjBlock; line l's mask words at
// words[l * stride + w], w < nw the ones of the staged entries) to acc[l][4]:
// pairs of digits as integers.  A warp takes 16 lines and a share of the words.
__device__ __forceinline__ void mask_sums(const unsigned* words, int stride, int n, int nw,
                                          const unsigned* B, unsigned long long* acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int groups = (n + 15) / 16;
  int ks = 1;
  while (2 * ks * groups <= W && 8 * ks < nw) ks *= 2;
  for (int task = warp; task < groups * ks; task += W) {
    const int grp = task / ks, part = task - grp * ks;
    const int w0 = nw * part / ks, w1 = nw * (part + 1) / ks;
    const int la = grp * 16 + g, lb = la + 8;
    const unsigned* const pa = words + (long long)min(la, n - 1) * stride;
    const unsigned* const pb = words + (long long)min(lb, n - 1) * stride;
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int w = w0; w < w1; w += 4) {
      unsigned xa[4], xb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        xa[u] = w + u < w1 ? __ldg(pa + w + u) >> (4 * t) : 0u;
        xb[u] = w + u < w1 ? __ldg(pb + w + u) >> (4 * t) : 0u;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (w + u >= w1) break;
        const uint4 b = *reinterpret_cast<const uint4*>(B + (w + u) * 128 + lane * 4);
        const unsigned a = xa[u], d = xb[u];
        mma_mask(c, a & 0x00010001u, d & 0x00010001u, a & 0x00020002u, d & 0x00020002u, b.x, b.y);
        mma_mask(c, a & 0x00040004u, d & 0x00040004u, a & 0x00080008u, d & 0x00080008u, b.z, b.w);
      }
    }
    // c[0], c[1]: digits 2 t, 2 t + 1 of line la; c[2], c[3]: of line lb
    const long long sa = (long long)(int)(c[0] * 16777216.0f) * 2048 + (int)(c[1] * 16777216.0f);
    const long long sb = (long long)(int)(c[2] * 16777216.0f) * 2048 + (int)(c[3] * 16777216.0f);
    if (la < n) atomicAdd(acc + 4 * la + t, (unsigned long long)sa);
    if (lb < n) atomicAdd(acc + 4 * lb + t, (unsigned long long)sb);
  }
}

// The FP64 value of a line's digit sums.
__device__ __forceinline__ double mask_sum_value(const unsigned long long* acc, int emax) {
  double s = (double)(long long)acc[0] * 73786976294838206464.0;     // 2^66
  s = fma((double)(long long)acc[1], 17592186044416.0, s);           // 2^44
  s = fma((double)(long long)acc[2], 4194304.0, s) + (double)(long long)acc[3];
  return emax == 0x7ff ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(s, emax - 1110);
}

// A warp: the sum over the set bits of a line's nw mask words of the entries src,
// in FP64.  nz: a bit per entry, set where it is not zero; src's first is bit
// `shift` of nz[0].
__device__ __noinline__ double line_walk(const unsigned* words, int nw, const double* src,
                                         const unsigned* nz, int shift) {
  double s = 0.0;
  bool any = false;
  for (int w = threadIdx.x & 31; w < nw; w += 32) {
    unsigned m = __ldg(words + w) & __funnelshift_r(nz[w], nz[w + 1], shift);
    any |= m != 0u;
    for (; m; m &= m - 1u) s += src[32 * w + __ffs(m) - 1];
  }
  return __any_sync(0xffffffffu, any) ? warp_sum_d(s) : 0.0;
}

// Degree of line l and the right-hand side entry of the adjoint system: the
// sum of the upstream gradient g over the line's support (rowsum(g o M) for
// a row, colsum(g o M) for a column), in FP64.  Lanes split the mask words;
// fixed shuffle trees, so the result is deterministic.
__device__ __forceinline__ void line_degree_rhs(const AdjParams& A, const AdjInst& I, int l,
                                                int lane, int& deg, double& rhs) {
  int c = 0;
  double s = 0.0;
  const float* g = A.g + I.c_off;
  if (l < I.nr) {  // row i = l: set bits are columns j, g at j * ld + i (strided gather)
    const unsigned* words = A.mrow + I.mr_off + (long long)l * I.nwc;
    for (int w = lane; w < I.nwc; w += 32) {
      unsigned m = __ldcg(words + w);
      c += __popc(m);
      while (m) {
        const int j = 32 * w + __ffs(m) - 1;
        s += (double)__ldg(g + (long long)j * I.ld + l);
        m &= m - 1u;
      }
    }
  } else {  // column j = l - nr: set bits are rows i, g contiguous down the column
    const int j = l - I.nr;
    const unsigned* words = A.mcol + I.mc_off + (long long)j * I.nwr;
    const float* gc = g + (long long)j * I.ld;
    for (int w = lane; w < I.nwr; w += 32) {
      unsigned m = __ldcg(words + w);
      c += __popc(m);
      while (m) {
        const int i = 32 * w + __ffs(m) - 1;
        s += (double)__ldg(gc + i);
        m &= m - 1u;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  deg = c;
  rhs = warp_sum_d(s);
}

// A warp: sum over the segments of an instance of slot[] (fixed order).
__device__ __forceinline__ double inst_sum(const double* slot, const AdjInst& I) {
  double s = 0.0;
  for (int t = threadIdx.x & 31; t < I.nseg; t += 32) s += __ldcg(slot + I.seg0 + t);
  return warp_sum_d(s);
}

// Block sums of one value per line of an n-line segment (thread i has lines i,
// i + blockDim.x, ...): only the warps that have lines take part.  Thread 0
// receives them.  Fixed trees.
template <int N>
__device__ __forceinline__ void line_sums(double (&v)[N], int n, double (*scratch)[16]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int active = min((int)blockDim.x >> 5, (n + 31) >> 5);
  if (w < active) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      v[k] = warp_sum_d(v[k]);
      if (lane == 0) scratch[k][w] = v[k];
    }
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = warp_sum_d(lane < active ? scratch[k][lane] : 0.0);
  }
}

// Vectors (r, d, q, z) and the staged direction are FP64: the adjoint system
// is a graph Laplacian whose support graph is often close to a forest (as
// many edges as vertices), so it is badly conditioned, and an FP32 CG stops
// at a solution error far above its residual.  The FP64 work is O(lines) vector
// updates; the scalars of an instance are one warp's work each (a division by
// every warp of the CTA took 3000 clocks).
__global__ void __launch_bounds__(kAdjThreads, 1) adj_pcg_kernel(const AdjParams A) {
  extern __shared__ __align__(16) unsigned char adj_smem[];
  unsigned long long* const acc = reinterpret_cast<unsigned long long*>(adj_smem);  // [kAdjBlock][4]
  unsigned* const digits = reinterpret_cast<unsigned*>(acc + 4 * kAdjBlock);  // [A.chunk] entries
  double* const sv = reinterpret_cast<double*>(
      adj_smem + 32 * kAdjBlock + (size_t)kAdjDigitBytes * A.chunk);  // the staged direction
  unsigned* const nz = reinterpret_cast<unsigned*>(sv + A.max_lines);  // bits of its nonzeros
  __shared__ int s_flag, s_emax;
  __shared__ unsigned s_emin;
  __shared__ double s_red[32 + 1];
  __shared__ double s_part[2][16];
  __shared__ double s_step;  // beta, then alpha
  __shared__ int s_done;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int sg0 = A.cta_seg0[blockIdx.x], sg1 = A.cta_seg0[blockIdx.x + 1];
  const double tol2 = A.tol * A.tol;
  unsigned epoch = 0;

  // Prologue: degrees, the right-hand side from g, r = rhs, z = 0; parity-0
  // slots r.y and r.r.
  for (int sg = sg0; sg < sg1; ++sg) {
    const AdjSeg S = A.seg[sg];
    const AdjInst I = A.inst[S.inst];
    double ry = 0.0, rr = 0.0;
    for (int l = S.l0 + warp; l < S.l1; l += W) {
      int dg;
      double rhs;
      line_degree_rhs(A, I, l, lane, dg, rhs);
      if (lane == 0) {
        const int gi = I.v_off + l;
        const double inv = dg > 0 ? 1.0 / (double)dg : 0.0;
        const double r0 = dg > 0 ? rhs : 0.0;
        A.invdiag[gi] = inv;
        A.deg[gi] = (double)dg;
        A.r[gi] = r0;
        A.y[gi] = inv * r0;
        A.z[gi] = 0.0;
        ry += r0 * (inv * r0);
        rr += r0 * r0;
      }
    }
    ry = block_sum_d(ry, s_red);
    rr = block_sum_d(rr, s_red);
    if (threadIdx.x == 0) {
      A.slot_ry[sg] = ry;
      A.slot_rr[sg] = rr;
      A.slot_rr0[sg] = rr;
    }
  }
  if (!grid_barrier(A.bar, A.abort_flag, A.timeout_ns, epoch, &s_flag)) return;

  int it = 0;
  for (; it < A.max_iters; ++it) {
    const int par = it & 1;
    double* dcur = par ? A.d1 : A.d0;
    const double* dold = par ? A.d0 : A.d1;
    const double* ry_cur = A.slot_ry + (size_t)par * A.n_seg;
    const double* ry_prev = A.slot_ry + (size_t)(par ^ 1) * A.n_seg;
    const double* rr_cur = A.slot_rr + (size_t)par * A.n_seg;

    // ---- phase A: d = y + beta d_old (staged), q = A d on this CTA's lines
    for (int sg = sg0; sg < sg1; ++sg) {
      const AdjSeg S = A.seg[sg];
      const int k = S.inst;
      const AdjInst I = A.inst[k];
      __syncthreads();  // the sums and staged vectors of the segment before are read
      if (warp == 0) {
        const double rr = inst_sum(rr_cur, I), rr0 = inst_sum(A.slot_rr0, I);
        if (lane == 0) s_done = !(rr > tol2 * rr0);
      } else if (warp == 1 && it > 0) {
        const double ry = inst_sum(ry_cur, I), ryp = inst_sum(ry_prev, I);
        if (lane == 0) s_step = ry / ryp;
      } else if (threadIdx.x == 64) {
        s_emax = 0;
        s_emin = 0xfffu;
      }
      __syncthreads();
      if (s_done) {
        if (sg == I.seg0 && threadIdx.x == 0 && !A.conv[k]) {
          A.conv[k] = 1;
          atomicAdd(A.conv_count, 1u);
        }
        continue;
      }
      const double beta = it == 0 ? 0.0 : s_step;
      const int nv = I.nr + I.nc;
      // Stage d = y + beta d_old for the whole instance: a thread takes 4
      // entries and issues their loads before using any.
      // upper words of the largest magnitude and of the smallest that is not zero
      // (less one, which puts zero last; an upper word of zero beside a lower one
      // that is not is a subnormal, which counts as zero)
      unsigned top = 0u, bottom = 0xffffffffu;
      for (int t0 = threadIdx.x; t0 < nv; t0 += 4 * blockDim.x) {
        double yv[4], dv0[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int t = t0 + u * blockDim.x;
          const int gi = I.v_off + (t < nv ? t : 0);
          yv[u] = __ldcg(A.y + gi);
          dv0[u] = it == 0 ? 0.0 : __ldcg(dold + gi);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int t = t0 + u * blockDim.x;
          if (t >= nv) break;
          const double dv = it == 0 ? yv[u] : fma(beta, dv0[u], yv[u]);
          sv[t] = dv;
          const unsigned size = (unsigned)__double2hiint(dv) & 0x7fffffffu;
          top = max(top, size);
          bottom = min(bottom, size - 1u);
          if (t >= S.l0 && t < S.l1) dcur[I.v_off + t] = dv;
        }
      }
      top = __reduce_max_sync(0xffffffffu, top);
      bottom = __reduce_min_sync(0xffffffffu, bottom);
      if (lane == 0) {
        atomicMax(&s_emax, (int)(top >> 20));
        atomicMin(&s_emin, bottom >> 20);
      }
      __syncthreads();
      const int emax = s_emax;
      // 2^(E-34) of the lines that are added in FP64, where entries are cut
      const double low = emax > 36 && emax < 0x7ff && s_emin < (unsigned)(emax - 35)
                             ? __hiloint2double((emax - 34) << 20, 0) : 0.0;
      if (low > 0.0) {  // the nonzeros of the direction, for line_walk
        for (int t0 = 32 * warp; t0 < nv; t0 += blockDim.x) {
          const unsigned b = __ballot_sync(0xffffffffu, t0 + lane < nv && sv[t0 + lane] != 0.0);
          if (lane == 0) nz[t0 >> 5] = b;
        }
        __syncthreads();
      }
      double dq = 0.0;
      // the segment's rows against the column entries, then its columns
      // against the row entries
      for (int side = 0; side < 2; ++side) {
        const int a0 = side ? max(S.l0, I.nr) : S.l0, a1 = side ? S.l1 : min(S.l1, I.nr);
        const int K = side ? I.nr : I.nc, stride = side ? I.nwr : I.nwc;
        const double* const src = side ? sv : sv + I.nr;
        const unsigned* const words =
            side ? A.mcol + I.mc_off - (long long)I.nr * I.nwr : A.mrow + I.mr_off;
        for (int b0 = a0; b0 < a1; b0 += kAdjBlock) {
          const int n = min(kAdjBlock, a1 - b0);
          for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) acc[i] = 0ull;
          for (int k0 = 0; k0 < K; k0 += A.chunk) {
            const int kn = min(A.chunk, K - k0);
            // a single chunk stays staged for the blocks that follow
            if (K > A.chunk || b0 == a0) stage_digits(src + k0, kn, emax, digits);
            __syncthreads();
            mask_sums(words + (long long)b0 * stride + (k0 >> 5), stride, n, (kn + 31) >> 5,
                      digits, acc);
            __syncthreads();
          }
          const unsigned* const bits = side ? nz : nz + (I.nr >> 5);
          const int shift = side ? 0 : I.nr & 31;
          for (int i0 = 32 * warp; i0 < n; i0 += blockDim.x) {
            const int i = i0 + lane, l = b0 + i, gi = I.v_off + l;
            double dl = 0.0, dg = 0.0, sum = 0.0;
            if (i < n) {
              dl = sv[l];
              dg = __ldcg(A.deg + gi);
              sum = mask_sum_value(acc + 4 * i, emax);
            }
            unsigned todo = __ballot_sync(0xffffffffu, fabs(dl) < low && fabs(sum) < dg * low);
            for (; todo; todo &= todo - 1u) {
              const int k = __ffs(todo) - 1;
              const double t = line_walk(words + (long long)(b0 + i0 + k) * stride, (K + 31) >> 5,
                                         src, bits, shift);
              if (lane == k) sum = t;
            }
            if (i < n) {
              const double qv = fma(dg, dl, sum);
              A.q[gi] = qv;
              dq += dl * qv;
            }
          }
          __syncthreads();
        }
      }
      double sums[1] = {dq};
      line_sums(sums, min(S.l1 - S.l0, kAdjBlock), s_part);
      if (threadIdx.x == 0) A.slot_dq[sg] = sums[0];
    }
    if (!grid_barrier(A.bar, A.abort_flag, A.timeout_ns, epoch, &s_flag)) return;
    if (__ldcg(A.conv_count) >= (unsigned)A.n_inst) break;

    // ---- phase B: z += alpha d, r -= alpha q; next-parity slots r.y, r.r
    double* ry_next = A.slot_ry + (size_t)(par ^ 1) * A.n_seg;
    double* rr_next = A.slot_rr + (size_t)(par ^ 1) * A.n_seg;
    for (int sg = sg0; sg < sg1; ++sg) {
      const AdjSeg S = A.seg[sg];
      const AdjInst I = A.inst[S.inst];
      __syncthreads();
      if (warp == 0) {
        const double rr = inst_sum(rr_cur, I), rr0 = inst_sum(A.slot_rr0, I);
        if (lane == 0) s_done = !(rr > tol2 * rr0);
      } else if (warp == 1) {
        const double ry = inst_sum(ry_cur, I), dq = inst_sum(A.slot_dq, I);
        if (lane == 0) s_step = dq > 0.0 ? ry / dq : 0.0;
      }
      __syncthreads();
      if (s_done) {
        // Converged: carry this segment's r.y and r.r into the next parity's
        // slots, so the instance reads the same (converged) sums on every
        // later iteration and stays stopped.  Without the copy the next
        // iteration would read the slots of two iterations back, find the
        // instance unconverged and step it again with stale CG scalars.
        if (threadIdx.x == 0) {
          ry_next[sg] = __ldcg(ry_cur + sg);
          rr_next[sg] = __ldcg(rr_cur + sg);
        }
        continue;
      }
      const double alpha = s_step;
      double sums[2] = {0.0, 0.0};  // r.y, r.r
      for (int l = S.l0 + threadIdx.x; l < S.l1; l += blockDim.x) {
        const int gi = I.v_off + l;
        const double zl = fma(alpha, __ldcg(dcur + gi), A.z[gi]);
        const double rl = fma(-alpha, __ldcg(A.q + gi), A.r[gi]);
        A.z[gi] = zl;
        A.r[gi] = rl;
        const double yl = __ldcg(A.invdiag + gi) * rl;
        A.y[gi] = yl;
        sums[0] += rl * yl;
        sums[1] += rl * rl;
      }
      line_sums(sums, S.l1 - S.l0, s_part);
      if (threadIdx.x == 0) {
        ry_next[sg] = sums[0];
        rr_next[sg] = sums[1];
        if (sg == I.seg0) A.iters[S.inst] = it + 1;
      }
    }
    if (!grid_barrier(A.bar, A.abort_flag, A.timeout_ns, epoch, &s_flag)) return;
  }
  // Final relative residual of each instance, from the slots of the parity
  // the last phase A read (written, and made visible by a grid barrier,
  // before the loop ended); the CTA of the instance's first segment writes it.
  const double* rr_fin = A.slot_rr + (size_t)(it & 1) * A.n_seg;
  for (int sg = sg0; sg < sg1; ++sg) {
    const AdjSeg S = A.seg[sg];
    const AdjInst I = A.inst[S.inst];
    if (sg == I.seg0 && warp == 0) {
      const double r0 = inst_sum(A.slot_rr0, I), r = inst_sum(rr_fin, I);
      if (lane == 0) A.relres[S.inst] = r0 > 0.0 ? sqrt(r / r0) : 0.0;
    }
  }
}

// ---------------------------------------------------------------------------
// gradient assembly
// ---------------------------------------------------------------------------

// dL/dC = (a_i + b_j - g_ij) / lambda on the support, 0 elsewhere (FP64
// arithmetic on the support entries, rounded once), for every element of an
// instance's n_rows x n_cols block; grid (column blocks, instances), a warp
// per column, a lane per 4 rows (one 128-row chunk per step).  Off-support
// groups of 4 rows are written as zeros without reading g.  Block 0 of each
// instance also writes dL/dp = a + t, dL/dq = b - t with the gauge t =
// (sum b - sum a) / (n_rows + n_cols) (FP64 sums in a fixed order).
__global__ void __launch_bounds__(256) adj_grad_kernel(const AdjParams A, float* __restrict__ gc,
                                                       float* __restrict__ gp,
                                                       float* __restrict__ gq) {
  __shared__ double s_red[32 + 1];
  const int k = blockIdx.y;
  const AdjInst I = A.inst[k];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const double* za = A.z + I.v_off;
  const double* zb = za + I.nr;
  const double inv_lam = 1.0 / (double)I.lam;
  for (int j = blockIdx.x * W + warp; j < I.nc; j += gridDim.x * W) {
    const unsigned* words = A.mcol + I.mc_off + (long long)j * I.nwr;
    const float* gcol = A.g + I.c_off + (long long)j * I.ld;
    float* ocol = gc + I.c_off + (long long)j * I.ld;
    const double bj = __ldcg(zb + j);
    for (int i0 = 0; i0 < I.nr; i0 += 128) {
      const int i = i0 + 4 * lane;
      if (i >= I.nr) continue;
      const unsigned wd = __ldcg(words + (i >> 5));
      const unsigned m4 = (wd >> (i & 31)) & 0xfu;
      float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (m4) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (((m4 >> e) & 1u) && i + e < I.nr)
            o[e] = (float)(((__ldcg(za + i + e) + bj) - (double)__ldg(gcol + i + e)) * inv_lam);
      }
      if (i + 4 <= I.nr && (((I.c_off + (long long)j * I.ld + i) & 3) == 0)) {
        *reinterpret_cast<float4*>(ocol + i) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i + e < I.nr) ocol[i + e] = o[e];
      }
    }
  }
  if (blockIdx.x == 0) {
    double sa = 0.0, sb = 0.0;
    for (int i = threadIdx.x; i < I.nr; i += blockDim.x) sa += __ldcg(za + i);
    for (int j = threadIdx.x; j < I.nc; j += blockDim.x) sb += __ldcg(zb + j);
    sa = block_sum_d(sa, s_red);
    sb = block_sum_d(sb, s_red);
    const double t = (sb - sa) / (double)(I.nr + I.nc);
    for (int i = threadIdx.x; i < I.nr; i += blockDim.x) gp[I.f1_off + i] = (float)(za[i] + t);
    for (int j = threadIdx.x; j < I.nc; j += blockDim.x) gq[I.f2_off + j] = (float)(zb[j] - t);
  }
}

}  // namespace drot

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

using namespace drot;

namespace {

struct AdjLayout {
  int grid = 0, threads = kAdjThreads, n_seg = 0, V = 0, chunk = 0, max_lines = 0;
  size_t smem = 0;
  std::vector<AdjInst> inst;
  std::vector<AdjSeg> seg;
  std::vector<int> cta_seg0;
  long long mcol_words = 0, mrow_words = 0;
  size_t off_ctrl = 0, off_inst = 0, off_seg = 0, off_cta = 0, off_mcol = 0, off_mrow = 0,
         off_vec = 0, off_slots = 0, off_iters = 0, off_conv = 0, off_relres = 0, total = 0;
};

size_t al256(size_t v) { return (v + 255) / 256 * 256; }

int adj_layout(int n_inst, const drot_adjoint_instance* d, AdjLayout& L) {
  if (n_inst <= 0 || n_inst > 65535 || !d) return DROT_ERR_INVALID_ARG;
  L.inst.resize(n_inst);
  long long V = 0, mc = 0, mr = 0, lines = 0;
  int maxv = 0, maxk = 0;
  for (int k = 0; k < n_inst; ++k) {
    const drot_adjoint_instance& a = d[k];
    if (a.n_rows <= 0 || a.n_cols <= 0 || a.ld < a.n_rows || a.c_offset < 0 ||
        a.v_offset < 0 || a.phi1_offset < 0 || a.phi2_offset < 0 || !(a.step_size > 0.0f) ||
        !(a.lambda > 0.0f) ||
        (long long)a.n_rows + a.n_cols > (1 << 24))
      return DROT_ERR_INVALID_ARG;
    AdjInst& I = L.inst[k];
    memset(&I, 0, sizeof(I));
    I.nr = a.n_rows;
    I.nc = a.n_cols;
    I.ld = a.ld;
    I.nwr = (a.n_rows + 31) / 32;
    I.nwc = (a.n_cols + 31) / 32;
    I.c_off = a.c_offset;
    I.f1_off = a.phi1_offset;
    I.f2_off = a.phi2_offset;
    I.s = a.step_size;
    I.lam = a.lambda;
    I.v_off = (int)a.v_offset;
    I.mc_off = mc;
    I.mr_off = mr;
    mc += (long long)a.n_cols * I.nwr;
    mr += (long long)a.n_rows * I.nwc;
    V = std::max(V, a.v_offset + a.n_rows + a.n_cols);
    lines += a.n_rows + a.n_cols;
    maxv = std::max(maxv, a.n_rows + a.n_cols);
    maxk = std::max(maxk, std::max(a.n_rows, a.n_cols));
  }
  if (V > INT32_MAX / 2) return DROT_ERR_UNSUPPORTED;
  L.V = (int)V;
  L.mcol_words = mc;
  L.mrow_words = mr;
  if (sizeof(double) * (size_t)maxv > 200 * 1024) return DROT_ERR_UNSUPPORTED;

  int dev = 0, sms = 0, coop = 0, occ = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return DROT_ERR_CUDA;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return DROT_ERR_CUDA;
  // The direction, the line sums, and as many of the digits as fit beside them
  // (all of one side for up to 4096 rows or columns).
  L.max_lines = maxv;
  L.smem = sizeof(double) * (size_t)maxv + sizeof(unsigned) * ((size_t)maxv / 32 + 2) +
           32 * (size_t)kAdjBlock;
  const long long room = ((long long)optin - 2048 - (long long)L.smem) / kAdjDigitBytes;
  L.chunk = (int)std::min<long long>(std::min(kAdjChunk, (maxk + 31) & ~31), room & ~31LL);
  if (L.chunk < 32) return DROT_ERR_UNSUPPORTED;
  L.smem += (size_t)kAdjDigitBytes * L.chunk;
  if (allow_shared_memory((const void*)adj_pcg_kernel) != cudaSuccess) return DROT_ERR_CUDA;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)adj_pcg_kernel, L.threads,
                                                    L.smem) != cudaSuccess || occ <= 0)
    return DROT_ERR_CUDA;
  // At least ~64 lines per CTA: tiny batches do not spread over every SM.
  const long long want = std::max(1LL, lines / 64);
  L.grid = (int)std::min<long long>((long long)occ * sms, want);

  L.cta_seg0.assign(L.grid + 1, 0);
  if (2 * n_inst <= L.grid) {
    // A CTA takes lines of one instance and one side (a second segment or side
    // doubles its work, and all wait for it: 8 instances of 512..2048 took 32
    // us per iteration with the even split below, 17 with this one).  CTA by
    // CTA to the side whose CTAs take longest, in about clocks: the digits of
    // the other side's entries, then its lines; whole groups of 16 lines.
    std::vector<int> ctas(2 * n_inst, 1);
    auto side = [&](int u) { return u & 1 ? L.inst[u / 2].nc : L.inst[u / 2].nr; };
    auto cost = [&](int u) {
      const double k = side(u ^ 1);
      return 2.0 * k + (double)side(u) / ctas[u] * (k / 32.0 + 15.0);
    };
    std::priority_queue<std::pair<double, int>> most;
    for (int u = 0; u < 2 * n_inst; ++u) most.push({cost(u), u});
    for (int c = 2 * n_inst; c < L.grid; ++c) {
      const int u = most.top().second;
      most.pop();
      ++ctas[u];
      most.push({cost(u), u});
    }
    int c = 0;
    for (int u = 0; u < 2 * n_inst; ++u) {
      const int groups = (side(u) + 15) / 16, l0 = u & 1 ? L.inst[u / 2].nr : 0;
      for (int j = 0; j < ctas[u]; ++j, ++c) {
        L.cta_seg0[c] = (int)L.seg.size();
        AdjSeg S;
        S.inst = u / 2;
        S.l0 = l0 + std::min(side(u), (int)((long long)groups * j / ctas[u]) * 16);
        S.l1 = l0 + std::min(side(u), (int)((long long)groups * (j + 1) / ctas[u]) * 16);
        S.cta = c;
        if (S.l1 > S.l0) L.seg.push_back(S);
      }
    }
  } else {
    // Lines [c*lines/G, (c+1)*lines/G) go to CTA c, cut at instance boundaries.
    long long base = 0;
    int k = 0;
    for (int c = 0; c < L.grid; ++c) {
      L.cta_seg0[c] = (int)L.seg.size();
      const long long g0 = lines * c / L.grid, g1 = lines * (c + 1) / L.grid;
      long long g = g0;
      while (g < g1) {
        while (g >= base + L.inst[k].nr + L.inst[k].nc) {
          base += L.inst[k].nr + L.inst[k].nc;
          ++k;
        }
        const long long end = std::min(g1, base + L.inst[k].nr + L.inst[k].nc);
        AdjSeg S;
        S.inst = k;
        S.l0 = (int)(g - base);
        S.l1 = (int)(end - base);
        S.cta = c;
        L.seg.push_back(S);
        g = end;
      }
    }
  }
  L.cta_seg0[L.grid] = (int)L.seg.size();
  L.n_seg = (int)L.seg.size();
  for (int t = 0; t < L.n_seg; ++t) {
    AdjInst& I = L.inst[L.seg[t].inst];
    if (I.nseg == 0) {
      I.seg0 = t;
      I.owner = L.seg[t].cta;
    }
    ++I.nseg;
  }

  size_t off = 0;
  L.off_ctrl = off;  off = al256(off + 512);
  L.off_inst = off;  off = al256(off + sizeof(AdjInst) * n_inst);
  L.off_seg = off;   off = al256(off + sizeof(AdjSeg) * L.n_seg);
  L.off_cta = off;   off = al256(off + sizeof(int) * (L.grid + 1));
  L.off_mcol = off;  off = al256(off + sizeof(unsigned) * (size_t)mc);
  L.off_mrow = off;  off = al256(off + sizeof(unsigned) * (size_t)mr);
  L.off_vec = off;   off = al256(off + sizeof(double) * (size_t)V * 7);
  L.off_slots = off; off = al256(off + sizeof(double) * (size_t)L.n_seg * 6);
  L.off_iters = off; off = al256(off + sizeof(int) * n_inst);
  L.off_conv = off;  off = al256(off + sizeof(int) * n_inst);
  L.off_relres = off; off = al256(off + sizeof(double) * n_inst);
  L.total = off;
  return DROT_OK;
}

}  // namespace

// Device pointers of a workspace laid out by L.
static void adj_params(const AdjLayout& L, char* ws, AdjParams& A) {
  memset(&A, 0, sizeof(A));
  double* vec = (double*)(ws + L.off_vec);
  A.r = vec;
  A.d0 = vec + (size_t)L.V;
  A.d1 = vec + 2 * (size_t)L.V;
  A.q = vec + 3 * (size_t)L.V;
  A.invdiag = vec + 4 * (size_t)L.V;
  A.deg = vec + 5 * (size_t)L.V;
  A.y = vec + 6 * (size_t)L.V;
  A.chunk = L.chunk;
  A.max_lines = L.max_lines;
  A.mcol = (unsigned*)(ws + L.off_mcol);
  A.mrow = (unsigned*)(ws + L.off_mrow);
  A.inst = (const AdjInst*)(ws + L.off_inst);
  A.seg = (const AdjSeg*)(ws + L.off_seg);
  A.cta_seg0 = (const int*)(ws + L.off_cta);
  double* slots = (double*)(ws + L.off_slots);
  A.slot_dq = slots;
  A.slot_ry = slots + L.n_seg;
  A.slot_rr = slots + 3 * (size_t)L.n_seg;
  A.slot_rr0 = slots + 5 * (size_t)L.n_seg;
  A.iters = (int*)(ws + L.off_iters);
  A.conv = (int*)(ws + L.off_conv);
  A.relres = (double*)(ws + L.off_relres);
  A.bar = (unsigned*)(ws + L.off_ctrl);
  A.abort_flag = (int*)(ws + L.off_ctrl + 64);
  A.conv_count = (unsigned*)(ws + L.off_ctrl + 128);
  const char* e = getenv("DROT_BARRIER_TIMEOUT_MS");
  const long long ms = (e && atoll(e) > 0) ? atoll(e) : 10000LL;
  A.timeout_ns = ms * 1000000LL;
  A.n_seg = L.n_seg;
}

extern "C" {

size_t drot_qr_adjoint_workspace_bytes(int n_inst, const drot_adjoint_instance* inst) {
  AdjLayout L;
  return adj_layout(n_inst, inst, L) == DROT_OK ? L.total : 0;
}

int drot_qr_adjoint_prepare(int n_inst, const drot_adjoint_instance* inst, const void* c,
                            int c_dtype, const float* phi1, const float* phi2,
                            unsigned char* mask, void* workspace, size_t workspace_bytes,
                            drot_stream_t stream) {
  if (!c || !phi1 || !phi2 || !workspace) return DROT_ERR_INVALID_ARG;
  if (c_dtype != DROT_C_F32 && c_dtype != DROT_C_BF16) return DROT_ERR_INVALID_ARG;
  AdjLayout L;
  int rc = adj_layout(n_inst, inst, L);
  if (rc != DROT_OK) return rc;
  if (workspace_bytes < L.total || ((uintptr_t)workspace & 255u)) return DROT_ERR_WORKSPACE;
  char* ws = (char*)workspace;
  cudaStream_t st = (cudaStream_t)stream;
  AdjParams A;
  adj_params(L, ws, A);
  A.c = c;
  A.c_bf16 = c_dtype == DROT_C_BF16;
  A.phi1 = phi1;
  A.phi2 = phi2;
  A.mask = mask;
  A.n_inst = n_inst;
  if (cudaMemcpyAsync(ws + L.off_inst, L.inst.data(), sizeof(AdjInst) * n_inst,
                      cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(ws + L.off_seg, L.seg.data(), sizeof(AdjSeg) * L.n_seg,
                      cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(ws + L.off_cta, L.cta_seg0.data(), sizeof(int) * (L.grid + 1),
                      cudaMemcpyHostToDevice, st) != cudaSuccess)
    return DROT_ERR_CUDA;
  long long maxblk = 0;
  for (const AdjInst& I : L.inst) maxblk = std::max(maxblk, (long long)I.nwr * I.nwc);
  const int mblocks = (int)std::min<long long>((maxblk + 7) / 8, 2048);
  adj_mask_kernel<<<dim3(mblocks, n_inst), 256, 0, st>>>(A);
  if (cudaGetLastError() != cudaSuccess) return DROT_ERR_CUDA;
  // The descriptors above are copied from pageable host memory that dies
  // with this call: wait for the copies (and the mask) to finish.
  return cudaStreamSynchronize(st) == cudaSuccess ? DROT_OK : DROT_ERR_CUDA;
}

int drot_qr_adjoint_solve(int n_inst, const drot_adjoint_instance* inst, const float* g,
                          double* z, double tol, int max_iters, void* workspace,
                          size_t workspace_bytes, int* iters, drot_stream_t stream) {
  if (!g || !z || !workspace || max_iters < 0 || !(tol >= 0.0)) return DROT_ERR_INVALID_ARG;
  AdjLayout L;
  int rc = adj_layout(n_inst, inst, L);
  if (rc != DROT_OK) return rc;
  if (workspace_bytes < L.total || ((uintptr_t)workspace & 255u)) return DROT_ERR_WORKSPACE;
  char* ws = (char*)workspace;
  cudaStream_t st = (cudaStream_t)stream;
  AdjParams A;
  adj_params(L, ws, A);
  A.g = g;
  A.z = z;
  A.n_inst = n_inst;
  A.max_iters = max_iters;
  A.tol = tol;
  if (cudaMemsetAsync(ws + L.off_ctrl, 0, 512, st) != cudaSuccess ||
      cudaMemsetAsync(ws + L.off_iters, 0, L.total - L.off_iters, st) != cudaSuccess)
    return DROT_ERR_CUDA;
  void* args[] = {(void*)&A};
  if (cudaLaunchCooperativeKernel((const void*)adj_pcg_kernel, dim3(L.grid), dim3(L.threads), args,
                                  L.smem, st) != cudaSuccess) {
    cudaGetLastError();
    return DROT_ERR_CUDA;
  }
  int abort_flag = 0;
  if ((iters && cudaMemcpyAsync(iters, ws + L.off_iters, sizeof(int) * n_inst,
                                cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
      cudaMemcpyAsync(&abort_flag, ws + L.off_ctrl + 64, sizeof(int), cudaMemcpyDeviceToHost,
                      st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return DROT_ERR_CUDA;
  return abort_flag ? DROT_ERR_BARRIER_TIMEOUT : DROT_OK;
}

int drot_qr_adjoint_grad(int n_inst, const drot_adjoint_instance* inst, const float* g,
                         const double* z, float* grad_c, float* grad_p, float* grad_q,
                         void* workspace, size_t workspace_bytes, drot_stream_t stream) {
  if (!g || !z || !grad_c || !grad_p || !grad_q || !workspace) return DROT_ERR_INVALID_ARG;
  AdjLayout L;
  int rc = adj_layout(n_inst, inst, L);
  if (rc != DROT_OK) return rc;
  if (workspace_bytes < L.total || ((uintptr_t)workspace & 255u)) return DROT_ERR_WORKSPACE;
  AdjParams A;
  adj_params(L, (char*)workspace, A);
  A.g = g;
  A.z = const_cast<double*>(z);
  A.n_inst = n_inst;
  int maxc = 1;
  for (const AdjInst& I : L.inst) maxc = std::max(maxc, I.nc);
  const int blocks = std::min((maxc + 7) / 8, 1024);
  adj_grad_kernel<<<dim3(blocks, n_inst), 256, 0, (cudaStream_t)stream>>>(A, grad_c, grad_p,
                                                                        grad_q);
  return cudaGetLastError() == cudaSuccess ? DROT_OK : DROT_ERR_CUDA;
}

int drot_qr_adjoint_residuals(int n_inst, const drot_adjoint_instance* inst,
                              const void* workspace, size_t workspace_bytes, double* rel_residual,
                              drot_stream_t stream) {
  if (!workspace || !rel_residual) return DROT_ERR_INVALID_ARG;
  AdjLayout L;
  int rc = adj_layout(n_inst, inst, L);
  if (rc != DROT_OK) return rc;
  if (workspace_bytes < L.total || ((uintptr_t)workspace & 255u)) return DROT_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemcpyAsync(rel_residual, (const char*)workspace + L.off_relres,
                      sizeof(double) * n_inst, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return DROT_ERR_CUDA;
  return DROT_OK;
}

}  // extern "C"

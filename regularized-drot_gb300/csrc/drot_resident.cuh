// drot_resident.cuh -- the solve loop of one problem whose plan stays on chip.
//
// The streaming kernel (drot_kernels.cuh) moves X through L2 or HBM on every
// iteration and meets twice per iteration at a grid barrier; for problems
// that fit the chip's shared memory both cost more than the arithmetic.  Here
// a CTA owns one tile of X and C in shared memory for the whole solve, and per
// iteration the CTAs exchange only the tiles' row and column sums.  Measured,
// us per iteration, streaming -> here: QR 96 x 80 6.9 -> 2.6, 1000 x 1000 9.6
// -> 3.1, 1500 x 1500 11.3 -> 4.1, 1850 x 1850 13.2 -> 5.7; GL 300 x 200 8.9
// -> 3.3, 1500 x 1000 (2 classes) 12.1 -> 5.8.  Bound by latency; the stages of
// CTA 0, as the kernel times them (drot_result.phase_ms), us per iteration:
//                          X-update   sums, exchange, duals   barrier   stop test
//   QR 96 x 80 (one CTA)     1.5              0.6               0.3        0.1
//   QR 1000 x 1000           1.2              1.3               0.4        0.1
//   GL 1500 x 1000           2.0              3.2               0.7        0.1
//   QR 3000 x 3000           7.4              2.6               0.7        0.7
//
// Tiles.  The grid is GR x GC CTAs, at most one per SM.  CTA (br, bc) owns the
// rows of band br (QR: equal heights, multiples of 4; GL: one class) and an
// equal share of the columns.  Inside, warp (wr, wc) of WR x WC owns 128 rows
// (lane: 4 consecutive ones) and cw columns; slot [j][thread] holds the
// thread's 4 rows of column j, so every access is a conflict-free 128-bit one.
// Rows and columns of the warps' tiles beyond the CTA's get phi = -inf, so
// their X is exactly zero with no masks in the element loop.  X in shared
// memory costs two more instructions per four elements than X in registers,
// but the column loop can be rolled: with 8 to 32 columns unrolled over
// registers the iteration missed the instruction cache on 43 % of its
// fetches (2000 x 1500: 700 cycles per column of a warp).
//
// Larger QR problems (about 1900 x 1900 to 4100 x 4100) keep the first nsx
// columns of every warp's X in shared memory and the first nsc of its C; the
// rest stays in global memory, in L2 at these sizes, and is read where it is
// used.  us per iteration, streaming -> here: 2000 x 2000 13.4 -> 6.9, 3000 x
// 3000 18.6 -> 11.3, 4000 x 4000 29.0 -> 22.8, 2600 x 4100 with BF16 C 22.1 ->
// 15.7.  (Loading a step's global values one step ahead costs the registers
// of 16 warps a CTA: 3000 x 3000 11.9.)
//
// Exchange.  One 64-bit word per row of a band and per column of a chunk, in
// L2: every CTA adds its partial sum as a fixed-point number (46 fraction
// bits; integer addition, so the total does not depend on the order) plus a
// count of one in the top byte (red.add), and polls the word until the count
// is complete: the reduction, the flag and the data are one word and one trip.
// The total mass is one word added to and polled by every CTA, with 38
// fraction bits.  The words are never cleared: they alternate by round, a
// reader subtracts what it last saw, and a CTA adds to round r + 2 only after
// round r + 1's mass word was complete, which every CTA adds to after it has
// read round r.  Measured, one exchange of 152 CTAs in 8 x 19 tiles of 128 x
// 53: 2000 cycles; with tagged words that each reader sums itself 5900, with
// a counter barrier and loads after it 5500.
//   Fixed point: a total has an error of at most GC 2^-47, an absolute one beside a
// mass of about 1: below the FP32 rounding of sums and duals above GC 2^-23.  Rows
// of smaller marginals keep fewer bits of their sums than FP32 has; the errors of
// plans and duals against 64 bits, marginals of 1e-8 and 1e-11 and cold starts
// included, are the streaming kernel's (its sums of a warp are float, too).  A CTA whose mass would exceed the words'
// range (or is not finite) adds a poison count to the mass word instead; then
// every CTA repeats the round with 8 fraction bits fewer (or, where all finite
// sums fit, adds a round of counts of infinities and NaNs), so the arithmetic
// depends on the data of the iteration alone and a solve split into segments gives
// the same bits.
//   The squared residual is published as tagged words {value, tag}, in two
// slots that take turns (drot_exchange.h: residual_slot, with the order that
// makes that safe), and read during the next iteration, whose X-update runs
// meanwhile into the second copy of X; a converged solve hands back the copy
// before it.  Where the
// shared memory has no room for two copies the CTAs wait for the residual.
//   Every poll is bounded by wall time like the streaming kernel's barriers.
#pragma once

#include "drot_resident.h"

namespace drot {

constexpr int kResidentMaxWarps = 16;
// Words that every CTA polls are published in copies, each polled by a share
// of the CTAs: 152 CTAs polling the same 19 lines of mass words took 7000
// cycles a trip, against 1300 for lines polled by at most 19.
constexpr int kPairCopies = 16;

// Dynamic shared memory, in order: X slots [nsx][threads] float4 (one or two
// copies), C slots [nsc][threads], warp row sums [WC][WR * 128], warp
// column sums [WR][ct], group norms [WR][ct] (GL), staged duals of two
// parities (t1 [rt], t2 [ct]); batches: words seen [2][rt + ct], and GL
// marginals and former duals [rt + ct].
__host__ __device__ constexpr size_t resident_smem_bytes(int threads, int nsx, int nsc, int wr,
                                                         int wc, int rt, int ct, size_t csize,
                                                         bool keep_x, bool gl, bool batch) {
  return (size_t)threads * 4 * (nsc * csize + nsx * sizeof(float) * (keep_x ? 2 : 1)) +
         sizeof(float) * ((size_t)wc * wr * 128 + (size_t)wr * ct * (gl ? 2 : 1) +
                          2 * ((size_t)rt + ct)) +
         (batch ? (2 * sizeof(unsigned long long) + (gl ? 2 * sizeof(float) : 0)) *
                      ((size_t)rt + ct)
                : 0) + 64;
}

// ---- tagged words ---------------------------------------------------------

__device__ __forceinline__ void ll_store(unsigned long long* p, float v, unsigned tag) {
  const unsigned long long w =
      ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(w) : "memory");
}

__device__ __forceinline__ void word_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long ll_load(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// Warp sum of non-negative float pairs, every lane's result.  The shuffle
// tree of pair additions (warp_sum_fp) is a chain of about 400 cycles, and
// three of them lie on the critical path of an iteration; here the pairs
// become two-word fixed-point numbers on the scale of the largest lane (24 + 24
// bits below it, the pair's own precision) and the words are summed by
// integer warp reductions, exactly.  Infinities and NaN take the tree.
__device__ __noinline__ fpair warp_sum_tree(fpair v) { return warp_sum_fp(v); }

__device__ __forceinline__ fpair warp_sum_nonneg(fpair v) {
  const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(v.hi));
  if (top >= 0x7f800000u) return warp_sum_tree(v);
  const int e = max((int)(top >> 23), 30);  // biased exponent of the largest lane
  // unit 2^(e - 127 - 24): |hi| < 2^25 units, 32 of them below 2^30
  const float up = __uint_as_float((unsigned)(127 + 127 + 24 - e) << 23);
  const float unit = __uint_as_float((unsigned)(e - 24) << 23);
  const float f = rintf(v.hi * up);
  const float rem = fmaf(-f, unit, v.hi) + v.lo;  // below 1.5 units
  const int s1 = __reduce_add_sync(0xffffffffu, (int)f);
  const int s2 = __reduce_add_sync(0xffffffffu, __float2int_rn((rem * up) * 16777216.0f));
  const float h1 = (float)s1, l1 = (float)(s1 - (int)h1);
  float hi, lo;
  two_sum(h1, fmaf((float)s2, 5.9604644775390625e-8f, l1), hi, lo);  // 2^-24
  return fpair{hi * unit, lo * unit};
}

// gamma = (2 (sigma - 1) - alpha) / n and alpha' = (alpha + 1) - sigma as the
// reference evaluates them in double (core/kernel_qr.hpp:405-467), on float
// pairs: the numerator is carried with its rounding errors, the quotient
// corrected by its residual, so the float results equal the rounded double
// ones except within 2^-44 of a rounding boundary.  FP64 arithmetic here
// costs about 1500 cycles of every iteration on this part.
__device__ __noinline__ float gamma_f64(float sigma, float alpha, float n) {
  return (float)((2.0 * ((double)sigma - 1.0) - (double)alpha) / (double)n);
}

__device__ __noinline__ float alpha_f64(float sigma, float alpha) {
  return (float)(((double)alpha + 1.0) - (double)sigma);
}

__device__ __forceinline__ float gamma_of(float sigma, float alpha, float n, float n_rcp) {
  if (!(fabsf(sigma) < 1e30f && fabsf(alpha) < 1e30f))
    return gamma_f64(sigma, alpha, n);
  float d, e1, h, e2, hi, lo;
  two_sum(sigma, -1.0f, d, e1);
  two_sum(2.0f * d, -alpha, h, e2);
  two_sum(h, fmaf(2.0f, e1, e2), hi, lo);
  const float q0 = hi * n_rcp;
  const float q1 = fmaf(fmaf(-q0, n, hi) + lo, n_rcp, q0);
  return fmaf(fmaf(-q1, n, hi) + lo, n_rcp, q1);
}

__device__ __forceinline__ float alpha_next(float sigma, float alpha) {
  if (!(fabsf(sigma) < 1e30f && fabsf(alpha) < 1e30f))
    return alpha_f64(sigma, alpha);
  float u, e1, h, e2;
  two_sum(alpha, 1.0f, u, e1);
  two_sum(u, -sigma, h, e2);
  return h + (e1 + e2);
}

__device__ __noinline__ float div_ieee(float a, float b) { return a / b; }

// r2 < T for the squared residual r2 = hi + lo: the heads decide unless they
// agree to within 2^-20, where the exact FP64 comparison does.
__device__ __forceinline__ int below(fpair r2, double T, float T_hi) {
  const float d = r2.hi - T_hi;
  if (fabsf(d) > 1e-6f * fabsf(r2.hi)) return d < 0.0f ? 1 : 0;
  return fp_value(r2) < T ? 1 : 0;
}

// Bounded polls of one thread: a wait longer than the limit (or another
// CTA's raised flag) sets `failed`; later polls of a failed thread return at
// once, and the CTA leaves its loop at its next vote.
struct LLWait {
  int* abort_flag;
  long long limit;
  bool failed;

  // Calls poll() until it returns true.
  template <typename Poll>
  __device__ __forceinline__ void until(Poll poll) {
    unsigned long long t0 = 0ull;
    for (unsigned spins = 0; !poll() && !failed; ++spins) {
      if ((spins & 63u) != 63u) continue;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0ull) t0 = now;
      if (ld_volatile_i32(abort_flag)) {
        failed = true;
      } else if ((long long)(now - t0) > limit) {
        atomicExch(abort_flag, 1);
        failed = true;
      }
    }
  }

  // Values of up to N words (at(u) their addresses, n of them live), every
  // word still missing loaded again in each round, so the wait is one trip
  // after the last word is there.
  template <int N, typename At>
  __device__ __forceinline__ void gather(At at, int n, unsigned tag, float (&v)[N]) {
    unsigned long long w[N];
#pragma unroll
    for (int u = 0; u < N; ++u) w[u] = u < n ? ll_load(at(u)) : (unsigned long long)tag << 32;
    until([&]() {
      bool all = true;
#pragma unroll
      for (int u = 0; u < N; ++u)
        if ((unsigned)(w[u] >> 32) != tag) {
          all = false;
          w[u] = ll_load(at(u));
        }
      return all;
    });
#pragma unroll
    for (int u = 0; u < N; ++u) v[u] = u < n ? __uint_as_float((unsigned)w[u]) : 0.0f;
  }

};

// Fixed-point words: 46 fraction bits for rows and columns, 38 for the mass,
// 8 fewer per level.  In a class round (level < 0) a contribution counts a
// NaN (bits 40 up) or an infinity (bits 20 up); it follows a round that held the
// finite sums, and replaces the others.
constexpr int kRowBits = 46, kMassBits = 38, kLevelBits = 8;
constexpr unsigned long long kCountOne = 1ull << 56, kPoisonOne = 1ull << 48;

__device__ __forceinline__ float pow2f(int k) {
  return __uint_as_float((unsigned)(127 + k) << 23);
}

// RN(v) for 0 <= v < 2^57, and back (both about 25 cycles; the 64-bit
// conversion instructions take 90).
__device__ __forceinline__ unsigned long long to_fixed(float v) {
  const unsigned b = __float_as_uint(v);
  const unsigned long long m = ((b & 0x7fffffu) | 0x800000u) * 2ull;  // 25 bits, half units
  const int sh = (int)(b >> 23) - 151;                                // v = m 2^sh
  if (sh >= 0) return m << sh;
  return sh < -25 ? 0ull : ((m << 1 >> -sh) + 1ull) >> 1;
}

__device__ __forceinline__ float from_fixed(unsigned long long n) {
  const unsigned hi = (unsigned)(n >> 24), lo = (unsigned)n & 0xffffffu;
  const float h = __uint2float_rn(hi);
  const float rest = hi < 0xffffff00u ? __int2float_rn((int)(hi - __float2uint_rz(h))) : 0.0f;
  return fmaf(h, 16777216.0f, fmaf(rest, 16777216.0f, __uint2float_rn(lo)));
}

__device__ __noinline__ unsigned long long class_word(float v) {
  return v != v ? 1ull << 40 : (fabsf(v) > 3.402823466e38f ? 1ull << 20 : 0ull);
}

__device__ __noinline__ float class_value(unsigned long long n) {
  return (n >> 40) != 0 ? __uint_as_float(0x7fffffffu)
                        : ((n >> 20) != 0 ? __uint_as_float(0x7f800000u) : 0.0f);
}

struct PairSum {
  fpair v;
  bool failed;
};

// Warp sum of the grid's n float pairs p[2 k], p[2 k + 1] (all non-negative).
__device__ __noinline__ PairSum ll_pairs(const unsigned long long* p, int n, unsigned tag,
                                         int* abort_flag, long long limit, bool failed) {
  LLWait wait = {abort_flag, limit, failed};
  fpair t = fp_make(0.0f);
  for (int k0 = threadIdx.x & 31; k0 < n; k0 += 5 * 32) {
    float v[10];
    wait.gather<10>([&](int u) { return p + 2 * (k0 + (u >> 1) * 32) + (u & 1); },
                    2 * min(5, (n - k0 + 31) / 32), tag, v);
    t = fp_add(t, fp_add(fp_add(fp_add(fpair{v[0], v[1]}, fpair{v[2], v[3]}),
                                fp_add(fpair{v[4], v[5]}, fpair{v[6], v[7]})),
                         fpair{v[8], v[9]}));
  }
  __syncwarp();
  return PairSum{warp_sum_nonneg(t), wait.failed};
}

// One step of a transposing warp sum: lanes with bit o of the lane index
// clear keep a's sum, the others b's.
__device__ __forceinline__ float fold_lanes(float a, float b, int o, int lane) {
  const bool up = (lane & o) != 0;
  const float keep = up ? b : a, send = up ? a : b;
  return keep + __shfl_xor_sync(0xffffffffu, send, o);
}

// Sums m[j] over the warp for NC columns: afterwards lane l holds column
// l & (NC - 1) (16 shuffles for 16 columns instead of 80).
template <int NC>
__device__ __forceinline__ float fold_columns(float (&m)[NC], int lane) {
#pragma unroll
  for (int w = NC; w > 1; w >>= 1)
#pragma unroll
    for (int j = 0; j < w / 2; ++j) m[j] = fold_lanes(m[2 * j], m[2 * j + 1], NC / w, lane);
  float t = m[0];
#pragma unroll
  for (int o = NC; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// ---------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------

// One CTA's part (tile `cta` of G) of one problem's solve.  BATCH: one of a
// batch's instances (drot_resident_batch_kernel), whose record is a batch
// record and whose final alpha goes to the slot of its iteration parity.
template <int MODE, typename CT, int T, bool BATCH>
__device__ __forceinline__ void resident_solve(const ResidentParams& P, const int* gbounds,
                                               const int cta, const int G) {
  constexpr bool F32C = std::is_same<CT, float>::value;
  using CSlot = typename std::conditional<F32C, float4, uint2>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int W = T / 32;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int WR = P.WR, WC = P.WC, rt = P.rt, ct = P.ct;
  const int wc = warp / WR, wr = warp - wc * WR;
  const int nsx = P.nsx, nsc = P.nsc;  // slots of X and of C (the rest stay in global memory)
  const int slots = nsx * T;
  float4* const xa = reinterpret_cast<float4*>(smem_raw) + tid;  // slot j: xa[j * T]
  float4* const xb = xa + (P.keep ? slots : 0);                  // after odd iterations
  CSlot* const cs = reinterpret_cast<CSlot*>(xb - tid + slots) + tid;
  float* s_row = reinterpret_cast<float*>(cs - tid + nsc * T);
  float* s_col = s_row + (size_t)WC * WR * 128;
  float* s_nrm = s_col + (size_t)WR * ct;
  float* s_t1 = s_nrm + (MODE == MODE_GL ? (size_t)WR * ct : 0);  // [2][rt]
  float* s_t2 = s_t1 + 2 * rt;                                    // [2][ct]
  __shared__ fpair s_sum[kResidentMaxWarps + 1], s_res[kResidentMaxWarps];
  __shared__ float s_gamma[2];
  __shared__ fpair s_r2, s_own;
  __shared__ int s_stop, s_level;

  const int br = cta / P.GC, bc = cta - br * P.GC;
  int lo, hi;
  if constexpr (MODE == MODE_QR) {
    lo = min(br * P.band_h, P.nr);
    hi = min(lo + P.band_h, P.nr);
  } else {
    lo = gbounds[br];
    hi = gbounds[br + 1];
  }
  const int base = lo & ~3;  // the tile's row 0 (16-byte columns: a vector boundary)
  const int c0 = (int)(((long long)P.nc * bc) / P.GC);
  const int c1 = (int)(((long long)P.nc * (bc + 1)) / P.GC);
  const int h = hi - base, w = c1 - c0;  // tile rows (from base) and columns
  const int head = lo - base;            // rows of another band at the top
  // this warp's columns and this lane's rows (tile coordinates)
  const int wj0 = min(wc * P.cw, w), ncw = min(P.cw, w - wj0);
  const int r0 = wr * 128 + lane * 4;
  const long long ld = P.ld;
  const bool inside = r0 >= head && r0 + 4 <= h;
  const bool whole = P.vec_ok && inside;
  // rows of the tile under every lane of the warp: no row masks
  const bool full = __all_sync(0xffffffffu, inside);
  // Slots in global memory are read as whole vectors (the columns are padded to
  // them; element by element in the one lane that straddles the edge, an
  // iteration took twice as long).  Rows of a vector beyond the tile get phi =
  // -inf, which turns any X there into zero, and in a batch a cost of zero (the
  // padding is the caller's and may hold anything; a single problem's is a copy
  // with zeros).  GL stores such a vector element by element: its other rows
  // are another class's.
  const bool live_lane = r0 + 4 > head && r0 < h;
  auto c_inside = [&](const float (&w)[4], f32x2& c01, f32x2& c23) {  // of load_c_raw's w
    float v[4] = {c_at<CT>(w, 0), c_at<CT>(w, 1), c_at<CT>(w, 2), c_at<CT>(w, 3)};
    if (BATCH && !full) {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = r0 + e >= head && r0 + e < h ? v[e] : 0.0f;
    }
    c01 = x2_pack(v[0], v[1]);
    c23 = x2_pack(v[2], v[3]);
  };
  auto set_x = [&](float* g, f32x2 x01, f32x2 x23) {
    float v[4];
    x2_unpack(x01, v[0], v[1]);
    x2_unpack(x23, v[2], v[3]);
    if (MODE == MODE_QR || inside) {
      store_vec<4>(g, v);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r0 + e >= head && r0 + e < h) g[e] = v[e];
    }
  };

  const CT* const cg = reinterpret_cast<const CT*>(P.c);
  // ---- the tile's X and C
  for (int j = 0; j < nsx; ++j) {
    const long long off = (long long)(c0 + wj0 + j) * ld + base + r0;
    float xv[4] = {0.0f, 0.0f, 0.0f, 0.0f}, cv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (j >= ncw) {
      // padding column: zero X and C, phi2 = -inf
    } else if (whole) {
      load_vec<4>(P.x + off, xv);
      load_c_raw<4, CT>(cg + off, cv);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r0 + e >= head && r0 + e < h) {
          xv[e] = P.x[off + e];
          if constexpr (F32C) {
            cv[e] = __ldg(cg + off + e);
          } else {
            const unsigned u = __ldg(reinterpret_cast<const unsigned short*>(cg) + off + e);
            cv[e >> 1] = __uint_as_float(__float_as_uint(cv[e >> 1]) | (u << (16 * (e & 1))));
          }
        }
    }
    xb[j * T] = make_float4(xv[0], xv[1], xv[2], xv[3]);
    if (j >= nsc) continue;
    if constexpr (F32C) cs[j * T] = make_float4(cv[0], cv[1], cv[2], cv[3]);
    else cs[j * T] = make_uint2(__float_as_uint(cv[0]), __float_as_uint(cv[1]));
  }
  // a slot of X or C as two packed pairs
  auto x_pairs = [](const float4& t, f32x2& x01, f32x2& x23) {
    const float4 v = t;
    x01 = x2_pack(v.x, v.y);
    x23 = x2_pack(v.z, v.w);
  };
  auto put_x = [](float4& t, f32x2 x01, f32x2 x23) {
    float v[4];
    x2_unpack(x01, v[0], v[1]);
    x2_unpack(x23, v[2], v[3]);
    t = make_float4(v[0], v[1], v[2], v[3]);
  };
  auto c_pairs = [](const CSlot& t, f32x2& c01, f32x2& c23) {
    const CSlot v = t;
    if constexpr (F32C) {
      c01 = x2_pack(v.x, v.y);
      c23 = x2_pack(v.z, v.w);
    } else {
      c01 = x2_pack(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u));
      c23 = x2_pack(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
    }
  };

  // ---- duals: item i is row head + i of the tile (i < hr), then column i -
  // hr.  Thread t of the item warps (all but the last two, which handle the
  // mass and the residual) owns items t + u * IT; the CTAs of a band hold equal
  // copies of its rows' duals (of a chunk, its columns'), and each counts and
  // writes back its share: rows [sr0, sr1), columns [sc0, sc1).
  constexpr int NI = BATCH && MODE == MODE_GL ? 6 : 4;
  const float most_r = (float)((1ull << 55) / (unsigned)P.GC);
  const float most_c = (float)((1ull << 55) / (unsigned)P.GR);
  const int hr = h - head, n_items = hr + w;
  const int sr0 = (int)(((long long)hr * bc) / P.GC), sr1 = (int)(((long long)hr * (bc + 1)) / P.GC);
  const int sc0 = hr + (int)(((long long)w * br) / P.GR);
  const int sc1 = hr + (int)(((long long)w * (br + 1)) / P.GR);
  const int mass_warp = W - 1, res_warp = W - 2;
  constexpr int IT = T - 64;
  const int item_warps = min(W - 2, (n_items + 31) >> 5);
  // The words as last read, by round parity.  Batches keep them in shared
  // memory: two CTAs per SM leave 128 registers a thread and an L1 too small to
  // hold what is spilled (83 % of the reloads missed it; 16 GL instances of
  // 256..2048 22.2 -> 19.5 ms with the planner's tiles).
  unsigned long long seen[2][NI];
  unsigned long long* const s_seen = reinterpret_cast<unsigned long long*>(s_t2 + 2 * ct);
  const int seen_n = rt + ct;
  constexpr bool LEAN = BATCH && MODE == MODE_GL;  // marg and dual_prev there, too
  float dual[NI], dual_prev[NI], marg[NI];
  float* const s_marg = reinterpret_cast<float*>(s_seen + 2 * seen_n);
  float* const s_prev = s_marg + seen_n;
#pragma unroll
  for (int u = 0; u < NI; ++u) {
    const int i = tid + u * IT;
    dual[u] = marg[u] = 0.0f;
    if (warp < res_warp && i < n_items) {
      marg[u] = i < hr ? P.p[lo + i] : P.q[c0 + i - hr];
      dual[u] = i < hr ? P.a[lo + i] : P.b[c0 + i - hr];
    }
    if constexpr (!LEAN) {
      dual_prev[u] = dual[u];
    } else if (warp < res_warp && i < n_items) {
      s_marg[i] = marg[u];
      s_prev[i] = dual[u];
    }
    if constexpr (!BATCH) seen[0][u] = seen[1][u] = 0ull;
    else if (warp < res_warp && i < n_items) s_seen[i] = s_seen[seen_n + i] = 0ull;
  }
  unsigned long long mass_seen[2] = {0ull, 0ull};

  const float NEG_INF = __int_as_float(0xff800000);
  const float s = P.s, kappa = P.kappa, kappa_rcp = P.kappa_rcp;
  const float nc_f = (float)P.nc, nr_f = (float)P.nr;
  // mass warp, lane 0 (in shared memory, out of every thread's registers):
  // alpha and the float total mass, and their values before the last update
  __shared__ float alpha, alpha_prev, sigma, sigma_prev;
  if (tid == mass_warp * 32) {
    alpha = alpha_prev = *P.alpha;
    sigma = sigma_prev = 0.0f;
  }
  LLWait wait = {P.abort_flag, P.timeout_ns, false};
  // objective of the last iteration that read C (lane part, four sums)
  f32x2 ob01 = x2_pack(0.0f, 0.0f), ob23 = ob01;
  int obj_valid = 0;
  int it = 0, stop_it = -1;
  int pend = -1;          // iteration whose residual is published but not decided
  unsigned pend_tag = 0;
  unsigned rd = 0;        // exchange rounds so far
  bool aborted = false;
  fpair last_r2 = fp_make(-1.0f);
  // Stage times of one CTA in SM clocks, scaled to ns at the end.
  __shared__ long long tacc[4], tp, tp0;
  __shared__ unsigned long long ns0;
  const bool timer = !BATCH && cta == P.timer_cta && tid == 0;
  if (!BATCH && tid == 0) {
    for (int k = 0; k < 4; ++k) tacc[k] = 0;
    tp = tp0 = clock64();
    ns0 = globaltimer_ns();
  }
  auto stamp = [&](int k) {
    if (timer) {
      const long long now = clock64();
      tacc[k] += now - tp;
      tp = now;
    }
  };
  // A warp: the CTA's pair to every copy of a grid-wide array; and the copy
  // this CTA reads.
  auto publish_pair = [&](unsigned long long* to, fpair t, unsigned tag) {
    ll_store(to + ((size_t)(lane >> 1) * G + cta) * 2 + (lane & 1),
             (lane & 1) ? t.lo : t.hi, tag);
  };
  const size_t my_copy = (size_t)(cta % kPairCopies) * G * 2;
  // the words of the residual of iteration k
  auto res_words = [&](int k) {
    return P.resx + residual_slot(k, MODE == MODE_GL || P.check_all) * ((size_t)kPairCopies * G * 2);
  };
  // Residual warp: the CTA's squared residual to the grid, and the grid's
  // with the decision.
  auto publish_res = [&](unsigned long long* to, unsigned tag, bool mute) {
    const fpair t = warp_sum_nonneg(lane < item_warps ? s_res[lane] : fp_make(0.0f));
    if (G == 1) {
      if (lane == 0) s_own = t;
    } else if (!mute) {
      publish_pair(to, t, tag);
    }
  };
  const float stop_hi = (float)P.res2_stop;
  auto decide = [&](const unsigned long long* from, unsigned tag) {
    if (G > 1) {
      const PairSum t = ll_pairs(from + my_copy, G, tag, P.abort_flag, P.timeout_ns, wait.failed);
      wait.failed = t.failed;
      if (lane == 0) s_r2 = t.v;
    } else if (lane == 0) {
      s_r2 = s_own;
    }
    __syncwarp();
    if (lane == 0) s_stop = below(s_r2, P.res2_stop, stop_hi);
  };

  for (; it < P.max_iters; ++it) {
    const int par = it & 1, prv = par ^ 1;
    const bool even = par == 0;
    const bool mute = it == 0 && cta == P.stall_cta;  // test hook
    if (BATCH && cta == 0 && tid == 0 && (it & 15) == 0) atomicAdd(P.beat, 1u);

    // ------------------------------------------------ X-update of the tile
    // phi = (staged dual + gamma) / n of this lane's rows and of the warp's
    // columns (lane j: column j); -inf beyond the tile.
    f32x2 f01, f23;
    float f2l, f2h = NEG_INF;  // columns below 32, and from 32 on
    {
      float f1[4] = {NEG_INF, NEG_INF, NEG_INF, NEG_INF};
      f2l = NEG_INF;
      if (it == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (r0 + e >= head && r0 + e < h) f1[e] = __ldg(P.phi1 + base + r0 + e);
        if (lane < ncw) f2l = __ldg(P.phi2 + c0 + wj0 + lane);
        if (lane + 32 < ncw) f2h = __ldg(P.phi2 + c0 + wj0 + lane + 32);
      } else {
        const float gamma = s_gamma[prv];
        float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r0 < h) d = *reinterpret_cast<const float4*>(s_t1 + prv * rt + r0);
        const float u[4] = {d.x + gamma, d.y + gamma, d.z + gamma, d.w + gamma};
        const float u2 = (lane < ncw ? s_t2[prv * ct + wj0 + lane] : 0.0f) + gamma;
        unsigned tiny = ((unsigned)__float_as_int(u2) & 0x7fffffffu) - 1u;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          tiny = min(tiny, ((unsigned)__float_as_int(u[e]) & 0x7fffffffu) - 1u);
        if (tiny < kDivTinyBitsM1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) f1[e] = u[e] / nc_f;
          f2l = u2 / nr_f;
        } else {
          const f32x2 nn = x2_pack(-nc_f, -nc_f), rr = x2_pack(P.nc_rcp, P.nc_rcp);
          x2_unpack(x2_div_rn_by_fma(x2_pack(u[0], u[1]), nn, rr), f1[0], f1[1]);
          x2_unpack(x2_div_rn_by_fma(x2_pack(u[2], u[3]), nn, rr), f1[2], f1[3]);
          f2l = div_rn_by_fma(u2, nr_f, P.nr_rcp);
        }
        if (!full) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (r0 + e < head || r0 + e >= h) f1[e] = NEG_INF;
        }
        if (lane >= ncw) f2l = NEG_INF;
        if (lane + 32 < ncw)
          f2h = div_rn_by(s_t2[prv * ct + wj0 + lane + 32] + gamma, nr_f, P.nr_rcp);
      }
      f01 = x2_pack(f1[0], f1[1]);
      f23 = x2_pack(f1[2], f1[3]);
    }
    const f32x2 ns2 = x2_pack(-s, -s);
    f32x2 a01 = x2_pack(0.0f, 0.0f), a23 = a01;  // row sums of the lane's rows
    float* const cpart = s_col + wr * ct + wj0;  // the warp's column sums
    if constexpr (MODE == MODE_QR) {
      // Even iterations read C and store the folded X^ - sC.  Four columns a
      // step (the slots are padded to whole steps).
      const f32x2 nk = x2_pack(-kappa, -kappa), ky = x2_pack(kappa_rcp, kappa_rcp);
      // where a step finds X and C: both in shared memory, C in global memory,
      // both in global memory (the lane's rows of a column are one vector)
      float* const xg = P.x + (long long)(c0 + wj0) * ld + base + r0;
      const CT* const ccol = cg + (long long)(c0 + wj0) * ld + base + r0;
      auto update = [&](auto even_tag, auto two_tag) {
        constexpr bool EV = decltype(even_tag)::value, TWO = decltype(two_tag)::value;
        const float4* xi = EV ? xb : xa;
        float4* xo = EV ? xa : xb;
        const CSlot* ci = cs;
        f32x2 o01 = x2_pack(0.0f, 0.0f), o23 = o01;
        auto divide = [&](float m0, float m1) {
          const f32x2 m = x2_pack(m0, m1);
          return TWO ? x2_div_rn_two(m, nk, ky) : x2_div_rn_by_fma(m, nk, ky);
        };
        auto steps = [&](auto place_tag, int j_from, int j_to) {
          constexpr int PLACE = decltype(place_tag)::value;  // 0, 1, 2 as above
#pragma unroll 1
          for (int j0 = j_from; j0 < j_to; j0 += 4) {
            float x[4][4], col[4];
            f32x2 c01[4], c23[4];
            unsigned tm[4];
            const float f2w = j0 < 32 ? f2l : f2h;
            f32x2 x01[4], x23[4];
            if constexpr (PLACE > 0) {
              // the global loads of the step first
              float v[4][4], w[4][4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[u][e] = w[u][e] = 0.0f;
                if (live_lane && j0 + u < ncw) {
                  if constexpr (PLACE == 2) load_vec<4>(xg + (long long)(j0 + u) * ld, v[u]);
                  if constexpr (EV) load_c_raw<4, CT>(ccol + (long long)(j0 + u) * ld, w[u]);
                }
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                if constexpr (PLACE == 2) {
                  x01[u] = x2_pack(v[u][0], v[u][1]);
                  x23[u] = x2_pack(v[u][2], v[u][3]);
                }
                if constexpr (EV) c_inside(w[u], c01[u], c23[u]);
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if constexpr (PLACE < 2) x_pairs(xi[u * T], x01[u], x23[u]);
              if constexpr (PLACE == 0 && EV) c_pairs(ci[u * T], c01[u], c23[u]);
              const float f2 = __shfl_sync(0xffffffffu, f2w, (j0 + u) & 31);
              const f32x2 f2b = x2_pack(f2, f2);
              f32x2 t01 = x2_add(x2_add(x01[u], f01), f2b);
              f32x2 t23 = x2_add(x2_add(x23[u], f23), f2b);
              if constexpr (EV) {
                t01 = x2_fma(ns2, c01[u], t01);
                t23 = x2_fma(ns2, c23[u], t23);
              }
              x2_unpack(t01, x[u][0], x[u][1]);
              x2_unpack(t23, x[u][2], x[u][3]);
            }
            // min of (bits - 1): one instruction per element
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              tm[u] = (unsigned)__float_as_int(x[u][0]) - 1u;
#pragma unroll
              for (int e = 1; e < 4; ++e)
                tm[u] = __viaddmin_u32((unsigned)__float_as_int(x[u][e]), 0xffffffffu, tm[u]);
            }
            // a nonzero dividend below 2^-90 anywhere: the IEEE division
            const bool slow = __any_sync(0xffffffffu,
                                         min(min(tm[0], tm[1]), min(tm[2], tm[3])) < kDivTinyBitsM1);
            f32x2 y01[4], y23[4];
            if (__builtin_expect(slow, 0)) {
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                y01[u] = x2_pack(div_ieee(fmaxf(x[u][0], 0.0f), kappa),
                                 div_ieee(fmaxf(x[u][1], 0.0f), kappa));
                y23[u] = x2_pack(div_ieee(fmaxf(x[u][2], 0.0f), kappa),
                                 div_ieee(fmaxf(x[u][3], 0.0f), kappa));
              }
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                y01[u] = divide(fmaxf(x[u][0], 0.0f), fmaxf(x[u][1], 0.0f));
                y23[u] = divide(fmaxf(x[u][2], 0.0f), fmaxf(x[u][3], 0.0f));
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              f32x2 n01 = y01[u], n23 = y23[u];
              if constexpr (EV) {
                n01 = x2_fma(ns2, c01[u], n01);
                n23 = x2_fma(ns2, c23[u], n23);
                o01 = x2_fma(y01[u], c01[u], o01);
                o23 = x2_fma(y23[u], c23[u], o23);
              }
              if constexpr (PLACE < 2) {
                put_x(xo[u * T], n01, n23);
              } else if (live_lane && j0 + u < ncw) {
                set_x(xg + (long long)(j0 + u) * ld, n01, n23);
              }
              float u0, u1;
              x2_unpack(x2_add(y01[u], y23[u]), u0, u1);
              col[u] = u0 + u1;
            }
            // the step's columns first: a quarter of the additions in one chain
            a01 = x2_add(a01, x2_add(x2_add(y01[0], y01[1]), x2_add(y01[2], y01[3])));
            a23 = x2_add(a23, x2_add(x2_add(y23[0], y23[1]), x2_add(y23[2], y23[3])));
            const float cv = fold_columns<4>(col, lane);
            if (lane < 4 && j0 + lane < ncw) cpart[j0 + lane] = cv;
            xi += 4 * T;
            xo += 4 * T;
            ci += 4 * T;
          }
          };
        steps(std::integral_constant<int, 0>(), 0, min(nsc, ncw));
        if (nsc < ncw) {
          steps(std::integral_constant<int, 1>(), nsc, min(nsx, ncw));
          steps(std::integral_constant<int, 2>(), nsx, ncw);
        }
        if constexpr (EV) {
          ob01 = o01;
          ob23 = o23;
        }
      };
      if (P.two_step) {
        if (even) update(std::true_type(), std::true_type());
        else update(std::false_type(), std::true_type());
      } else {
        if (even) update(std::true_type(), std::false_type());
        else update(std::false_type(), std::false_type());
      }
    } else {
      // y = max((X + phi1) + phi2 - sC, 0) and the class's norm per column,
      // then the shrink; eight columns a step.
      const float4* xi = even ? xb : xa;
      float4* xo = even ? xa : xb;
      const CSlot* ci = cs;
      float* const xg = P.x + (long long)(c0 + wj0) * ld + base + r0;
      const CT* const ccol = cg + (long long)(c0 + wj0) * ld + base + r0;
      auto steps = [&](auto place_tag, int j_from, int j_to) {
        constexpr int PLACE = decltype(place_tag)::value;  // 0, 1, 2 as for QR
#pragma unroll 1
        for (int j0 = j_from; j0 < j_to; j0 += 8) {
          f32x2 y01[8], y23[8];
          float col[8];
          const float f2w = j0 < 32 ? f2l : f2h;
          [[maybe_unused]] float gv[4][4], gw[4][4];  // four columns in flight
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if constexpr (PLACE > 0) {
              if ((u & 3) == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
#pragma unroll
                  for (int e = 0; e < 4; ++e) gv[k][e] = gw[k][e] = 0.0f;
                  if (live_lane && j0 + u + k < ncw) {
                    const long long off = (long long)(j0 + u + k) * ld;
                    if constexpr (PLACE == 2) load_vec<4>(xg + off, gv[k]);
                    load_c_raw<4, CT>(ccol + off, gw[k]);
                  }
                }
              }
            }
            f32x2 t01, t23, c01, c23;
            if constexpr (PLACE < 2) {
              x_pairs(xi[u * T], t01, t23);
            } else {
              t01 = x2_pack(gv[u & 3][0], gv[u & 3][1]);
              t23 = x2_pack(gv[u & 3][2], gv[u & 3][3]);
            }
            if constexpr (PLACE == 0) c_pairs(ci[u * T], c01, c23);
            else c_inside(gw[u & 3], c01, c23);
            const float f2 = __shfl_sync(0xffffffffu, f2w, (j0 + u) & 31);
            const f32x2 f2b = x2_pack(f2, f2);
            t01 = x2_fma(ns2, c01, x2_add(x2_add(t01, f01), f2b));
            t23 = x2_fma(ns2, c23, x2_add(x2_add(t23, f23), f2b));
            float v[4];
            x2_unpack(t01, v[0], v[1]);
            x2_unpack(t23, v[2], v[3]);
            y01[u] = x2_pack(fmaxf(v[0], 0.0f), fmaxf(v[1], 0.0f));
            y23[u] = x2_pack(fmaxf(v[2], 0.0f), fmaxf(v[3], 0.0f));
            x2_unpack(x2_fma(y23[u], y23[u], x2_mul(y01[u], y01[u])), v[0], v[1]);
            col[u] = v[0] + v[1];
          }
          const int jl = j0 + (lane & 7);
          float nsl = fold_columns<8>(col, lane);
          if (WR > 1) {
            if (lane < 8 && jl < ncw) s_nrm[wr * ct + wj0 + jl] = nsl;
            asm volatile("bar.sync %0, %1;" :: "r"(1 + wc), "r"(WR * 32) : "memory");
            nsl = 0.0f;
            if (jl < ncw)
              for (int k = 0; k < WR; ++k) nsl += s_nrm[k * ct + wj0 + jl];
          }
          const float scale = gl_shrink(nsl, P.lambda);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const float sc = __shfl_sync(0xffffffffu, scale, u);
            const f32x2 sc2 = x2_pack(sc, sc);
            const f32x2 z01 = x2_mul(y01[u], sc2), z23 = x2_mul(y23[u], sc2);
            if constexpr (PLACE < 2) {
              put_x(xo[u * T], z01, z23);
            } else if (live_lane && j0 + u < ncw) {
              set_x(xg + (long long)(j0 + u) * ld, z01, z23);
            }
            a01 = x2_add(a01, z01);
            a23 = x2_add(a23, z23);
            float u0, u1;
            x2_unpack(x2_add(z01, z23), u0, u1);
            col[u] = u0 + u1;
          }
          const float cv = fold_columns<8>(col, lane);
          if (lane < 8 && jl < ncw) cpart[jl] = cv;
          xi += 8 * T;
          xo += 8 * T;
          ci += 8 * T;
        }
      };
      steps(std::integral_constant<int, 0>(), 0, min(nsc, ncw));
      if constexpr (BATCH) {
        if (nsc < ncw) {
          steps(std::integral_constant<int, 1>(), nsc, min(nsx, ncw));
          steps(std::integral_constant<int, 2>(), nsx, ncw);
        }
      }
    }
    // ------------------------------------------------ the tile's sums
    if (wc < WC)  // warps beyond the tiling hold nothing
      put_x(*reinterpret_cast<float4*>(s_row + wc * WR * 128 + r0), a01, a23);
    __syncthreads();
    stamp(0);
    // n partials, `stride` floats apart, four at a time
    auto add_up = [](const float* p, int n, int stride) {
      if (n == 1) return p[0];
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
      for (int k = 0; k < n; k += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] += k + u < n ? p[(k + u) * stride] : 0.0f;
      return (v[0] + v[1]) + (v[2] + v[3]);
    };
    auto row_sum = [&](int i) { return add_up(s_row + i, WC, WR * 128); };
    auto col_sum = [&](int j) { return add_up(s_col + j, WR, ct); };
    const bool check = MODE == MODE_GL || even || P.check_all;
    // ------------------------------------------------ exchange and duals
    int level = 0;  // < 0: class round
    bool decided = false;
    for (;; ++rd) {
      const int rp = rd & 1;
      const float up = level < 0 ? 0.0f : pow2f(kRowBits - kLevelBits * level);
      if (warp == mass_warp) {
        // the plan's mass, then gamma and alpha
        float sg = 0.0f;
        int next = 0;  // next round's level: 0 none
        if (G == 1) {
          fpair t = fp_make(0.0f);
          for (int j = lane; j < w; j += 32) t = fp_add(t, fp_make(col_sum(j)));
          t = warp_sum_nonneg(t);
          sg = t.hi + t.lo;
        } else {
          const float upm = level < 0 ? 0.0f : pow2f(kMassBits - kLevelBits * level);
          const unsigned long long most = (1ull << 47) / (unsigned)G;
          unsigned long long n = 0ull;
          bool odd_value = false, over = false;
          for (int j = lane; j < w; j += 32) {
            const float v = col_sum(j);
            if (level < 0) {
              n += class_word(v);
            } else {
              const bool fin = v <= 3.402823466e38f;
              odd_value |= !fin;
              const float f = fin ? v * upm : 0.0f;
              over |= !(f < (float)most);
              if (f < (float)most) n += to_fixed(f);
            }
          }
          // exact warp sum of 49-bit numbers in three words
          const unsigned n0 = __reduce_add_sync(0xffffffffu, (unsigned)(n & 0xfffffu));
          const unsigned n1 = __reduce_add_sync(0xffffffffu, (unsigned)((n >> 20) & 0xfffffu));
          const unsigned n2 = __reduce_add_sync(0xffffffffu, (unsigned)(n >> 40));
          n = n0 + ((unsigned long long)n1 << 20) + ((unsigned long long)n2 << 40);
          odd_value = __any_sync(0xffffffffu, odd_value);
          over = __any_sync(0xffffffffu, over) || n >= most;
          if (level < 0) {
            n = (n >> 40) ? 1ull << 40 : (n >> 20) ? 1ull << 20 : 0ull;
            over = odd_value = false;
          }
          unsigned long long* const mw = P.massx + 32 * rp;
          if (lane == 0) {
            if (over) {
              atomicExch(P.over_flag, (int)(rd + 1u));
              __threadfence();
            }
            if (!mute)
              word_add(mw, kCountOne + (over || odd_value ? kPoisonOne : n));
            unsigned long long got = ll_load(mw);
            wait.until([&]() {
              if ((unsigned)((got - mass_seen[rp]) >> 56) == (unsigned)G) return true;
              got = ll_load(mw);
              return false;
            });
            const unsigned long long d = got - mass_seen[rp];
            mass_seen[rp] = got;
            if (level < 0) {
              sg = class_value(d & (kPoisonOne - 1ull));
            } else if ((d >> 48) & 0xffull) {
              __threadfence();
              next = ld_volatile_i32(P.over_flag) == (int)(rd + 1u) ? level + 1 : -1;
            } else {
              sg = from_fixed(d & (kPoisonOne - 1ull)) * pow2f(kLevelBits * level - kMassBits);
            }
          }
        }
        if (lane == 0) {
          s_level = next;
          if (next == 0) {
            const float al = alpha;
            s_gamma[par] = gamma_of(sg, al, (float)(P.nr + P.nc), P.n_rcp);
            alpha_prev = al;
            alpha = alpha_next(sg, al);
            sigma_prev = sigma;
            sigma = sg;
          }
        }
      } else if (warp == res_warp) {
        // the residual of the iteration before (once), then this one's
        if (P.keep && pend >= 0 && !decided)
          decide(res_words(pend), pend_tag);
        if (check) {
          asm volatile("bar.sync 15, %0;" :: "r"((item_warps + 1) * 32) : "memory");
          publish_res(res_words(it), rd + 1u, mute);
        }
      } else if (warp < item_warps) {
        unsigned long long* const rowp = P.rowx + (size_t)(rp * P.GR + br) * rt;
        unsigned long long* const colp = P.colx + (size_t)(rp * P.GC + bc) * ct;
        float tot[NI];
#pragma unroll
        for (int u = 0; u < NI; ++u) {
          const int i = tid + u * IT;
          if (u * IT >= n_items) break;
          tot[u] = 0.0f;
          if (i < n_items) {
            const bool row = i < hr;
            const float v = row ? row_sum(head + i) : col_sum(i - hr);
            tot[u] = v;
            const int np = row ? P.GC : P.GR;
            if (np > 1 && !mute) {
              unsigned long long n;
              if (level < 0) n = class_word(v);
              else n = to_fixed(fminf(v * up, np == 1 ? 0.0f : (row ? most_r : most_c)));
              word_add(row ? rowp + head + i : colp + i - hr, kCountOne + n);
            }
          }
        }
        // One word at a time: the later ones are complete when the first is,
        // and polls of lines that additions still go to delay these (all of a
        // thread's words polled together: GL 1500 x 1000 6.6 us per iteration
        // against 5.7).
        fpair res = fp_make(0.0f);
#pragma unroll
        for (int u = 0; u < NI; ++u) {
          const int i = tid + u * IT;
          if (u * IT >= n_items) break;
          if (i < n_items) {
            const bool row = i < hr;
            const int np = row ? P.GC : P.GR;
            if (np > 1) {
              const unsigned long long* const wp = row ? rowp + head + i : colp + i - hr;
              unsigned long long old;
              if constexpr (BATCH) old = s_seen[(rp ? seen_n : 0) + i];
              else old = rp ? seen[1][u] : seen[0][u];
              unsigned long long got = ll_load(wp);
              wait.until([&]() {
                if ((unsigned)((got - old) >> 56) == (unsigned)np) return true;
                got = ll_load(wp);
                return false;
              });
              const unsigned long long n = (got - old) & (kCountOne - 1ull);
              if constexpr (BATCH) s_seen[(rp ? seen_n : 0) + i] = got;
              else if (rp) seen[1][u] = got;
              else seen[0][u] = got;
              tot[u] = level < 0 ? class_value(n)
                                 : from_fixed(n) * pow2f(kLevelBits * level - kRowBits);
            }
            if (level < 0) {
              if (np == 1 || tot[u] == 0.0f) continue;  // finite: the round before updated it
              if constexpr (LEAN) dual[u] = s_prev[i];
              else dual[u] = dual_prev[u];
            }
            const float rs = tot[u] - (LEAN ? s_marg[i] : marg[u]);
            if constexpr (LEAN) s_prev[i] = dual[u];
            else dual_prev[u] = dual[u];
            dual[u] = dual[u] - rs;
            if (row) s_t1[par * rt + head + i] = dual[u] - rs;
            else s_t2[par * ct + i - hr] = dual[u] - rs;
            if (row ? i >= sr0 && i < sr1 : i >= sc0 && i < sc1) res = fp_add(res, fp_sqr(rs));
          }
        }
        if (check) {
          if (__any_sync(0xffffffffu, res.hi != 0.0f)) res = warp_sum_nonneg(res);
          if (lane == 0) s_res[warp] = res;
          asm volatile("bar.arrive 15, %0;" :: "r"((item_warps + 1) * 32) : "memory");
        }
      }
      stamp(1);
      if (__syncthreads_or(wait.failed ? 1 : 0)) { aborted = true; break; }
      if (P.keep && pend >= 0 && !decided) {
        last_r2 = s_r2;
        decided = true;
      }
      const int next = s_level;
      if (next == 0) {
        // a stop ends the loop after a round that the words held, which leaves
        // alpha and the duals one iteration ahead together
        if (decided && s_stop) stop_it = pend;
        break;
      }
      // The words could not hold this round: again on a coarser scale, or the
      // sums that are not finite.
      level = next;
      if (next > 0) {
#pragma unroll
        for (int u = 0; u < NI; ++u) {
          const int i = tid + u * IT;
          if constexpr (!LEAN) dual[u] = dual_prev[u];
          else if (warp < res_warp && i < n_items) dual[u] = s_prev[i];
        }
      }
      __syncthreads();
    }
    ++rd;
    stamp(2);
    if (aborted || stop_it >= 0) break;
    if (MODE == MODE_GL || even) obj_valid = 1;
    pend = -1;
    if (check) {
      pend = it;
      pend_tag = rd;
      if (!P.keep) {
        if (warp == res_warp) decide(res_words(it), pend_tag);
        if (__syncthreads_or(wait.failed ? 1 : 0)) { aborted = true; break; }
        last_r2 = s_r2;
        if (s_stop) { stop_it = it; break; }
      }
    }
    stamp(3);
  }
  if (P.keep && stop_it < 0 && !aborted && pend >= 0) {
    // max_iters ended on an iteration that is checked: its residual is still out
    if (warp == res_warp) decide(res_words(pend), pend_tag);
    if (__syncthreads_or(wait.failed ? 1 : 0)) aborted = true;
    last_r2 = s_r2;
    if (!aborted && s_stop) stop_it = pend;
  }

  // ------------------------------------------------ epilogue
  const bool converged = stop_it >= 0;
  const int last_it = converged ? stop_it : it - 1;
  const bool back = converged && it > stop_it && it < P.max_iters;  // X is one step ahead
  const bool unfold = MODE == MODE_QR && (converged || P.check_all) && last_it >= 0 &&
                      (last_it & 1) == 0 && !aborted;
  // where the last iteration left X (nothing run: where it was loaded)
  const float4* const xf = last_it >= 0 && (last_it & 1) == 0 ? xa : xb;
  for (int j = 0; j < ncw; ++j) {
    f32x2 x01, x23, c01, c23;
    float v[4];
    float* const xp = P.x + (long long)(c0 + wj0 + j) * ld + base + r0;
    if (j < nsx) {
      x_pairs(xf[j * T], x01, x23);
    } else {
      if ((MODE == MODE_QR && !unfold) || !live_lane) continue;  // in place already
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = 0.0f;
      load_vec<4>(xp, v);
      x01 = x2_pack(v[0], v[1]);
      x23 = x2_pack(v[2], v[3]);
    }
    if (j < nsc) {
      c_pairs(cs[j * T], c01, c23);
    } else {
      float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (live_lane) load_c_raw<4, CT>(cg + (long long)(c0 + wj0 + j) * ld + base + r0, w);
      c_inside(w, c01, c23);
    }
    if constexpr (MODE == MODE_QR) {
      const f32x2 s2 = x2_pack(s, s);
      if (unfold) {
        x01 = x2_fma(s2, c01, x01);
        x23 = x2_fma(s2, c23, x23);
      }
      x2_unpack(x01, v[0], v[1]);
      x2_unpack(x23, v[2], v[3]);
      if (unfold) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = fmaxf(v[e], 0.0f);
      }
    } else {
      // <C, X> of the last iteration: X is that iteration's
      x2_unpack(x01, v[0], v[1]);
      x2_unpack(x23, v[2], v[3]);
      ob01 = x2_fma(x01, c01, ob01);
      ob23 = x2_fma(x23, c23, ob23);
    }
    if (whole) {
      store_vec<4>(xp, v);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r0 + e >= head && r0 + e < h) xp[e] = v[e];
    }
  }
  if (!aborted && last_it >= 0 && warp < res_warp) {
    const int fp = last_it & 1;
    const float gamma = s_gamma[fp];
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int i = tid + u * IT;
      float d = dual[u];
      if (back) {
        if constexpr (!LEAN) d = dual_prev[u];
        else if (i < n_items) d = s_prev[i];
      }
      if (i >= sr0 && i < sr1) {
        P.a[lo + i] = d;
        P.phi1[lo + i] = div_rn_by(s_t1[fp * rt + head + i] + gamma, nc_f, P.nc_rcp);
      } else if (i >= sc0 && i < sc1) {
        P.b[c0 + i - hr] = d;
        P.phi2[c0 + i - hr] = div_rn_by(s_t2[fp * ct + i - hr] + gamma, nr_f, P.nr_rcp);
      }
    }
  }
  if (cta == 0 && warp == mass_warp && lane == 0) {
    if constexpr (!BATCH) P.stats->sigma = back ? sigma_prev : sigma;
    P.alpha[BATCH ? ((last_it + 1) & 1) * P.alpha_stride : 0] = back ? alpha_prev : alpha;
  }
  // objective: CTA pairs to CTA 0
  float u[4];
  x2_unpack(ob01, u[0], u[1]);
  x2_unpack(ob23, u[2], u[3]);
  const fpair ob = fp_add(fp_add(fp_make(u[0]), fp_make(u[1])),
                          fp_add(fp_make(u[2]), fp_make(u[3])));
  const fpair cta_ob = block_sum_fp(ob, s_sum);
  if (warp == 0) {
    if (lane < 2 && G > 1 && !aborted)
      ll_store(P.objx + 2 * cta + lane, lane == 0 ? cta_ob.hi : cta_ob.lo, 1u);
    if (cta == 0) {
      fpair t = cta_ob;
      if (G > 1 && !aborted) {
        const PairSum all = ll_pairs(P.objx, G, 1u, P.abort_flag, P.timeout_ns, wait.failed);
        wait.failed = all.failed;
        t = all.v;
      }
      const bool late = __any_sync(0xffffffffu, wait.failed);
      const double r2 = fp_value(last_r2);
      if (BATCH && lane == 0) {
        BatchRecord r;
        r.iters_run = last_it + 1;
        r.n_iter = MODE == MODE_QR ? (converged ? stop_it : it) + 1 : r.iters_run;
        r.converged = converged ? 1 : 0;
        r.objective_valid = obj_valid;
        r.objective = obj_valid && !aborted ? fp_value(t) : 0.0;
        r.residual = r2;  // squared; -1 before the first test
        *P.record = r;
      }
      if (!BATCH && lane == 0) {
        DeviceStats* st = P.stats;
        st->iters_run = converged ? stop_it + 1 : it;
        // QR: index of the last iteration + 1, max_iters + 1 without
        // convergence (drot_qr.hpp:233); GL: iterations run (drot_glr.hpp:354)
        st->n_iter = MODE == MODE_QR ? (converged ? stop_it : it) + 1 : st->iters_run;
        st->converged = converged ? 1 : 0;
        st->status = (aborted || late || ld_volatile_i32(P.abort_flag)) ? 3 : 0;
        st->objective_valid = obj_valid;
        st->objective = obj_valid && !aborted ? fp_value(t) : 0.0;
        st->residual = r2 >= 0.0 ? sqrt(r2) : r2;
      }
    }
  }
  if (!BATCH && timer) {
    const double scale = (double)(globaltimer_ns() - ns0) / (double)max(1ll, clock64() - tp0);
    for (int k = 0; k < 4; ++k) P.stats->phase_ns[k] = (double)tacc[k] * scale;
  }
}

template <int MODE, typename CT, int T>
__global__ void __launch_bounds__(T, 1)
drot_resident_kernel(const __grid_constant__ ResidentParams P,
                     const __grid_constant__ ResidentBounds B) {
  resident_solve<MODE, CT, T, false>(P, B.row, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// Batches
// ---------------------------------------------------------------------------
//
// Many problems in one cooperative launch of two 8-warp CTAs per SM.  Every
// instance runs on as many CTAs as its tiling has, from its first iteration
// to its stop, and meets no other instance; two instances share an SM, so one
// computes while the other waits for its exchange.  The streaming batch kernel
// takes all instances through every iteration together, so their X and C pass
// through HBM once per iteration; here only the few that run at a time are
// read, from L2 where shared memory does not hold them.  us per iteration,
// streaming -> here: QR 4 instances of 64..512 rows and columns 19 -> 3.5, 8 of
// 64..2048 30 -> 14, 32 of them (34 M elements) 86 -> 50, 256 (296 M) 501 ->
// 442; GL 4 of 256..1024 22 -> 7.6, 16 of 256..2048 96 -> 67.  Bound by the
// arithmetic and the shared-memory pipe of the steps, 0.35 clocks per element
// and SM for QR (of 0.30 with one tile of 16 warps), and by the CTAs that have
// nothing to run towards the end (15 % for the 32).
//
// CTAs wait in a mailbox for (instance, tile); the last CTA of an instance to
// finish returns its CTAs to the free list and starts the next instances that
// fit (in order of work, the first that fits), under a lock; the first ones are
// in the mail at the launch.  Which CTAs run a tile does not enter any sum.
// Every wait is bounded: for work, by the time since any instance made progress
// (the heartbeat that first tiles raise every 16 iterations); for the lock, by
// the limit of the exchanges.

// Warp 0 with the lock held: starts instances while one fits the free CTAs.
__device__ __noinline__ void resident_schedule(const ResidentBatch& B) {
  const int lane = threadIdx.x & 31;
  int free = __ldcg(B.sched + kSchedFree), head = __ldcg(B.sched + kSchedHead);
  for (;;) {
    // the first one not started, then the first from there on that fits
    while (head < B.n_inst) {
      const int i = head + lane;
      const unsigned open =
          __ballot_sync(0xffffffffu, i < B.n_inst && __ldcg(B.taken + i) == 0u);
      head += open ? __ffs(open) - 1 : 32;
      if (open) break;
    }
    unsigned fits[kBatchWindow / 32];
#pragma unroll
    for (int r = 0; r < kBatchWindow / 32; ++r) {
      const int i = head + 32 * r + lane;
      fits[r] = __ballot_sync(0xffffffffu, i < B.n_inst && __ldcg(B.taken + i) == 0u &&
                                               B.need[i] <= free);
    }
    int pick = -1;
#pragma unroll
    for (int r = kBatchWindow / 32 - 1; r >= 0; --r)
      if (fits[r]) pick = head + 32 * r + __ffs(fits[r]) - 1;
    if (pick < 0) break;
    const int n = B.need[pick];
    for (int t = lane; t < n; t += 32) {
      const int c = __ldcg(B.free_list + free - 1 - t);
      B.cta_of[B.inst[pick].tile0 + t] = c;
      asm volatile("st.release.gpu.global.u32 [%0], %1;"
                   :: "l"(B.mail + c), "r"(((unsigned)(pick + 1) << kMailTileBits) | (unsigned)t)
                   : "memory");
    }
    if (lane == 0) B.taken[pick] = 1u;
    free -= n;
    __syncwarp();
  }
  if (lane == 0) {
    B.sched[kSchedFree] = free;
    B.sched[kSchedHead] = head;
  }
  __threadfence();
  __syncwarp();
}

// Warp 0 of the last CTA of instance k: its CTAs are free again.
__device__ __noinline__ void resident_finish(const ResidentBatch& B, const ResidentInst& I) {
  const int lane = threadIdx.x & 31;
  int locked = 1;
  if (lane == 0) {
    LLWait wait = {B.abort_flag, B.timeout_ns, false};
    wait.until([&]() {
      if (atomicCAS(B.sched + kSchedLock, 0, 1) == 0) return true;
      __nanosleep(100);
      return false;
    });
    locked = !wait.failed;
  }
  if (!__shfl_sync(0xffffffffu, locked, 0)) return;
  __threadfence();
  const int free = __ldcg(B.sched + kSchedFree);
  for (int t = lane; t < I.n; t += 32) B.free_list[free + t] = __ldcg(B.cta_of + I.tile0 + t);
  const int left = __ldcg(B.sched + kSchedLeft) - 1;
  __syncwarp();
  if (lane == 0) {
    B.sched[kSchedFree] = free + I.n;
    B.sched[kSchedLeft] = left;
  }
  __threadfence();
  __syncwarp();
  if (left == 0) {
    for (int c = lane; c < (int)gridDim.x; c += 32)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(B.mail + c), "r"(kMailEnd)
                   : "memory");
  } else {
    resident_schedule(B);
  }
  __threadfence();
  __syncwarp();
  if (lane == 0) atomicExch(B.sched + kSchedLock, 0);
}

// One thread: the next mail of this CTA.
__device__ __noinline__ unsigned resident_mail(const ResidentBatch& B) {
  unsigned* const mine = B.mail + blockIdx.x;
  unsigned long long t0 = globaltimer_ns();
  int beat = 0;
  for (unsigned spins = 0;; ++spins) {
    unsigned m;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(m) : "l"(mine) : "memory");
    if (m == kMailEnd) return m;
    if (m != 0u) {
      // the next one cannot be written before this CTA has finished this tile
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" :: "l"(mine), "r"(0u) : "memory");
      return m;
    }
    if ((spins & 15u) == 15u) {
      if (ld_volatile_i32(B.abort_flag)) return kMailEnd;
      const unsigned long long now = globaltimer_ns();
      const int b = ld_volatile_i32(B.sched + kSchedBeat);
      if (b != beat) {
        beat = b;
        t0 = now;
      } else if ((long long)(now - t0) > B.timeout_ns) {
        atomicExch(B.abort_flag, 1);
        return kMailEnd;
      }
    }
    __nanosleep(200);
  }
}

template <int MODE, typename CT>
__global__ void __launch_bounds__(256, 2)
drot_resident_batch_kernel(const __grid_constant__ ResidentBatch B) {
  __shared__ ResidentParams prm;
  __shared__ unsigned s_mail;
  const int tid = threadIdx.x, lane = tid & 31, me = blockIdx.x;
  for (;;) {
    if (tid == 0) s_mail = resident_mail(B);
    __syncthreads();
    const unsigned m = s_mail;
    if (m == kMailEnd) break;
    const int k = (int)(m >> kMailTileBits) - 1, tile = (int)(m & ((1u << kMailTileBits) - 1u));
    const ResidentInst& I = B.inst[k];
    if (tid == 0) {
      const ResidentTiling& g = I.tiling;
      prm.c = reinterpret_cast<const CT*>(B.c) + I.c_off;
      prm.x = B.x + I.x_off;
      prm.p = B.p + I.p_off;
      prm.q = B.q + I.q_off;
      prm.a = B.a + I.row_off;
      prm.phi1 = B.phi1 + I.row_off;
      prm.b = B.b + I.col_off;
      prm.phi2 = B.phi2 + I.col_off;
      prm.alpha = B.alpha + I.index;
      prm.alpha_stride = B.n_inst;
      prm.nr = I.nr; prm.nc = I.nc; prm.ld = I.ld;
      prm.vec_ok = 1;  // the plan takes only columns on vector boundaries
      prm.s = I.s; prm.kappa = I.kappa; prm.kappa_rcp = I.kappa_rcp;
      prm.nc_rcp = I.nc_rcp; prm.nr_rcp = I.nr_rcp; prm.n_rcp = I.n_rcp;
      prm.lambda = I.lambda;
      prm.two_step = I.two_step;
      prm.res2_stop = I.res2_stop;
      prm.max_iters = B.max_iters;
      prm.check_all = 0;
      prm.GR = g.GR; prm.GC = g.GC; prm.WR = g.WR; prm.WC = g.WC;
      prm.band_h = g.band_h; prm.rt = g.rt; prm.ct = g.ct;
      prm.cw = g.cw; prm.cwp = g.cwp; prm.nsx = g.nsx; prm.nsc = g.nsc; prm.keep = g.keep;
      prm.massx = B.words + I.mass_off;
      prm.resx = B.words + I.res_off;
      prm.objx = B.words + I.obj_off;
      prm.rowx = B.words + I.rowx_off;
      prm.colx = B.words + I.colx_off;
      prm.abort_flag = B.abort_flag;
      prm.over_flag = reinterpret_cast<int*>(prm.massx + 64);
      prm.record = B.records + I.index;
      prm.beat = reinterpret_cast<unsigned*>(B.sched + kSchedBeat);
      prm.stall_cta = B.stall_cta == me ? tile : -1;  // the test hook names a CTA of the launch
      prm.timeout_ns = B.timeout_ns;
    }
    __syncthreads();
    resident_solve<MODE, CT, 256, true>(prm, B.bounds + I.bounds_off, tile, I.n);
    // every thread's writes, then the CTA's count
    __threadfence();
    __syncthreads();
    if (tid < 32) {
      int last = 0;
      if (lane == 0) last = atomicAdd(B.finished + k, 1u) + 1u == (unsigned)I.n;
      if (__shfl_sync(0xffffffffu, last, 0)) {
        __threadfence();
        resident_finish(B, I);
      }
    }
    __syncthreads();
  }
}

}  // namespace drot

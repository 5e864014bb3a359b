// drot_resident.h -- host interface of the resident solve (drot_resident.cu):
// planning and launch of the kernel that keeps one problem's plan on chip.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

#include "drot_exchange.h"
#include "drot_kernels.cuh"

namespace drot {

struct ResidentParams {
  const void* c;  // float or __nv_bfloat16
  const float* p;
  const float* q;
  float* x;
  float *a, *b, *phi1, *phi2, *alpha;
  int nr, nc;
  long long ld;  // leading dimension of X and C
  int vec_ok;  // columns of X and C start on vector boundaries
  float s, kappa, kappa_rcp, nc_rcp, nr_rcp, n_rcp, lambda;  // n_rcp: RN(1 / (nr + nc))
  double res2_stop;
  int max_iters;
  int check_all;  // QR: residual tested on every iteration and a final unfold
                  // whenever the last one folded (numpy-API loop)
  int GR, GC, WR, WC;
  int band_h;     // QR: rows per band
  int rt, ct;     // rows / columns of the largest tile (strides of the buffers)
  int cw, cwp;    // columns per warp, and rounded up to whole steps
  int nsx, nsc;   // columns per warp with X / C in shared memory (nsc <= nsx <= cwp)
  int two_step;   // QR: the short division sequence is exact for kappa
  int keep;       // two copies of X (see the kernel)
  unsigned long long *rowx, *colx;  // [2][GR][rt], [2][GC][ct] counted fixed-point sums
  unsigned long long* massx;        // [2] of them, 256 bytes apart
  unsigned long long* resx;         // [2 slots][kPairCopies][grid][2] tagged (hi, lo)
  unsigned long long* objx;         // [grid][2]
  int *abort_flag, *over_flag;      // over_flag: round + 1 of a mass beyond the words' range
  DeviceStats* stats;
  struct BatchRecord* record;  // batches: instead of stats
  int alpha_stride;            // batches: floats between the parity slots of alpha
  unsigned* beat;              // batches: raised every 16 iterations
  int timer_cta, stall_cta;
  long long timeout_ns;
};

struct ResidentBounds {
  int row[kMaxGroups + 1];  // GL: row boundaries of the classes
};

// An instance's result record in a batch's workspace.
struct BatchRecord {
  int n_iter, iters_run, converged, objective_valid;
  double objective, residual;  // residual: squared on the device, rooted by the host
};

// How an instance of a batch is cut into tiles (fields as in ResidentParams).
struct ResidentTiling {
  int GR, GC, WR, WC, band_h, rt, ct, cw, cwp, nsx, nsc, keep;
};

// One instance of a resident batch launch.
struct ResidentInst {
  long long c_off, x_off, p_off, q_off, ld;             // elements of the caller's buffers
  long long mass_off, res_off, obj_off, rowx_off, colx_off;  // its exchange words
  int nr, nc, row_off, col_off, index;  // index: its place in the caller's list
  int n, tile0, bounds_off;             // CTAs, first entry of its tiles, of its boundaries
  float s, kappa, kappa_rcp, nc_rcp, nr_rcp, n_rcp, lambda;
  int two_step;
  double res2_stop;
  ResidentTiling tiling;
};

// Mail of a CTA of a batch launch: 0 none, kMailEnd, or (instance + 1) <<
// kMailTileBits | tile.
constexpr unsigned kMailEnd = 0xffffffffu;
constexpr int kMailTileBits = 9;
constexpr int kBatchWindow = 64;  // instances looked at for one that fits
// Words of the scheduler's state: lock, free CTAs, first instance not started,
// instances left to finish, heartbeat.
enum { kSchedLock = 0, kSchedFree, kSchedHead, kSchedLeft, kSchedBeat, kSchedWords = 64 };

// A batch launch (drot_resident_batch_kernel).
struct ResidentBatch {
  const void* c;
  const float *p, *q;
  float* x;
  const ResidentInst* inst;
  const int* bounds;       // GL: row boundaries, inst.bounds_off
  float *a, *b, *phi1, *phi2, *alpha;
  BatchRecord* records;
  unsigned long long* words;  // zeroed
  const int* need;         // [n_inst] CTAs of an instance
  // the scheduler's state, as ResidentBatchPlan::state starts it
  int* sched;              // [kSchedWords]
  unsigned* mail;          // [grid]
  unsigned* taken;         // [n_inst] the instance has been started
  unsigned* finished;      // [n_inst] CTAs done
  int* free_list;          // [grid]
  int* cta_of;             // per instance tile: the CTA that runs it
  int* abort_flag;
  int n_inst, max_iters, stall_cta;
  long long timeout_ns;
};

struct ResidentPlan {
  int mode = 0, ctype = 0;
  int GR = 1, GC = 1, WR = 1, WC = 1, band_h = 0, rt = 0, ct = 0, cw = 0, cwp = 0, nsx = 0, nsc = 0,
      keep = 0;
  bool aligned = false;  // needs columns that start on vector boundaries
  int threads = 0, grid = 0;
  size_t smem = 0;
  size_t off_rowx = 0, off_colx = 0, off_massx = 0, off_resx = 0,
         off_objx = 0, total = 0;  // workspace offsets; [0, total) is zeroed before the launch
};

// Plan for a problem whose tiles fit the chip; false where the streaming
// kernel is the one to run.  bounds: GL row boundaries (G + 1 of them).
bool resident_plan(int mode, int nr, int nc, int G, const int* bounds, int ctype, bool check_all,
                   int sms, int smem_optin, ResidentPlan& pl);

// At least the total of every plan of the problem.
size_t resident_most_bytes(int mode, int nr, int nc, int G, const int* bounds, int sms);

// Enqueues the solve; ws holds pl.total bytes, zeroed by the caller on the
// same stream.  prm: problem fields set by the caller, plan fields by this.
cudaError_t resident_launch(const ResidentPlan& pl, ResidentParams& prm,
                            const ResidentBounds& bounds, void* ws, cudaStream_t stream);

// Streaming's estimate holds while every instance is active.  With a budget of
// kLongIters iterations the instances stop one by one, and streaming ends on a
// few that leave the GPU idle: resident tiles are taken up to kLongSolve times
// its estimate there.  Seconds to relative 1e-4, streaming -> resident: 64 QR
// instances of 512..4096 (377 M elements; with all active resident tiles are 3 %
// behind) 5.03 -> 4.66, with BF16 C 4.72 -> 4.46; 256 of 64..2048 with BF16 C
// 2.38 -> 1.87.
constexpr double kLongSolve = 1.1;
constexpr int kLongIters = 2000;

// How a batch runs on resident tiles.  inst: in the order the instances start
// (by decreasing work).
struct ResidentBatchPlan {
  bool ok = false;
  int grid = 0, tiles = 0, first_n = 0;  // first_n: CTAs of the first instance
  size_t smem = 0, words = 0;            // words: 64-bit exchange words of all instances
  // Estimated microseconds per iteration here, and of the streaming kernel with
  // a float and a BF16 cost.
  double us = 0.0, stream_us[2] = {0.0, 0.0};
  std::vector<ResidentInst> inst;
  std::vector<int> bounds, need, state;  // state: the scheduler's at the launch
};

// Tilings for every instance; ok false where an instance has none or the
// streaming kernel is the faster one.  inst: problem fields and `index` set;
// gl_bounds: row boundaries of instance k (GL).
void resident_batch_plan(int mode, const std::vector<ResidentInst>& inst,
                         const std::vector<std::vector<int>>& gl_bounds, int sms,
                         ResidentBatchPlan& pl);

cudaError_t resident_batch_launch(const ResidentBatchPlan& pl, int mode, int ctype,
                                  const ResidentBatch& b, cudaStream_t stream);

}  // namespace drot

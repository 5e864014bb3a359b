// drot_resident.h -- host interface of the resident solve (drot_resident.cu):
// planning and launch of the kernel that keeps one problem's plan on chip.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

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
  unsigned long long* resx;         // [2][kPairCopies][grid][2] tagged (hi, lo)
  unsigned long long* objx;         // [grid][2]
  int *abort_flag, *odd_flag;       // odd_flag: iteration + 1 of a sum that was not finite
  DeviceStats* stats;
  int timer_cta, stall_cta;
  long long timeout_ns;
  int gbounds[kMaxGroups + 1];
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

// Enqueues the solve; ws holds pl.total bytes, zeroed by the caller on the
// same stream.  prm: problem fields set by the caller, plan fields by this.
cudaError_t resident_launch(const ResidentPlan& pl, ResidentParams& prm, void* ws,
                            cudaStream_t stream);

}  // namespace drot

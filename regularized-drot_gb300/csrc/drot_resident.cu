// drot_resident.cu -- planning and launch of the resident solve kernel
// (drot_resident.cuh).
#include "drot_resident.cuh"

#include <algorithm>

#include "drot_gb300.h"

namespace drot {

typedef void (*ResidentFn)(const ResidentParams);

template <typename CT>
static ResidentFn resident_ct(int mode, int threads) {
  if (mode == MODE_GL)
    return threads == 256 ? drot_resident_kernel<MODE_GL, CT, 256>
                          : drot_resident_kernel<MODE_GL, CT, 512>;
  return threads == 256 ? drot_resident_kernel<MODE_QR, CT, 256>
                        : drot_resident_kernel<MODE_QR, CT, 512>;
}

static ResidentFn resident_fn(int mode, int ctype, int threads) {
  return ctype == DROT_C_BF16 ? resident_ct<__nv_bfloat16>(mode, threads)
                              : resident_ct<float>(mode, threads);
}

static size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// Estimated clocks per iteration of a tiling, fitted to measured ones (QR 96 x
// 80 to 4000 x 4000, GL 300 x 200 to 1500 x 1000; within 15 %).  A step (four
// columns a warp, GL eight) takes 920 clocks with two warps a scheduler and
// 1450 with four, which share its arithmetic and shared-memory pipes, and more
// where C (and X) come from L2; eight warps leave 800 clocks less of work
// repeated by every warp.  adds: additions to the exchange words per
// iteration, 64-bit ones in L2; parts: additions to one word.
constexpr double kStepL2 = 350.0, kStepL2X = 500.0;

static double tile_cost(bool gl, bool keep, int warps, int used, int cw, int grid, int items,
                        double adds, int parts) {
  const int steps = gl ? (cw + 7) / 8 : (cw + 3) / 4;
  const double step = gl ? (used <= 8 ? 2000.0 : used <= 12 ? 2300.0 : 3800.0)
                         : (warps == 8 ? 920.0 : 1450.0);
  double t = (warps == 8 ? 2200.0 : 3000.0) + steps * step +
             400.0 * ((items - 1) / (32 * (warps - 2)));
  if (grid > 1) {
    t += 1900.0 + 0.0145 * adds * std::max(1.0, parts / 24.0);
    if (!keep) t += gl ? 2200.0 : 1100.0;
  }
  return t;
}

bool resident_plan(int mode, int nr, int nc, int G, const int* bounds, int ctype, bool check_all,
                   int sms, int smem_optin, ResidentPlan& best) {
  const size_t csize = ctype == DROT_C_BF16 ? 2 : 4;
  const size_t budget = (size_t)std::max(smem_optin, 48 * 1024) - 2048;
  const bool gl = mode == MODE_GL;
  int hmax = 0;
  if (gl) {
    if (G > sms) return false;
    for (int k = 0; k < G; ++k) {
      if (bounds[k + 1] <= bounds[k]) return false;
      hmax = std::max(hmax, bounds[k + 1] - (bounds[k] & ~3));
    }
  }
  sms = std::min(sms, 255);  // a word's count has one byte
  double best_cost = 0.0;
  bool found = false;
  for (int wk = 0; wk < 2 * kResidentMaxWarps; ++wk) {
    const int warps = wk & 1 ? 16 : 8, WR = wk / 2 + 1, WC = warps / WR;
    const int rows = 128 * WR;
    if (WC < 1 || (gl ? hmax > rows : (WR & (WR - 1)) != 0)) continue;
    const int gr_min = gl ? G : (nr + rows - 1) / rows;
    if (gr_min > sms) continue;
    // QR: as few bands as cover the rows, or more of fewer rows each (a
    // squarer grid)
    const int gr_max = gl ? G : std::min(std::min(sms, (nr + 31) / 32), 4 * gr_min + 8);
    for (int GR = gr_min; GR <= gr_max; ++GR) {
      int band_h = 0, rt = hmax;
      if (!gl) {
        band_h = (((nr + GR - 1) / GR) + 3) & ~3;
        if (band_h > rows || (nr + band_h - 1) / band_h != GR) continue;
        rt = band_h;
      }
      rt = (rt + 3) & ~3;
      for (int GC = 1; GC <= std::min(sms / GR, nc); ++GC) {
        const int w = (nc + GC - 1) / GC, ct = (w + 3) & ~3, cw = (w + WC - 1) / WC;
        const int cwp = gl ? (cw + 7) & ~7 : (cw + 3) & ~3;
        if (cw > (gl ? 32 : 64) || rt + w > 4 * 32 * (warps - 2)) continue;
        // tested on every iteration, QR may stop on one without an objective
        // of its own: no running ahead
        for (int keep = check_all ? 0 : 1; keep >= 0; --keep) {
          auto smem_of = [&](int x, int c) {
            return resident_smem_bytes(32 * warps, x, c, WR, WC, rt, ct, csize, keep, gl);
          };
          int nsx = cwp, nsc = cwp;
          if (smem_of(nsx, nsc) > budget) {
            // QR: what does not fit stays in global memory (L2), C first
            if (gl || keep || warps < 16) continue;
            while (nsc > 0 && smem_of(nsx, nsc) > budget) nsc -= 4;
            while (nsx > 0 && smem_of(nsx, nsc) > budget) nsx -= 4;
            if (nsx <= 0) continue;
          }
          const size_t smem = smem_of(nsx, nsc);
          double cost = tile_cost(gl, keep, warps, WR * WC, cw, GR * GC, rt + w,
                                  (double)(rt + w) * GR * GC, std::max(GR, GC)) +
                        kStepL2 * ((cwp - nsc) / 4) + kStepL2X * ((cwp - nsx) / 4);
          // Bands below 400 rows stream shorter runs of a column: 3000 x 3000
          // in bands of 500 11.3 us, of 250 12.1 us; 4000 x 4000 22.8, 24.2.
          if (nsc < cwp && band_h < 400) cost *= 1.05;
          if (found && cost >= best_cost) continue;
          found = true;
          best_cost = cost;
          best.mode = mode; best.ctype = ctype; best.keep = keep;
          best.GR = GR; best.GC = GC; best.WR = WR; best.WC = WC;
          best.band_h = band_h; best.rt = rt; best.ct = ct; best.cw = cw; best.cwp = cwp;
          best.nsx = nsx; best.nsc = nsc; best.aligned = nsc < cwp;
          best.threads = 32 * warps; best.grid = GR * GC; best.smem = smem;
        }
      }
    }
  }
  if (!found) return false;
  const ResidentFn fn = resident_fn(mode, ctype, best.threads);
  int occ = 0;
  if (cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)best.smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)fn, best.threads,
                                                    best.smem) != cudaSuccess ||
      occ < 1) {
    cudaGetLastError();
    return false;
  }
  size_t off = 512;
  auto take = [&](size_t words) {
    const size_t at = off;
    off = up256(off + words * sizeof(unsigned long long));
    return at;
  };
  best.off_massx = take(64);
  best.off_resx = take(4 * (size_t)kPairCopies * best.grid);
  best.off_objx = take(2 * (size_t)best.grid);
  best.off_rowx = take(2 * (size_t)best.GR * best.rt);
  best.off_colx = take(2 * (size_t)best.GC * best.ct);
  best.total = off;
  return true;
}

cudaError_t resident_launch(const ResidentPlan& pl, ResidentParams& prm, void* ws,
                            cudaStream_t stream) {
  char* const w = (char*)ws;
  auto at = [&](size_t off) { return (unsigned long long*)(w + off); };
  prm.GR = pl.GR; prm.GC = pl.GC; prm.WR = pl.WR; prm.WC = pl.WC; prm.keep = pl.keep;
  prm.band_h = pl.band_h; prm.rt = pl.rt; prm.ct = pl.ct; prm.cw = pl.cw; prm.cwp = pl.cwp;
  prm.nsx = pl.nsx; prm.nsc = pl.nsc;
  prm.rowx = at(pl.off_rowx); prm.colx = at(pl.off_colx);
  prm.massx = at(pl.off_massx); prm.resx = at(pl.off_resx); prm.objx = at(pl.off_objx);
  const ResidentFn fn = resident_fn(pl.mode, pl.ctype, pl.threads);
  cudaError_t rc = cudaFuncSetAttribute((const void*)fn,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)pl.smem);
  if (rc != cudaSuccess) return rc;
  void* args[] = {(void*)&prm};
  return cudaLaunchCooperativeKernel((const void*)fn, dim3(pl.grid), dim3(pl.threads), args,
                                     pl.smem, stream);
}

}  // namespace drot

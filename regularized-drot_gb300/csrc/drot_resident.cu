// drot_resident.cu -- planning and launch of the resident solve kernel
// (drot_resident.cuh).
#include "drot_resident.cuh"

#include <algorithm>
#include <functional>
#include <map>
#include <queue>
#include <utility>

#include "drot_gb300.h"
#include "drot_launch.h"

namespace drot {

typedef void (*ResidentFn)(const ResidentParams, const ResidentBounds);

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

// Workspace of a tiling: the statistics and flags, then the exchange words.
static void resident_layout(ResidentPlan& pl) {
  size_t off = 512;
  auto take = [&](size_t words) {
    const size_t at = off;
    off = up256(off + words * sizeof(unsigned long long));
    return at;
  };
  pl.off_massx = take(64);
  pl.off_resx = take(4 * (size_t)kPairCopies * pl.grid);
  pl.off_objx = take(2 * (size_t)pl.grid);
  pl.off_rowx = take(2 * (size_t)pl.GR * pl.rt);
  pl.off_colx = take(2 * (size_t)pl.GC * pl.ct);
  pl.total = off;
}

size_t resident_most_bytes(int mode, int nr, int nc, int G, const int* bounds, int sms) {
  // QR bands and chunks share the rows and columns out in whole vectors
  ResidentPlan most;
  most.grid = sms;
  most.GR = most.GC = 1;
  most.rt = nr + 4 * sms;
  most.ct = nc + 4 * sms;
  if (mode == MODE_GL) {
    int h = 0;
    for (int k = 0; k < G; ++k) h = std::max(h, bounds[k + 1] - (bounds[k] & ~3));
    if (G > sms || h > 128 * kResidentMaxWarps) return 0;  // no tiling
    most.GR = G;
    most.rt = (h + 3) & ~3;
  }
  resident_layout(most);
  return most.total;
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
            return resident_smem_bytes(32 * warps, x, c, WR, WC, rt, ct, csize, keep, gl,
                                       false);
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
  resident_layout(best);
  const ResidentFn fn = resident_fn(mode, ctype, best.threads);
  int occ = 0;
  if (allow_shared_memory((const void*)fn) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)fn, best.threads,
                                                    best.smem) != cudaSuccess ||
      occ < 1) {
    cudaGetLastError();
    return false;
  }
  return true;
}

cudaError_t resident_launch(const ResidentPlan& pl, ResidentParams& prm,
                            const ResidentBounds& bounds, void* ws, cudaStream_t stream) {
  char* const w = (char*)ws;
  auto at = [&](size_t off) { return (unsigned long long*)(w + off); };
  prm.GR = pl.GR; prm.GC = pl.GC; prm.WR = pl.WR; prm.WC = pl.WC; prm.keep = pl.keep;
  prm.band_h = pl.band_h; prm.rt = pl.rt; prm.ct = pl.ct; prm.cw = pl.cw; prm.cwp = pl.cwp;
  prm.nsx = pl.nsx; prm.nsc = pl.nsc;
  prm.rowx = at(pl.off_rowx); prm.colx = at(pl.off_colx);
  prm.massx = at(pl.off_massx); prm.resx = at(pl.off_resx); prm.objx = at(pl.off_objx);
  const ResidentFn fn = resident_fn(pl.mode, pl.ctype, pl.threads);
  const cudaError_t rc = allow_shared_memory((const void*)fn);
  if (rc != cudaSuccess) return rc;
  void* args[] = {(void*)&prm, (void*)&bounds};
  return cudaLaunchCooperativeKernel((const void*)fn, dim3(pl.grid), dim3(pl.threads), args,
                                     pl.smem, stream);
}

// ---------------------------------------------------------------------------
// Batches
// ---------------------------------------------------------------------------

typedef void (*ResidentBatchFn)(const ResidentBatch);

static ResidentBatchFn resident_batch_fn(int mode, int ctype) {
  if (ctype == DROT_C_BF16)
    return mode == MODE_GL ? drot_resident_batch_kernel<MODE_GL, __nv_bfloat16>
                           : drot_resident_batch_kernel<MODE_QR, __nv_bfloat16>;
  return mode == MODE_GL ? drot_resident_batch_kernel<MODE_GL, float>
                         : drot_resident_batch_kernel<MODE_QR, float>;
}

// A tiling of one instance: n CTAs, about t clocks per iteration.
struct BatchTiling {
  int n;
  double t;
  ResidentTiling tiling;
};

// Estimated clocks per iteration of an 8-warp tile that shares its SM with
// another one, fitted to measured ones within 15 % (tiles of 128 to 1024 rows
// and 16 to 512 columns).  Terms as in tile_cost.
static double batch_tile_cost(bool gl, bool keep, int steps, int c_steps, int x_steps, int cols,
                              int grid, int items, int parts) {
  double t = gl ? 2600.0 + 3800.0 * steps + 1500.0 * c_steps + 700.0 * x_steps +
                      800.0 * ((items - 1) / 192)
                : 2600.0 + 1400.0 * steps + 350.0 * c_steps + 500.0 * x_steps +
                      400.0 * ((items - 1) / 192);
  if (grid > 1) {
    t += 2200.0 + 0.0145 * items * grid * std::max(1.0, parts / 24.0);
    if (!keep) t += gl ? 4400.0 : 1100.0;
  }
  // Past 48 columns a warp the tiles of all CTAs no longer fit L2 (32 QR
  // instances of 34 M elements: 20.1 ms with 47, 25.4 ms with 60).
  return cols > 48 ? 1.25 * t : t;
}

// The tilings of a problem that no other one beats in both CTAs and clocks, by
// rising n.
static std::vector<BatchTiling> batch_tilings(bool gl, int nr, int nc, const std::vector<int>* bounds,
                                              int max_n, size_t budget) {
  std::vector<BatchTiling> best;
  constexpr int warps = 8;
  int hmax = 0, G = 0;
  if (gl) {
    G = (int)bounds->size() - 1;
    for (int k = 0; k < G; ++k)
      hmax = std::max(hmax, (*bounds)[k + 1] - ((*bounds)[k] & ~3));
  }
  const int most_items = (gl ? 6 : 4) * 32 * (warps - 2), unit = gl ? 8 : 4;
  for (int WR = 1; WR <= warps; ++WR) {
    const int WC = warps / WR, rows = 128 * WR;
    if (gl ? hmax > rows : (WR & (WR - 1)) != 0) continue;
    const int gr_min = gl ? G : (nr + rows - 1) / rows;
    const int gr_max = gl ? G : std::min((nr + 31) / 32, 2 * gr_min);
    for (int GR = gr_min; GR <= std::min(gr_max, max_n); ++GR) {
      int band_h = 0, rt = hmax;
      if (!gl) {
        band_h = (((nr + GR - 1) / GR) + 3) & ~3;
        if (band_h > rows || (nr + band_h - 1) / band_h != GR) continue;
        rt = band_h;
      }
      rt = (rt + 3) & ~3;
      int GC_last = 0;
      for (int cwp = unit; cwp <= 64; cwp += unit) {
        const int GC = (nc + WC * cwp - 1) / (WC * cwp);
        if (GC == GC_last || GR * GC > max_n) continue;
        GC_last = GC;
        const int w = (nc + GC - 1) / GC, ct = (w + 3) & ~3, cw = (w + WC - 1) / WC;
        if (rt + w > most_items) continue;
        const int cwr = (cw + unit - 1) / unit * unit;
        for (int keep = 1; keep >= 0; --keep) {
          auto smem_of = [&](int x, int c) {
            return resident_smem_bytes(32 * warps, x, c, WR, WC, rt, ct, sizeof(float), keep, gl,
                                       true);
          };
          int nsx = cwr, nsc = cwr;
          while (nsc > 0 && smem_of(nsx, nsc) > budget) nsc -= unit;
          while (!keep && nsx > 0 && smem_of(nsx, nsc) > budget) nsx -= unit;
          if (nsx <= 0 || smem_of(nsx, nsc) > budget) continue;
          BatchTiling b;
          b.n = GR * GC;
          b.t = batch_tile_cost(gl, keep, cwr / unit, (cwr - nsc) / unit, (cwr - nsx) / unit, cwr,
                                b.n, rt + w, std::max(GR, GC));
          b.tiling = ResidentTiling{GR, GC, WR, WC, band_h, rt, ct, cw, cwr, nsx, nsc, keep};
          best.push_back(b);
        }
      }
    }
  }
  std::stable_sort(best.begin(), best.end(), [](const BatchTiling& a, const BatchTiling& b) {
    return a.n != b.n ? a.n < b.n : a.t < b.t;
  });
  std::vector<BatchTiling> out;
  for (const BatchTiling& b : best)
    if (out.empty() || b.t < out.back().t) out.push_back(b);
  return out;
}

void resident_batch_plan(int mode, const std::vector<ResidentInst>& inst,
                         const std::vector<std::vector<int>>& gl_bounds, int sms,
                         ResidentBatchPlan& pl) {
  const bool gl = mode == MODE_GL;
  const int n_inst = (int)inst.size();
  pl = ResidentBatchPlan();
  // Planning takes 0.6 ms for 32 instances of different shapes and 12 ms for
  // 512; more of them keep the streaming kernel busy.
  if (n_inst > 512) return;
  int dev = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) !=
          cudaSuccess) {
    cudaGetLastError();
    return;
  }
  // two CTAs per SM; 1 KB of each is reserved, 2 KB cover the static part
  const size_t budget = (size_t)std::max(per_sm / 2 - 3 * 1024, 16 * 1024);
  const int grid = 2 * sms, max_n = std::min(grid, 255);  // a word's count has one byte
  // The tilings of every shape
  std::vector<const std::vector<BatchTiling>*> of(n_inst);
  std::map<std::vector<int>, std::vector<BatchTiling>> shapes;
  for (int k = 0; k < n_inst; ++k) {
    std::vector<int> key = {inst[k].nr, inst[k].nc};
    if (gl) key.insert(key.end(), gl_bounds[k].begin(), gl_bounds[k].end());
    auto it = shapes.find(key);
    if (it == shapes.end())
      it = shapes.emplace(key, batch_tilings(gl, inst[k].nr, inst[k].nc,
                                             gl ? &gl_bounds[k] : nullptr, max_n, budget)).first;
    if (it->second.empty()) return;
    of[k] = &it->second;
  }
  // For a limit T on an instance's time, every instance takes its tiling of the
  // least n t below T (the fastest, if none is).  Which T is best shows when the
  // batch is played through with the kernel's own order.
  std::vector<std::pair<double, int>> order(n_inst);
  std::vector<const BatchTiling*> chosen(n_inst);
  auto choose = [&](double T) {
    for (int k = 0; k < n_inst; ++k) {
      chosen[k] = &of[k]->back();
      for (const BatchTiling& x : *of[k])
        if (x.t <= T && x.n * x.t < chosen[k]->n * chosen[k]->t) chosen[k] = &x;
      order[k] = {-chosen[k]->n * chosen[k]->t, k};
    }
    std::sort(order.begin(), order.end());
  };
  auto duration = [&]() {
    std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>,
                        std::greater<std::pair<double, int>>> running;  // end, CTAs
    std::vector<char> taken(n_inst, 0);
    int free = grid, head = 0, left = n_inst;
    double now = 0.0;
    while (left > 0 || !running.empty()) {
      for (int i = head; i < std::min(n_inst, head + kBatchWindow); ++i) {
        const BatchTiling* b = chosen[order[i].second];
        if (taken[i] || b->n > free) continue;
        taken[i] = 1;
        --left;
        free -= b->n;
        running.push({now + b->t, b->n});
        while (head < n_inst && taken[head]) ++head;
      }
      now = running.top().first;
      free += running.top().second;
      running.pop();
    }
    return now;
  };
  double t_lo = 1e30, t_hi = 0.0;
  for (auto& s : shapes) {
    t_lo = std::min(t_lo, s.second.back().t);
    t_hi = std::max(t_hi, s.second.front().t);
  }
  double best = 1e30, best_T = t_hi;
  for (double T = t_lo; T < t_hi * 1.1; T *= 1.03) {
    choose(T);
    const double d = duration();
    if (d < best) {
      best = d;
      best_T = T;
    }
  }
  choose(best_T);
  // Streaming or resident, from measured batches of 8 to 365 M elements (us per
  // iteration, streaming -> resident, where streaming the instances' X and C from
  // HBM is at its best): QR 296 M 501 -> 456, 365 M 586 -> 585, with BF16 C 365 M
  // 547 -> 564, 101 M 168 -> 161; GL 131 M in classes of 400 rows 377 -> 398, of
  // 200 rows 612 -> 385, 91 M 277 -> 257.  Below, resident is ahead by more: QR
  // 67 M 123 -> 86, 8.7 M 30 -> 14, GL 23 M 96 -> 67.  A GL class short of whole
  // 512-row steps idles lanes there.
  pl.us = 1.2 * best / 1900.0;
  for (int ctype : {DROT_C_F32, DROT_C_BF16}) {
    const bool bf16 = ctype == DROT_C_BF16;
    double us = gl ? 30.0 : 20.0;
    for (int k = 0; k < n_inst; ++k) {
      const double e = 1e-6 * inst[k].nr * inst[k].nc;
      if (!gl) {
        us += (bf16 ? 1.44 : 1.56) * e;
        continue;
      }
      double steps = 0.0;
      for (size_t g = 0; g + 1 < gl_bounds[k].size(); ++g)
        steps += (gl_bounds[k][g + 1] - (gl_bounds[k][g] & ~3) + 511) / 512;
      us += (bf16 ? 2.15 : 2.25) * e * (0.5 + 0.5 * 512.0 * steps / inst[k].nr);
    }
    pl.stream_us[bf16 ? 1 : 0] = us;
  }
  if (pl.us >= kLongSolve * std::max(pl.stream_us[0], pl.stream_us[1])) return;
  pl.grid = grid;
  auto take = [&](size_t words) {  // whole 256-byte units
    const size_t at = pl.words;
    pl.words += (words + 31) & ~(size_t)31;
    return (long long)at;
  };
  for (const auto& o : order) {
    const int k = o.second;
    ResidentInst I = inst[k];
    const ResidentTiling& g = chosen[k]->tiling;
    I.tiling = g;
    I.n = chosen[k]->n;
    I.tile0 = pl.tiles;
    pl.tiles += I.n;
    I.bounds_off = (int)pl.bounds.size();
    if (gl) pl.bounds.insert(pl.bounds.end(), gl_bounds[k].begin(), gl_bounds[k].end());
    I.mass_off = take(96);
    I.res_off = take(I.n > 1 ? 4 * (size_t)kPairCopies * I.n : 0);
    I.obj_off = take(I.n > 1 ? 2 * (size_t)I.n : 0);
    I.rowx_off = take(g.GC > 1 ? 2 * (size_t)g.GR * g.rt : 0);
    I.colx_off = take(g.GR > 1 ? 2 * (size_t)g.GC * g.ct : 0);
    pl.smem = std::max(pl.smem, resident_smem_bytes(256, g.nsx, g.nsc, g.WR, g.WC, g.rt, g.ct,
                                                    sizeof(float), g.keep != 0, gl, true));
    pl.inst.push_back(I);
  }
  pl.first_n = pl.inst[0].n;
  // The scheduler's state with the instances that start at once.
  for (const ResidentInst& I : pl.inst) pl.need.push_back(I.n);
  pl.state.assign(kSchedWords + grid + 2 * (size_t)n_inst + grid + pl.tiles, 0);
  int* const sched = pl.state.data();
  int* const mail = sched + kSchedWords;
  int* const taken = mail + grid;
  int* const free_list = taken + 2 * n_inst;
  int* const cta_of = free_list + grid;
  int used = 0;
  for (int i = 0; i < n_inst && used < grid; ++i) {
    const ResidentInst& I = pl.inst[i];
    if (used + I.n > grid) continue;
    for (int t = 0; t < I.n; ++t) {
      cta_of[I.tile0 + t] = used + t;
      mail[used + t] = (i + 1) << kMailTileBits | t;
    }
    taken[i] = 1;
    used += I.n;
  }
  for (int c = used; c < grid; ++c) free_list[c - used] = c;
  sched[kSchedFree] = grid - used;
  sched[kSchedLeft] = n_inst;
  for (int ctype : {DROT_C_F32, DROT_C_BF16}) {
    const void* fn = (const void*)resident_batch_fn(mode, ctype);
    int occ = 0;
    if (allow_shared_memory(fn) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 256, pl.smem) != cudaSuccess ||
        occ < 2) {
      cudaGetLastError();
      return;
    }
  }
  pl.ok = true;
}

cudaError_t resident_batch_launch(const ResidentBatchPlan& pl, int mode, int ctype,
                                  const ResidentBatch& b, cudaStream_t stream) {
  const void* fn = (const void*)resident_batch_fn(mode, ctype);
  const cudaError_t rc = allow_shared_memory(fn);
  if (rc != cudaSuccess) return rc;
  void* args[] = {(void*)&b};
  return cudaLaunchCooperativeKernel(fn, dim3(pl.grid), dim3(256), args, pl.smem, stream);
}

}  // namespace drot

// Kernel lookup and launch helpers shared by the plan.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.h"
#include "plan_kernels.cuh"
#include "repick_ff.cuh"
#include "search_inst.cuh"

namespace semb {

SearchEntry search_entry_cmp_plain(int w, int variant);
SearchEntry search_entry_cmp_fast(int w, int variant);
SearchEntry search_entry_crs_plain(int w, int variant);
SearchEntry search_entry_crs_fast(int w, int variant);

static SearchEntry lookup(int method, int form, int w, int v) {
  if (method == METHOD_CMP) return form == FORM_PLAIN ? search_entry_cmp_plain(w, v) : search_entry_cmp_fast(w, v);
  return form == FORM_PLAIN ? search_entry_crs_plain(w, v) : search_entry_crs_fast(w, v);
}

int search_variant(int method, int form, int w, int v, int* rc, int* minb, int* brun, int* nt, int* pipe, int* lay,
                   int* glob, int* z0) {
  if (v < 0 || v >= kMaxVariants) return 0;
  SearchEntry e = lookup(method, form, w, v);
  *rc = e.rc;
  *minb = e.minb;
  *brun = e.brun;
  *nt = e.nt;
  if (pipe) *pipe = e.pipe;
  if (lay) *lay = e.lay;
  if (glob) *glob = e.glob;
  if (z0) *z0 = e.z0;
  return e.fn != nullptr;
}

// Candidate slots of one (A, C) group's run of nb B values padded to a multiple of rc.
static int brun_slots(int nb, int rc) { return (std::max(nb, 1) + rc - 1) / rc * rc; }

// Launch shape of semb_plain_kernel and semb_ring_kernel for ncand candidates at rc per
// thread and at most max_warps warps per SM: warps per CTA and CTAs per SM (several where
// one needs few warps).  Returns its cost, time per aperture trace in candidates per lane:
// a pass of nw warps takes its schedulers ceil(nw / 4) warps' time each, and not less than
// `few` warps' (with fewer, the latency of a warp's own chain shows).
double plain_shape(int ncand, int rc, int max_warps, int* nwarps, int* ctas) {
  const double few = rc == 4 ? 4.0 : 2.5;
  double best = 1e300;
  for (int nw = max_warps; nw >= 4; --nw) {
    const int npass = (ncand + nw * rc - 1) / (nw * rc), k = std::min(4, max_warps / nw);
    const double cost = (double)npass * rc * std::max((double)((nw * k + 3) / 4), few) / k;
    if (cost < best) {
      best = cost;
      *nwarps = nw;
      *ctas = k;
    }
  }
  return best;
}

// Plain form, windows up to 5: 8 candidates per thread (variant 0) unless 4 (variant 1)
// use the warps better; where both come out even and 8 need one pass of a whole SM, 4 for
// the windows whose per-candidate chain is short.  Measured, variant 0 / 1 / the two-barrier
// kernel (ms): 256 candidates, w = 5: 8.66 / 9.21 / 11.44; 200, w = 3: 3.24 / 3.19 / 5.03;
// 101, w = 3: 1.86 / 1.74 / 2.37; 90, w = 5: 1.98 / 2.09 / 2.57; 64, w = 3: 1.96 / 2.19 /
// 2.42; 33, w = 1: 0.50 / 0.44 / 0.80; 125, w = 1, 234 tasks: 0.100 / 0.083 / 0.096, w = 3:
// 0.125 / 0.114 / 0.131, w = 5: 0.156 / 0.159 / 0.163.
static int plain_variant(int w, int ncand) {
  int nw, k4, k8;
  const double c4 = plain_shape(ncand, 4, 26, &nw, &k4), c8 = plain_shape(ncand, 8, 16, &nw, &k8);
  return c4 < (w <= 3 && k8 == 1 && ncand <= 8 * nw ? 1.03 : 0.97) * c8 ? 1 : 0;
}

// Batched CMP: the ring kernel (30, 31) or -1 for the two-barrier one.  `fold`: the aperture
// traces of the average trace-evaluation; `tasks_per_sm` of the plan.
//
// Up to w = 5 the two-barrier kernel evaluates 64 candidates per pass on two CTAs per SM.
// The ring kernel is ahead where its shape computes at most 0.85 of the padded candidates
// (20 to 40, 65 to 95, 129 to 160 of them, ...); where both compute the same, its planner,
// staging and merges show on small folds: from 110 traces it pays with several passes a
// chunk, from 150 with w = 1.  Measured, ring / two-barrier, folds of 30, 62 and 150: w = 5,
// 160 candidates 0.83, 0.82, 0.81; 80 0.86, 0.81, 0.80; 256 1.11, 1.03, 0.95 (uneven folds of
// 12 to 240 9.45 / 10.28 ms); 128 1.27, 1.12, 0.98; w = 3, 33 candidates 0.98, 0.88, 0.87; 64
// 1.01, 0.99, 1.00; w = 1, 128 1.27, 1.06, 0.86.
//
// From w = 7 on the two-barrier kernel's entries of 16 bytes per window sample and its few
// candidates per thread put it behind from 80 candidates on, unless those fill its warps on
// small folds (w = 7, 128 candidates, fold 20: 1.17; 40: 1.06; 90: 0.96) or, at w = 15, by
// its narrow passes (80 candidates 1.00).  Several ring CTAs to the SM need the tasks to
// fill them.  Measured: w = 7, 80 candidates 0.77; w = 11, 90 0.46 / 0.57 ms, 128 0.72, 200
// 0.70; w = 15, 101 0.66, 200 0.63, 256 0.88.
//
// Records whose last tile of 32 samples reaches more than 3% beyond the end: its items
// take the range-checked path, which costs 31 more than a third (w = 5, 34 candidates, 304
// samples: 31 1.20, 30 1.03, 80 candidates 1.09 and 0.98; 320 samples: 0.90 and 0.92).
static int ring_variant(int w, int ncand, int ns, double fold, double tasks_per_sm) {
  int nw = 0, k0 = 1, k1 = 1;
  if (((ns + 31) / 32 * 32 - ns) * 100 > 3 * ns) {
    if (w > 5 || (w > 1 && ncand > 24 && ncand <= 64)) return -1;
    return plain_shape(ncand, 8, 16, &nw, &k0) <= 0.85 * ((ncand + 63) / 64 * 16.0) ? 30 : -1;
  }
  if (w >= 7) {
    const double c4 = plain_shape(ncand, 4, 16, &nw, &k0), c6 = plain_shape(ncand, 6, 12, &nw, &k1);
    const int v = c6 <= 1.03 * c4 ? 31 : 30;
    if (ncand < (w >= 13 ? 96 : 80) || ((v == 31 ? k1 : k0) > 1 && tasks_per_sm < 3.0)) return -1;
    return w <= 9 && ncand % 32 == 0 && fold < 60.0 ? -1 : v;
  }
  const double c8 = plain_shape(ncand, 8, 16, &nw, &k0), c10 = plain_shape(ncand, 10, 12, &nw, &k1);
  const int v = c10 <= c8 ? 31 : 30;
  const double pad = (ncand + 63) / 64 * 16.0, c = std::min(c8, c10);
  if (c <= 0.85 * pad) return v;
  if (fold >= 110.0 && ncand > 128 && c8 <= pad) return 30;
  return w == 1 && fold >= 150.0 && c <= pad ? v : -1;
}

// Variant a plan starts with (before any autotuning), the fastest measured on GB300
// for the benchmark workloads of each window: for CRS the pipelined B-run kernel
// (packed value/difference staging with a two-way trace unroll and the central traces'
// sums shared over A and B for w = 3, packed pairs otherwise); for CMP the ring kernel
// where ring_variant() says (fold > 0), else the two-barrier kernel with packed pairs (w =
// 3) or packed pairs formed by scalar FMAs (w = 5); variant 0 elsewhere.  For CRS with w = 3
// the B-run length follows the grid's nb: runs of 7 (variant 30, 512 threads) unless nb
// pads less to a multiple of 8 (variant 33, 384 threads; nb = 31 takes 32 slots per (A, C)
// instead of 35; per slot the two run at the same speed).  fallback_variant() is the one to
// use where the default does not fit the plan (a grid whose passes span more C values than
// the central-trace sharing takes).
int default_variant(int method, int form, int w, int nb, int ncand, int ns, double fold, double tasks_per_sm) {
  if (form != FORM_FAST) return w <= 5 ? plain_variant(w, ncand) : 0;
  if (method == METHOD_CMP && fold > 0.0) {
    const int v = ring_variant(w, ncand, ns, fold, tasks_per_sm);
    if (v >= 0) return v;
  }
  if (method == METHOD_CRS && w == 3) return brun_slots(nb, 8) < brun_slots(nb, 7) ? 33 : 30;
  if (method == METHOD_CRS && w <= 5) return 14;
  if (method == METHOD_CMP && w == 3) return 8;
  if (method == METHOD_CMP && w == 5) return 21;
  return 0;
}

int fallback_variant(int method, int form, int w, int nb) {
  if (form != FORM_FAST) return w <= 5 ? 2 : 0;
  if (form == FORM_FAST && method == METHOD_CRS && w == 3) return brun_slots(nb, 8) < brun_slots(nb, 7) ? 32 : 13;
  return 0;
}

int search_occupancy(int method, int form, int w, int v, int nwarps, size_t smem, int* ctas_per_sm) {
  SearchEntry e = lookup(method, form, w, v);
  if (!e.fn) return fail(SEMB_E_WINDOW, "no search kernel for w = %d", w);
  // the most any plan takes: the limit belongs to the kernel, and live plans of other sizes
  // (a ring kernel's depends on the candidate count) launch it too
  SEMB_CUDA(cudaFuncSetAttribute(e.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem));
  SEMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, e.fn, nwarps * 32, smem));
  return SEMB_OK;
}

int launch_search(int method, int form, int w, int v, const KParams& P, int nwarps, int grid, size_t smem,
                  cudaStream_t st) {
  SearchEntry e = lookup(method, form, w, v);
  if (!e.fn) return fail(SEMB_E_WINDOW, "no search kernel for w = %d", w);
  void* args[] = {const_cast<KParams*>(&P)};
  SEMB_CUDA(cudaLaunchKernel(e.fn, dim3(grid), dim3(nwarps * 32), args, smem, st));
  return SEMB_OK;
}

int launch_stt00(int w, int cdp0, int cdp1, const KParams& P, float a, float b, float c, float* out, cudaStream_t st) {
  const int grid = (cdp1 - cdp0 + 127) / 128;
  if (grid <= 0) return SEMB_OK;
  switch (w) {
    case 1: k_crs_stt00<1><<<grid, 128, 0, st>>>(cdp0, cdp1, P, a, b, c, out); break;
    case 3: k_crs_stt00<3><<<grid, 128, 0, st>>>(cdp0, cdp1, P, a, b, c, out); break;
    case 5: k_crs_stt00<5><<<grid, 128, 0, st>>>(cdp0, cdp1, P, a, b, c, out); break;
    default: return fail(SEMB_E_WINDOW, "no CRS kernel for w = %d", w);
  }
  SEMB_CUDA(cudaGetLastError());
  return SEMB_OK;
}

// Items per warp: 32, so that one warp screens 32 consecutive items with one load each, but
// fewer where that would leave the GPU's warps without work, as the near ties of a warp's
// items run one after the other: 64 warps' worth of items per SM for CRS, most of whose items
// are near ties (24 CDPs x 601 samples, w = 5: 3.2 ms at 32 per warp in FP64; 0.26 so, in
// pairs of FP32 numbers).  For CMP 1% are, and the screening of the others counts up to w = 5
// (100 x 1000, w = 5: 44 us at 8 warps' worth, 54 at 32); a wider window's ties are the longer
// ones (75 x 751, w = 11: 147 us at 8, 114 at 16, 109 at 32; 100 x 1000, w = 15: 183, 183, 136).
int launch_repick(int w, RepickParams R, int sms, cudaStream_t st) {
  const int64_t items = R.item_end - R.item0;
  if (items <= 0) return SEMB_OK;
  R.per_warp = 32;
  while (R.per_warp > 1 && items < (int64_t)sms * (R.method == METHOD_CRS ? 64 : w <= 5 ? 8 : 32) * R.per_warp) R.per_warp /= 2;
  const int grid = (int)((items + 8 * R.per_warp - 1) / (8 * R.per_warp));   // 8 warps per CTA
  switch (w) {
    case 1: k_repick<1><<<grid, 256, 0, st>>>(R); break;
    case 3: k_repick<3><<<grid, 256, 0, st>>>(R); break;
    case 5: k_repick<5><<<grid, 256, 0, st>>>(R); break;
    case 7: k_repick<7><<<grid, 256, 0, st>>>(R); break;
    case 9: k_repick<9><<<grid, 256, 0, st>>>(R); break;
    case 11: k_repick<11><<<grid, 256, 0, st>>>(R); break;
    case 13: k_repick<13><<<grid, 256, 0, st>>>(R); break;
    case 15: k_repick<15><<<grid, 256, 0, st>>>(R); break;
    default: return fail(SEMB_E_WINDOW, "no re-pick kernel for w = %d", w);
  }
  SEMB_CUDA(cudaGetLastError());
  return SEMB_OK;
}

}  // namespace semb

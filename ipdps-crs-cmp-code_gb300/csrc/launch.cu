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

// Launch shape of semb_plain_kernel and semb_ring_kernel for ncand candidates at rc per thread and at most
// max_warps warps per SM: warps per CTA and CTAs per SM (several where one needs few
// warps).  Returns its cost, time per aperture trace in candidates per lane: a pass of nw
// warps takes its schedulers ceil(nw / 4) warps' time each, and not less than `few` warps'
// (with fewer, the latency of a warp's own chain shows).
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
// use the warps better.  Measured, variant 0 / 1 / the two-barrier kernel (ms): 256
// candidates, w = 5: 8.66 / 9.21 / 11.44; 200, w = 3: 3.24 / 3.19 / 5.03; 101, w = 3: 1.86 /
// 1.74 / 2.37; 90, w = 5: 1.98 / 2.09 / 2.57; 64, w = 3: 1.96 / 2.19 / 2.42; 33, w = 1: 0.50 /
// 0.44 / 0.80.
static int plain_variant(int ncand) {
  int nw, k;
  return plain_shape(ncand, 4, 26, &nw, &k) < 0.97 * plain_shape(ncand, 8, 16, &nw, &k) ? 1 : 0;
}

// Batched CMP: the ring kernel (30, 31) or -1 for the two-barrier one, which runs two CTAs
// per SM whatever the candidate count.  `fold`: the aperture traces of the average
// trace-evaluation.  Where one ring CTA has to fill an SM its planner, merges and staging
// show on small folds: it pays from about 60 traces (150 for w = 3), and always where
// several CTAs share the SM.  Measured, ring / two-barrier (ms): w = 5, 256 candidates, fold
// 12 to 240 (mean 126) 9.34 / 10.29, fold 60 3.41 / 3.46, fold 12 1.20 / 1.01; w = 3, 101
// candidates, fold 200 1.93 / 2.05, fold 60 1.38 / 1.36; 40 candidates, fold 60 0.58 / 0.68,
// fold 12 0.33 / 0.38; w = 11, 90 candidates, fold 37 0.46 / 0.57; w = 15, 200 candidates 1.21
// / 1.95; w = 7, 64 candidates 0.32 / 0.27.
static int ring_variant(int w, int ncand, double fold) {
  int nw = 0, k8 = 1, k10 = 1;
  if (w >= 7) return ncand >= 80 && fold >= 30.0 ? 31 : -1;
  const double c8 = plain_shape(ncand, 8, 16, &nw, &k8), c10 = plain_shape(ncand, 10, 12, &nw, &k10);
  const int v = c10 < c8 ? 31 : 30;
  if ((v == 31 ? k10 : k8) >= 2) return v;
  return fold >= (w == 3 ? 150.0 : 60.0) ? v : -1;
}

// Variant a plan starts with (before any autotuning), the fastest measured on GB300
// for the benchmark workloads of each window: for CRS the pipelined B-run kernel
// (packed value/difference staging with a two-way trace unroll and the central traces'
// sums shared over A and B for w = 3, packed pairs otherwise); for CMP the ring kernel
// where ring_variant() says (fold > 0), else the two-barrier kernel with packed pairs (w =
// 3) or packed pairs formed by scalar FMAs (w = 5); variant 0 elsewhere.  For CRS with w = 3 the B-run length follows the
// grid's nb: runs of 7 (variant 30, 512 threads) unless nb pads less to a multiple of
// 8 (variant 33, 384 threads; nb = 31 takes 32 slots per (A, C) instead of 35; per
// slot the two run at the same speed).  fallback_variant() is the one to use where the
// default does not fit the plan (a grid whose passes span more C values than the
// central-trace sharing takes).
int default_variant(int method, int form, int w, int nb, int ncand, double fold) {
  if (form != FORM_FAST) return w <= 5 ? plain_variant(ncand) : 0;
  if (method == METHOD_CMP && fold > 0.0) {
    const int v = ring_variant(w, ncand, fold);
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
  SEMB_CUDA(cudaFuncSetAttribute(e.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
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
// are near ties (24 CDPs x 601 samples, w = 5: 3.2 ms at 32 per warp in FP64; 0.23 so, in
// pairs of FP32 numbers), 8 for CMP, where 1% are and the screening of the others counts (75 x
// 751, w = 11: 2% of the whole pass).
int launch_repick(int w, RepickParams R, int sms, cudaStream_t st) {
  const int64_t items = R.item_end - R.item0;
  if (items <= 0) return SEMB_OK;
  R.per_warp = 32;
  while (R.per_warp > 1 && items < (int64_t)sms * (R.method == METHOD_CRS ? 64 : 8) * R.per_warp) R.per_warp /= 2;
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

// Instantiations and launchers of the CRS filter and refine kernels.
#include <cuda_runtime.h>

#include "common.h"
#include "refine_kernel.cuh"

namespace semb {

namespace {

struct FilterShape {
  int rc, nt;   // slots per run, threads per CTA
};
// Long runs and the threads that their per-item sums (w + 1 floats per slot) leave registers
// for.  The fewest runs per (A, C) win (filter_kernel.cuh has both sides measured); among
// those the shortest slots, which cost less per crossing.
constexpr FilterShape kShapes3[] = {{12, 384}, {16, 384}, {22, 384}, {32, 256}};   // w = 1, 3
constexpr FilterShape kShapes5[] = {{8, 384}, {14, 256}, {22, 256}};               // w = 5

int shape_count(int w) { return w == 5 ? (int)(sizeof(kShapes5) / sizeof(kShapes5[0])) : (int)(sizeof(kShapes3) / sizeof(kShapes3[0])); }

template <int W, bool F32, int KT, int S>
const void* shape_fn(int s) {
  constexpr int n = W == 5 ? (int)(sizeof(kShapes5) / sizeof(kShapes5[0])) : (int)(sizeof(kShapes3) / sizeof(kShapes3[0]));
  if constexpr (S < n) {
    constexpr FilterShape f = W == 5 ? kShapes5[S < n && W == 5 ? S : 0] : kShapes3[S];
    if (s == S) return (const void*)semb_filter_kernel<W, F32, KT, f.rc, f.nt>;
    return shape_fn<W, F32, KT, S + 1>(s);
  } else {
    return nullptr;
  }
}

const void* filter_fn(int form, int w, int storage, int s) {
  if (form == FORM_PLAIN) {
    switch (w) {
      case 1: return shape_fn<1, true, 1, 0>(s);
      case 3: return shape_fn<3, true, 1, 0>(s);
      case 5: return shape_fn<5, true, 1, 0>(s);
      default: return nullptr;
    }
  }
  const bool f32 = storage == STORE_F32;
  switch (w) {
    case 3: return f32 ? shape_fn<3, true, kTopK, 0>(s) : shape_fn<3, false, kTopK, 0>(s);
    case 5: return f32 ? shape_fn<5, true, kTopK, 0>(s) : shape_fn<5, false, kTopK, 0>(s);
    default: return nullptr;
  }
}

}  // namespace

// The filter shape for B axes of nb values: its slot in the table, slots per run, threads.
// The fewest runs per (A, C), then the shortest slots that hold them.
int filter_shape(int w, int nb, int* rc, int* nt) {
  int best = 0, best_runs = 1 << 30;
  for (int s = 0; s < shape_count(w); ++s) {
    const FilterShape f = w == 5 ? kShapes5[s] : kShapes3[s];
    const int runs = (nb + f.rc - 1) / f.rc;
    if (runs < best_runs) {
      best_runs = runs;
      best = s;
      *rc = f.rc;
      *nt = f.nt;
    }
  }
  return best;
}

// Shared memory of the filter kernel for a staging capacity of cap samples.
size_t filter_smem(int form, int storage, int nt, int cap) {
  return filter_layout(cap, form == FORM_PLAIN || storage == STORE_F32, form == FORM_PLAIN ? 1 : kTopK, nt).total;
}

// Whether the direct configuration (window, layout) has a filter and refine pair.  Not with
// the global-memory path: a window longer than its stage comes from the FP32 store and ends
// no chunk, and the refine knows neither.
bool filter_exists(int form, int w, int brun, int pipe, int lay, int glob) {
  if (form == FORM_PLAIN) return w == 1 || w == 3 || w == 5;
  return pipe && brun && !glob && ((w == 3 && (lay == LAY_PD || lay == LAY_P2)) || (w == 5 && lay == LAY_P2));
}

// Once per plan configuration, before its launches (which may be captured).
int filter_prepare(int form, int w, int storage, int shape) {
  const void* fn = filter_fn(form, w, storage, shape);
  if (!fn) return fail(SEMB_E_WINDOW, "no filter kernel for w = %d", w);
  SEMB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem));
  return SEMB_OK;
}

int launch_filter(int form, int w, int storage, int shape, const FilterParams& F, int nwarps, int grid, size_t smem,
                  cudaStream_t st) {
  const void* fn = filter_fn(form, w, storage, shape);
  if (!fn) return fail(SEMB_E_WINDOW, "no filter kernel for w = %d", w);
  void* args[] = {const_cast<FilterParams*>(&F)};
  SEMB_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(nwarps * 32), args, smem, st));
  return SEMB_OK;
}

int launch_refine(int form, int w, int lay, const RefineParams& R, cudaStream_t st) {
  const int64_t units = (int64_t)R.ntasks * (kTB * kRefineLanes / 32);   // warps
  const int grid = (int)((units + 7) / 8);
  if (grid <= 0) return SEMB_OK;
  if (form == FORM_PLAIN) {
    switch (w) {
      case 1: k_refine_plain<1><<<grid, 256, 0, st>>>(R); break;
      case 3: k_refine_plain<3><<<grid, 256, 0, st>>>(R); break;
      case 5: k_refine_plain<5><<<grid, 256, 0, st>>>(R); break;
      default: return fail(SEMB_E_WINDOW, "no refine kernel for w = %d", w);
    }
  } else if (w == 3 && lay == LAY_PD) {
    k_refine_fast<3, LAY_PD><<<grid, 256, 0, st>>>(R);
  } else if (w == 3 && lay == LAY_P2) {
    k_refine_fast<3, LAY_P2><<<grid, 256, 0, st>>>(R);
  } else if (w == 5 && lay == LAY_P2) {
    k_refine_fast<5, LAY_P2><<<grid, 256, 0, st>>>(R);
  } else {
    return fail(SEMB_E_WINDOW, "no refine kernel for w = %d, layout %d", w, lay);
  }
  SEMB_CUDA(cudaGetLastError());
  return SEMB_OK;
}

}  // namespace semb

// Instantiations and launchers of the CRS filter and refine kernels.
#include <cuda_runtime.h>

#include "common.h"
#include "refine_kernel.cuh"

namespace semb {

namespace {

const void* filter_fn(int form, int w, int storage) {
  if (form == FORM_PLAIN) {
    switch (w) {
      case 1: return (const void*)semb_filter_kernel<1, true, 1>;
      case 3: return (const void*)semb_filter_kernel<3, true, 1>;
      case 5: return (const void*)semb_filter_kernel<5, true, 1>;
      default: return nullptr;
    }
  }
  const bool f32 = storage == STORE_F32;
  switch (w) {
    case 3:
      return f32 ? (const void*)semb_filter_kernel<3, true, kTopK> : (const void*)semb_filter_kernel<3, false, kTopK>;
    case 5:
      return f32 ? (const void*)semb_filter_kernel<5, true, kTopK> : (const void*)semb_filter_kernel<5, false, kTopK>;
    default: return nullptr;
  }
}

}  // namespace

// Shared memory of the filter kernel for a staging capacity of cap samples.
size_t filter_smem(int form, int storage, int cap) {
  return filter_layout(cap, form == FORM_PLAIN || storage == STORE_F32, form == FORM_PLAIN ? 1 : kTopK).total;
}

// Whether the direct configuration (window, layout) has a filter and refine pair.
bool filter_exists(int form, int w, int brun, int pipe, int lay) {
  if (form == FORM_PLAIN) return w == 1 || w == 3 || w == 5;
  return pipe && brun && ((w == 3 && (lay == LAY_PD || lay == LAY_P2)) || (w == 5 && lay == LAY_P2));
}

// Once per plan configuration, before its launches (which may be captured).
int filter_prepare(int form, int w, int storage, size_t smem) {
  const void* fn = filter_fn(form, w, storage);
  if (!fn) return fail(SEMB_E_WINDOW, "no filter kernel for w = %d", w);
  SEMB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return SEMB_OK;
}

int launch_filter(int form, int w, int storage, const FilterParams& F, int nwarps, int grid, size_t smem,
                  cudaStream_t st) {
  const void* fn = filter_fn(form, w, storage);
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

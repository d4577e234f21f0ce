// dispatch.cu -- choice of gridding kernel for one batch.
//
// Automatic: the stream kernel (grid_stream.cu), one visibility per group of
// warps, takes the batches its plan says it is the faster for; the tiled
// kernel (grid_tiled.cu) those with large multi-plane CF slices, and every
// batch when its plan was set by hand or it is selected; the per-visibility
// kernels (grid_direct.cu) what fits neither, or every batch when selected
// with hpgb_set_gridding_kernel.

#include "gridder.cuh"

namespace hpgb {

Status grid_batch(hpgb_gridder* g, const void* d_vis, size_t n,
                  unsigned flags) {
  bool streamed = false;
  HPGB_TRY(grid_stream(g, const_cast<void*>(d_vis), n, flags, &streamed));
  if (streamed) return Status::ok();
  if (n > 0) g->last_streamed = false;
  if (g->kernel_kind != HPGB_KERNEL_DIRECT) {
    bool used = false;
    HPGB_TRY(grid_tiled(g, const_cast<void*>(d_vis), n, flags, &used));
    if (used) {
      if (n > 0) g->last_kernel = HPGB_KERNEL_TILED;
      return Status::ok();
    }
    if (g->kernel_kind == HPGB_KERNEL_TILED)
      return Status::err(HPGB_ERROR_OTHER,
                         "the tiled kernel cannot take this CF or grid");
  }
  if (n > 0) g->last_kernel = HPGB_KERNEL_DIRECT;
  return grid_direct(g, d_vis, n, flags);
}

}  // namespace hpgb

// stream_launch.cuh -- the launcher of stream_kernel.cuh for one arithmetic
// form and polarization count; the stream_<form>_<n>.cu files instantiate it
// (separate files only so that they compile side by side).
#pragma once

#include "grid_stream.cuh"

namespace hpgb {
namespace stream {

template <int N, bool DIAG, int FORM, int W, bool RING, int PASS>
Status launch_pass(hpgb_gridder* g, const StreamPlan& pl,
                      const StreamParams& p) {
  auto kern = stream_kernel<N, DIAG, FORM, W, RING, PASS>;
  HPGB_CUDA_TRY(allow_dynamic_smem(kern));
  // (gridding launches only, as the tiled kernel's)
  const bool profile = FORM != kLinear && g->profile;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (profile) {
    HPGB_CUDA_TRY(cudaEventCreate(&ev[0]));
    HPGB_CUDA_TRY(cudaEventCreate(&ev[1]));
    HPGB_CUDA_TRY(cudaEventRecord(ev[0], g->stream));
  }
  kern<<<unsigned(pl.ctas), 32 * warps_of(RING, W), size_t(pl.smem),
         g->stream>>>(p);
  HPGB_CUDA_TRY(cudaGetLastError());
  ++g->launches;
  if (profile) {
    HPGB_CUDA_TRY(cudaEventRecord(ev[1], g->stream));
    g->prof_events.emplace_back(ev[0], ev[1]);
  }
  return Status::ok();
}

template <int N, bool DIAG, int FORM, int W, bool RING>
Status launch_variant(hpgb_gridder* g, const StreamPlan& pl,
                      const StreamParams& p) {
  if constexpr (DIAG) {
    // (degridding alone, the compiler spreads two polarizations' loads so that
    // they take longer than in the kernel with both passes: 2.8 against 2.4
    // ms for supports 8 to 64, 500k visibilities)
    if (!p.do_grid)
      return launch_pass<N, DIAG, FORM, W, RING, N == 1 ? 1 : 0>(g, pl, p);
    if constexpr (FORM != kLinear)
      if (p.do_degrid && p.has_model)
        return launch_pass<N, DIAG, FORM, W, RING, 3>(g, pl, p);
    return launch_pass<N, DIAG, FORM, W, RING, 2>(g, pl, p);
  } else {
    return launch_pass<N, DIAG, FORM, W, RING, 0>(g, pl, p);
  }
}

// the variants the plan picks from (make_stream_plan)
template <int N, bool DIAG, int FORM>
Status launch_variants(hpgb_gridder* g, const StreamPlan& pl,
                       const StreamParams& p) {
  if constexpr (DIAG) {
    if (!pl.ring) {
      if (pl.warps == 4) return launch_variant<N, true, FORM, 4, false>(g, pl, p);
      if (pl.warps == 2) return launch_variant<N, true, FORM, 2, false>(g, pl, p);
      if (pl.warps == 1) return launch_variant<N, true, FORM, 1, false>(g, pl, p);
    }
  } else if (pl.ring) {
    if (pl.warps == 7) return launch_variant<N, false, FORM, 7, true>(g, pl, p);
    if (pl.warps == 2) return launch_variant<N, false, FORM, 2, true>(g, pl, p);
  } else {
    // (slices that only the per-visibility kernels would take: FP64)
    if constexpr (FORM == kFP64)
      if (pl.warps == 16) return launch_variant<N, false, FORM, 16, false>(g, pl, p);
    if (pl.warps == 1) return launch_variant<N, false, FORM, 1, false>(g, pl, p);
  }
  return Status::err(HPGB_ERROR_OTHER, "stream kernel variant missing");
}

template <int FORM, int N>
Status launch_stream_n(hpgb_gridder* g, const StreamPlan& pl,
                       const StreamParams& p) {
  if (pl.diag) return launch_variants<N, true, FORM>(g, pl, p);
  if constexpr (N > 1) return launch_variants<N, false, FORM>(g, pl, p);
  return Status::err(HPGB_ERROR_OTHER, "stream kernel variant missing");
}

}  // namespace stream
}  // namespace hpgb

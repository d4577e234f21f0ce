// grid_stream.cuh -- plan and launch of the stream kernel
// (stream_kernel.cuh), shared by grid_stream.cu, grid_batch.cu and adjoint.cu.
#pragma once

#include "stream_kernel.cuh"

namespace hpgb {
namespace stream {

struct StreamPlan {
  bool ok = false;
  bool diag = false;   // one active element per row, a row per polarization
  bool ring = false;   // CF slices through the shared-memory ring
  int warps = 0;       // per group
  int ctas = 0, smem = 0;
  StreamParams p{};
};

// what the CFs of a launch look like (of one gridder, or of all of a batch)
struct CFShape {
  int max_plane_bytes = 0;  // largest plane
  int max_taps = 0;         // taps_x + taps_y, largest
  int max_side = 0;         // widest footprint
  double mean_plane_bytes = 0;  // over the groups
  size_t table_bytes = 0;
  void add(const hpgb_gridder* g);
};

// The plan of a launch over nvis visibilities with g's polarizations and
// Mueller tables.  dset, gset: the degridding and gridding index tables for
// w <= 0 and w > 0.  tiles_fp32: the tiled kernel would take FP32 tiles;
// tiled_takes: slices beyond the ring are for another kernel.  Not ok where
// another kernel is the faster one, or the only one.
StreamPlan make_stream_plan(const hpgb_gridder* g, const CFShape& cf,
                            bool degrid, bool grid, bool has_model,
                            const int (*const dset[2])[4],
                            const int (*const gset[2])[4], size_t nvis,
                            bool tiles_fp32, bool tiled_takes);

// whether a batch's visibilities are put into tile order
bool stream_sorted(const hpgb_gridder* g, size_t n, bool has_model);

template <int FORM, int N>
Status launch_stream_n(hpgb_gridder* g, const StreamPlan& pl,
                       const StreamParams& p);

// form: Form
Status launch_stream(hpgb_gridder* g, int form, const StreamPlan& pl,
                     const StreamParams& p);

}  // namespace stream
}  // namespace hpgb

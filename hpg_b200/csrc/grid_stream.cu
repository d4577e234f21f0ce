// grid_stream.cu -- plan of the stream kernel (stream_kernel.cuh) and its
// launches for one gridder: gridding, degridding and both, and the linear
// operators.

#include <algorithm>
#include <cmath>
#include <cstring>

#include "grid_stream.cuh"
#include "tiled_kernel.cuh"

namespace hpgb {
namespace stream {

void CFShape::add(const hpgb_gridder* g) {
  double sum = 0.0;
  for (const CFGroup& G : g->cf.groups) {
    max_plane_bytes = std::max(max_plane_bytes, G.plane_stride * 8);
    max_taps = std::max(max_taps, G.taps_x + G.taps_y);
    max_side = std::max(max_side, std::max(G.taps_x, G.taps_y));
    sum += G.plane_stride * 8.0;
  }
  if (!g->cf.groups.empty())
    mean_plane_bytes =
        std::max(mean_plane_bytes, sum / double(g->cf.groups.size()));
  table_bytes += g->cf.data.bytes;
}

// The batch goes into tile order when its footprints cover the grid (and
// model) several times over and those do not stay in L2 anyway: the sort's
// ~10 launches and descriptor gathers cost 60-100 us, unsorted footprints in
// a grid larger than L2 a DRAM read and write of every sector they touch.
bool stream_sorted(const hpgb_gridder* g, size_t n, bool has_model) {
  const double grid = 16.0 * double(g->grid_elems()) * (has_model ? 2.0 : 1.0);
  double cells = 0.0;
  for (const CFGroup& G : g->cf.groups) cells += double(G.taps_x) * G.taps_y;
  cells /= std::max<size_t>(g->cf.groups.size(), 1);
  const double touched =
      double(n) * cells * double(g->grid_size[2]) * 16.0;
  return grid > 64e6 && touched > 2.0 * grid;
}

StreamPlan make_stream_plan(const hpgb_gridder* g, const CFShape& cf,
                            bool degrid, bool grid, bool has_model,
                            const int (*const dset[2])[4],
                            const int (*const gset[2])[4], size_t nvis,
                            bool tiles_fp32, bool tiled_takes) {
  StreamPlan pl;
  StreamParams& p = pl.p;
  std::memset(&p, 0, sizeof(p));
  const int nrow = int(g->grid_size[2]), n = int(g->npol);
  // (the cell loops' row arithmetic holds for supports below 128)
  if (nrow < 1 || nrow > 4 || g->cf.groups.empty() || cf.max_side > 127)
    return pl;
  p.nrow = nrow;
  p.do_degrid = degrid;
  p.do_grid = grid;
  p.has_model = has_model;
  const bool use_d = degrid && has_model, use_g = grid;
  // one active element per row, the same for both signs of w, and a row per
  // polarization
  pl.diag = nrow == n;
  for (int r = 0; r < nrow && pl.diag; ++r) {
    int act[4] = {0, 0, 0, 0}, cnt = 0;
    for (int v = 0; v < n; ++v) {
      int on = 0, all = 0;
      for (int w = 0; w < 2; ++w) {
        if (use_d) on += dset[w][r][v] >= 0, ++all;
        if (use_g) on += gset[w][r][v] >= 0, ++all;
      }
      if (on != 0 && on != all) pl.diag = false;
      act[v] = on != 0;
      cnt += act[v];
      if (act[v]) p.vact[r] = v;
    }
    pl.diag = pl.diag && cnt == 1;
  }
  if (n == 1 && !pl.diag) return pl;
  // planes used, and their places: in a ring slot, or in the slice
  bool need[64] = {false};
  for (int r = 0; r < nrow; ++r)
    for (int v = 0; v < n; ++v)
      for (int w = 0; w < 2; ++w)
        for (int set = 0; set < 2; ++set) {
          if (!(set ? use_g : use_d)) continue;
          const int m = (set ? gset : dset)[w][r][v];
          if (m >= 64) return pl;
          if (m >= 0) need[m] = true;
        }
  int pos[64], np = 0, nr = 0;
  bool runs_fit = true;
  for (int m = 0; m < 64; ++m) {
    pos[m] = -1;
    if (!need[m]) continue;
    pos[m] = np;
    if (m > 0 && need[m - 1]) {
      if (runs_fit) p.run_len[nr - 1]++;
    } else if (nr == kMaxRuns) {
      runs_fit = false;
    } else {
      p.run_plane[nr] = m;
      p.run_len[nr] = 1;
      p.run_dst[nr] = np;
      ++nr;
    }
    ++np;
  }
  p.nplanes = np;
  p.nruns = nr;
  // shared memory: partial sums and screen tables per group, then the ring
  const int kBudget = 227 * 1024;
  const int part = (np * cf.max_plane_bytes + 127) / 128 * 128;
  const double mean = np * cf.mean_plane_bytes;
  p.tab_taps = cf.max_taps;
  auto layout = [&](int warps, bool ring) {
    const int groups =
        (ring ? kWarps - kProducers : warps_of(false, warps)) / warps;
    p.off_part = ring ? Fixed::kEnd : 0;
    p.off_offs = (p.off_part + groups * warps * 2 * n * 8 + 15) / 16 * 16;
    p.off_tab = p.off_offs + kWarps * 32 * 4;
    p.off_ring = (p.off_tab + groups * p.tab_taps * 16 + 127) / 128 * 128;
    return p.off_ring;
  };
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
  const double cells = cf.mean_plane_bytes / 8.0;
  if (pl.diag) {
    // One plane per row: read from global memory (a bulk copy each, ~430
    // cycles per SM whatever its size, bounds the kernel: supports 8 to 32,
    // one polarization, 1M visibilities degridded 1.6 against 3.7 ms), a
    // warp per visibility, two when footprints are wide (2 polarizations,
    // supports 8 to 64, 500k visibilities, both passes: 8.4 against 8.8 ms;
    // degridding 2.8 against 2.5), four when there are too few visibilities
    // for every warp.
    pl.warps = cells < 128 || nvis >= size_t(sms) * 32 ? (cells > 1024 ? 2 : 1) : 4;
    // FP32 grid tiles take a wide footprint's additions faster than the
    // grid's FP64 reductions do (that configuration, gridding only: 5.0
    // against 6.8 ms; the FP64 form's tiles do not, 8.0 against 6.8).
    if (tiles_fp32 && !use_d && cells > 900) return pl;
  } else {
    // Several planes per row: through the ring from 10 KB of slice on (4x4
    // planes, supports 8 to 16, 300k visibilities, both passes: 2.7 against
    // 5.4 ms; below, supports 4 to 8, 1M: 5.3 against 4.7 ms, but degridding
    // 3.1 against 3.9, gridding 3.4 against 4.3).  Beyond 48 KB the ring
    // holds too few visibilities, and the tiled kernel, which splits a slice
    // over the CTAs of a cluster, is faster (supports 8 to 32: 183 ms
    // per 10M visibilities against 315) once its pipeline has work: 5k
    // visibilities take 0.63 ms there, 0.49 here.
    pl.ring = mean >= 10 * 1024;
    pl.warps = !pl.ring ? 1 : part > 40 * 1024 ? 7 : 2;
    // whole KB of what the fixed parts leave; the largest slice must fit it
    if (pl.ring)
      p.ring_bytes = (kBudget - 1024 - layout(pl.warps, true)) / 1024 * 1024;
    if (pl.ring && !(runs_fit && np > 0 && part <= p.ring_bytes)) {
      // Slices beyond the ring and the tiled kernel (4x4 planes of supports
      // beyond 45) go to groups of 16 warps, one visibility per SM, whose
      // slices, read again for gridding, stay in L2 (supports 48 and 64, 20k
      // visibilities: 7.0 ms; groups of 8, two per SM, 7.9; the
      // per-visibility kernels 8.7).
      if (tiled_takes) return pl;
      pl.ring = false;
      pl.warps = 16;
    } else if (pl.ring && part > 48 * 1024 &&
               nvis > size_t(tiles_fp32 || use_g ? 6000 : 3000)) {
      return pl;
    }
  }
  if (pl.ring) {
    pl.smem = p.off_ring + p.ring_bytes;
  } else {
    p.ring_bytes = 0;
    pl.smem = std::max(layout(pl.warps, false), 1024);
    if (pl.smem * ctas_per_sm(false, n, pl.warps) > kBudget) return pl;
  }
  for (int r = 0; r < nrow; ++r)
    for (int w = 0; w < 2; ++w)
      for (int k = 0; k < (pl.diag ? 1 : n); ++k) {
        const int v = pl.diag ? p.vact[r] : k;
        auto place = [&](int m) {
          return uint32_t((m < 0 ? -1 : pl.ring ? pos[m] : m) & 0xff);
        };
        if (use_d) p.dpack[r][w] |= place(dset[w][r][v]) << (8 * k);
        if (use_g) p.gpack[r][w] |= place(gset[w][r][v]) << (8 * k);
      }
  // every element of every row active
  p.dense = 1;
  for (int r = 0; r < nrow; ++r)
    for (int w = 0; w < 2; ++w)
      for (int v = 0; v < n; ++v) {
        if (use_d && dset[w][r][v] < 0) p.dense = 0;
        if (use_g && gset[w][r][v] < 0) p.dense = 0;
      }
  p.evict_first = cf.table_bytes > size_t(96) << 20;
  pl.ctas = sms * ctas_per_sm(pl.ring, n, pl.warps);
  // whole rounds of blocks over the CTAs, several where there are
  // visibilities for it, so that the CTAs end level
  const size_t per_cta = (nvis + pl.ctas - 1) / size_t(pl.ctas);
  const size_t most = pl.ring ? kBlockVis : kFreeBlockVis;
  const size_t rounds = std::max<size_t>(per_cta >= 64 ? 4 : 1,
                                         (per_cta + most - 1) / most);
  p.block_vis = int(std::max<size_t>(
      1, (nvis + pl.ctas * rounds - 1) / (pl.ctas * rounds)));
  pl.ok = true;
  return pl;
}

// For tests (no device needed): the plan of a single launch of one gridder.
Status debug_stream_plan(unsigned npol, unsigned nrow, const int* mueller,
                         const int* taps, size_t ngroups, size_t nvis,
                         unsigned flags, bool has_model, bool mixed,
                         bool tiled_takes, hpgb_stream_plan* out) {
  hpgb_gridder g;
  g.npol = npol;
  g.grid_size[2] = nrow;
  g.grid_size[3] = 1;
  int set[4][4];
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c)
      set[r][c] = r < int(nrow) && c < int(npol) ? mueller[r * npol + c] : -1;
  for (size_t k = 0; k < ngroups; ++k) {
    CFGroup G{};
    G.taps_x = taps[2 * k];
    G.taps_y = taps[2 * k + 1];
    G.plane_stride = (G.taps_x * G.taps_y + 1) & ~1;
    g.cf.groups.push_back(G);
  }
  CFShape cf;
  cf.add(&g);
  const int(*both[2])[4] = {set, set};
  const StreamPlan pl = make_stream_plan(
      &g, cf, flags & HPGB_DO_DEGRID, flags & HPGB_DO_GRID, has_model, both,
      both, nvis, mixed, tiled_takes);
  *out = hpgb_stream_plan{pl.ok, pl.ring, pl.warps, pl.smem, pl.p.ring_bytes,
                          pl.p.off_ring, pl.p.nplanes * cf.max_plane_bytes};
  return Status::ok();
}

Status launch_stream(hpgb_gridder* g, int form, const StreamPlan& pl,
                     const StreamParams& p) {
  auto with = [&](auto f) -> Status {
    constexpr int F = decltype(f)::value;
    switch (g->npol) {
      case 1: return launch_stream_n<F, 1>(g, pl, p);
      case 2: return launch_stream_n<F, 2>(g, pl, p);
      case 3: return launch_stream_n<F, 3>(g, pl, p);
      case 4: return launch_stream_n<F, 4>(g, pl, p);
      default: return Status::err(HPGB_ERROR_OTHER, "bad polarization count");
    }
  };
  if (form == kLinear) return with(std::integral_constant<int, kLinear>());
  if (form == kMixed) return with(std::integral_constant<int, kMixed>());
  return with(std::integral_constant<int, kFP64>());
}

}  // namespace stream

using namespace stream;

// in_place: the records are the caller's, read where they lie; with `returned`
// they are copied there first and their values written there, without nothing
// is written back.
static Status grid_stream_run(hpgb_gridder* g, void* d_vis, size_t n,
                              unsigned flags, bool in_place, void* returned,
                              bool* used) {
  *used = false;
  const bool degrid = flags & HPGB_DO_DEGRID, grid = flags & HPGB_DO_GRID;
  if (n == 0 || n > size_t(0x7fffffff) || !(degrid || grid))
    return Status::ok();
  // (the mixed form degrids odd grid widths in FP64, by the kernels that do
  // not need its FP32 model)
  if (g->precision == HPGB_PRECISION_MIXED && degrid && g->has_model &&
      (g->grid_size[0] & 1))
    return Status::ok();
  // pos_w (w = 1): degrid uses conjugate indexes, grid uses indexes
  const int(*dset[2])[4] = {g->mt.m, g->mt.c};
  const int(*gset[2])[4] = {g->mt.c, g->mt.m};
  CFShape cf;
  cf.add(g);
  int side = 0;
  const bool tiled = tiled_plan_side(g, flags, n, &side);
  // The mixed form's FP32 arithmetic is the tiled kernel's: what that refuses
  // (footprints and slices too wide for its shared memory) was always computed
  // in FP64, by the per-visibility kernels (1 polarization, supports 8 and
  // 100: error against 64 bits 0 there, 1.0e-7 in the mixed form).
  const bool mixed = g->precision == HPGB_PRECISION_MIXED && tiled;
  const StreamPlan pl =
      make_stream_plan(g, cf, degrid, grid, g->has_model, dset, gset, n, mixed,
                       tiled);
  // (the hook that withholds a copy is for kernels that copy)
  if (!pl.ok || (g->withhold_vis >= 0 && !pl.ring)) return Status::ok();
  *used = true;
  g->last_kernel = tiled ? HPGB_KERNEL_TILED : HPGB_KERNEL_DIRECT;
  g->last_streamed = true;
  if (in_place && returned && returned != d_vis) {
    HPGB_CUDA_TRY(cudaMemcpyAsync(returned, d_vis, n * visdata_size(g->npol),
                                  cudaMemcpyDeviceToDevice, g->stream));
    d_vis = returned;
  }
  StreamPrep prep;
  HPGB_TRY(prepare_stream(g, d_vis, n,
                          stream_sorted(g, n, degrid && g->has_model), degrid,
                          grid, false, &prep, g->stream));
  if (mixed && degrid && g->has_model)
    HPGB_TRY(tiled::ensure_model32(g, g->stream));
  StreamParams p = pl.p;
  p.job.descs = prep.descs;
  p.job.srefs = prep.srefs;
  p.job.num_vis = prep.num_vis;
  p.job.cf = g->cf.data.as<const float2>();
  p.job.model = mixed ? g->model32.ptr : g->model.ptr;
  p.job.grid = g->grid.as<double2>();
  p.job.weights = g->weights.as<double>();
  p.job.records = static_cast<unsigned char*>(d_vis);
  p.job.nx = int(g->grid_size[0]);
  p.job.ny = int(g->grid_size[1]);
  p.update_weights = (flags & HPGB_UPDATE_GRID_WEIGHTS) != 0;
  p.rec_stride = int(visdata_size(g->npol));
  p.write_back = !in_place || returned;
  p.status = g->vb.counters.as<unsigned>();
  p.wait_limit_ns = g->wait_limit_ns;
  if (g->withhold_vis >= 0) p.withhold = prep.descs + g->withhold_vis;
  return launch_stream(g, mixed ? kMixed : kFP64, pl, p);
}

// the automatic choice, unless the tiled kernel's plan was set by hand
static bool automatic(const hpgb_gridder* g) {
  return g->kernel_kind == HPGB_KERNEL_AUTO && g->tplan.ring_parts == 0 &&
         g->tplan.chunk_vis == 0 && g->tplan.tile_side == 0;
}

Status grid_stream(hpgb_gridder* g, void* d_vis, size_t n, unsigned flags,
                   bool* used) {
  *used = false;
  if (!automatic(g)) return Status::ok();
  return grid_stream_run(g, d_vis, n, flags, false, nullptr, used);
}

// A copy takes records at any address, of any device or of the host, and
// into a buffer that overlaps them; the kernels want them aligned, in their
// own device's memory, and results in the same place or another.
bool records_in_place(int device, const void* vis, size_t bytes,
                      const void* returned) {
  auto usable = [device](const void* p) {
    cudaPointerAttributes a;
    if (reinterpret_cast<uintptr_t>(p) % 8 != 0) return false;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == device;
  };
  if (!usable(vis)) return false;
  if (!returned || returned == vis) return true;
  const uintptr_t a = reinterpret_cast<uintptr_t>(vis);
  const uintptr_t b = reinterpret_cast<uintptr_t>(returned);
  return (b >= a ? b - a : a - b) >= bytes && usable(returned);
}

Status grid_stream_device(hpgb_gridder* g, const void* vis, size_t n,
                          unsigned flags, void* returned, bool* used) {
  *used = false;
  if (!automatic(g) ||
      !records_in_place(g->device, vis, n * visdata_size(g->npol), returned))
    return Status::ok();
  return grid_stream_run(g, const_cast<void*>(vis), n, flags, true, returned,
                         used);
}

// Wide footprints that meet in the same tiles are gathered from, or added
// into, a tile in shared memory faster than they are in the grid, once a
// tile's visibilities pay for reading or adding the tile itself.  Nanoseconds
// on one B200 for c thousand cells (all rows) a visibility and v visibilities
// a tile: adjoint 4.85 c here against 1.8 + 3 c + 105 / v there, forward
// 2.3 c against 1.6 + 1.6 c + 95 / v (2 polarizations, supports 8 to 64, 3M
// visibilities on 2048^2: adjoint 49.3 against 37.2 ms, forward 23.1 against
// 21.5; 1M on 4096^2: 16.2 against 19.1 and 8.2 against 12.4; 1 polarization,
// supports 8 to 32, 1M on 1024^2: 2.4 against 3.2 and 1.2 against 2.3).  The
// tiles' passes (one a tile, of 2048 visibilities at most) must go several
// times round the SMs.  Slices that go through the ring stay there (4x4
// planes, supports 8 to 16, 500k visibilities on 1024^2: adjoint 4.0 against
// 6.9 ms), but for the forward operator on full tiles (3.8 against 3.6 ms with
// 800 visibilities a tile; 100k on 2048^2, 40 a tile, 0.89 against 0.99).
static bool tiles_for_linear(const hpgb_gridder* g, const StreamPlan& pl,
                             size_t n, bool gather) {
  if (!pl.diag && !(pl.ring && gather)) return false;
  if (!linear_tiled_fits(g)) return false;
  const double T = linear_tile_side(g);
  const double tiles = std::ceil(double(g->grid_size[0]) / T) *
                       std::ceil(double(g->grid_size[1]) / T);
  double c = 0.0;
  for (const CFGroup& G : g->cf.groups) c += double(G.taps_x) * G.taps_y;
  c *= 1e-3 * double(g->grid_size[2]) / double(g->cf.groups.size());
  const double v = double(n) / tiles;
  if (std::max(tiles, double(n) / 2048.0) < 4.0 * 148.0) return false;
  if (pl.ring) return v > 200.0;
  return gather ? 2.3 * c > 1.6 + 1.6 * c + 95.0 / v
                : 4.85 * c > 1.8 + 3.0 * c + 105.0 / v;
}

Status linear_op_stream(hpgb_gridder* g, const void* d_vis, size_t n, int op,
                        const void* in, void* out, bool* used) {
  *used = false;
  if (n == 0 || n > size_t(0x7fffffff)) return Status::ok();
  const bool gather = op == 0 || op == 3;
  // D and D^H use the degridding indexes, G and G^H the gridding ones
  const int(*set[2])[4] = {g->mt.m, g->mt.c};
  if (op >= 2) std::swap(set[0], set[1]);
  CFShape cf;
  cf.add(g);
  // (slices beyond the ring stay with the tiled or per-visibility operators)
  const StreamPlan pl =
      make_stream_plan(g, cf, gather, !gather, gather, set, set, n, false, true);
  if (!pl.ok || tiles_for_linear(g, pl, n, gather))
    return Status::ok();
  *used = true;
  StreamPrep prep;
  HPGB_TRY(prepare_stream(g, d_vis, n,
                          stream_sorted(g, n, false), gather, !gather, true,
                          &prep, g->stream));
  StreamParams p = pl.p;
  p.op = op;
  p.job.descs = prep.descs;
  p.job.srefs = prep.srefs;
  p.job.num_vis = prep.num_vis;
  p.job.cf = g->cf.data.as<const float2>();
  p.job.nx = int(g->grid_size[0]);
  p.job.ny = int(g->grid_size[1]);
  if (gather) {
    p.job.model = in;
    p.vals_out = static_cast<double2*>(out);
    // visibilities off the grid get zero
    HPGB_CUDA_TRY(cudaMemsetAsync(out, 0, n * g->npol * sizeof(double2),
                                  g->stream));
  } else {
    p.vals_in = static_cast<const double2*>(in);
    p.job.grid = static_cast<double2*>(out);
  }
  p.status = g->vb.counters.as<unsigned>();
  p.wait_limit_ns = g->wait_limit_ns;
  return launch_stream(g, kLinear, pl, p);
}

}  // namespace hpgb

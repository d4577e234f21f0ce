// stream_kernel.cuh -- one visibility per group of warps, from its CF slice
// to the grid, with no uv tiles and no exchange between CTAs: the automatic
// choice for degridding, gridding and both and for the linear operators
// (grid_stream.cu), and for batched launches (grid_batch.cu), where its plan
// says it is the faster one.
//
// A group of W warps takes one visibility with all its grid rows: it sums
// the footprint of every row against the model (read from global memory, L2
// mostly: the batch is sorted by uv tile where the grid exceeds that), adds
// the warps' partial sums through shared memory, forms the residual, and adds
// the footprint's increments to the FP64 grid with global reductions.
//
// What bounds it and why this shape.  The tiled kernel takes ~1000 cycles a
// visibility and CTA whatever the footprint: its roles hand a visibility on
// through shared memory, the CTAs of a cluster wait for one another's sums,
// and tiles want passes and flushes.  Large multi-plane slices hide that (74
// KB at the mean footprint of the full-polarization workload are 3230 cycles
// of an SM's share of HBM) and stay there; for footprints of 49 to a few
// thousand cells with a plane per row it is several times what their CF
// values and additions cost.  The additions can go straight to the grid:
// reductions on B200 are fast where a warp's lanes fall on consecutive 8-byte
// words, 640-660 G FP64 reductions a second measured into an L2-resident grid
// (lanes 16 bytes apart, real part then imaginary part: 330 G).  So lanes
// work in pairs that exchange one component.  Small footprints are then bound
// by instruction issue and the latency of their first loads, wide ones by
// the CF loads in flight (degridding) and the reductions (gridding).
//
// RING: slices stream into a byte ring of shared memory (bulk copies issued
// by two producer warps, as in tiled_kernel.cuh), each used twice, for
// degridding and for gridding; else the cell loops read them from global
// memory, twice when both passes are asked for (the second time from L2):
// for footprints so small that a bulk copy each (~430 cycles per SM whatever
// its size) would bound the kernel, and for slices that do not fit the ring.
#pragma once

#include <string>
#include <type_traits>

#include "gridder.cuh"
#include "ptx.cuh"
#include "tiles.cuh"

namespace hpgb {
namespace stream {

// Warps of a CTA.  With the ring, one CTA per SM, whose last two warps issue
// the copies; without, CTAs of eight warps, as many per SM as registers
// allow: the loops wait on global loads, so warps in flight are what they
// need.  One polarization runs in 80 registers (24 warps against 16: 1M
// visibilities of supports 8, 16 and 32 degridded and gridded 3.97 -> 3.22
// ms); more would spill there (two: 2.50 -> 2.87 ms degridding).
constexpr int kWarps = 16;      // ring
constexpr int kFreeWarps = 8;   // no ring
constexpr int kProducers = 2;
constexpr int warps_of(bool ring, int W) {
  return ring || W > kFreeWarps ? kWarps : kFreeWarps;
}
constexpr int ctas_per_sm(bool ring, int npol, int W) {
  return ring || W > kFreeWarps ? 1 : npol == 1 ? 3 : 2;
}
constexpr int kSlots = 32;      // visibilities in flight (ring)
constexpr int kMaxRuns = 8;
constexpr int kBlockVis = 16;   // consecutive visibilities a CTA takes, at most
constexpr int kFreeBlockVis = 64;  // without the ring

enum Form : int { kFP64 = 0, kMixed = 1, kLinear = 2 };

// per-gridder part of a batched launch, in global memory
struct StreamJob {
  const TileDesc* descs;
  const SliceRef* srefs;
  const float2* cf;
  const void* model;
  double2* grid;
  double* weights;
  unsigned char* records;
  const unsigned* num_vis;  // visibilities in descs
  int nx, ny;
};

struct StreamParams {
  StreamJob job;           // the gridder of a launch for one
  const StreamJob* jobs;   // batched launches: the job table, else null
  int njobs;
  int nrow;
  int do_degrid, do_grid, update_weights, has_model;
  int write_back;   // predictions or residuals go into the records
  int rec_stride;
  // slot planes (ring) or Mueller planes (no ring) of each row's elements
  // for w <= 0 and w > 0, a signed byte per element (-1: inactive); with one
  // element per row (DIAG), that element's in the lowest byte
  uint32_t dpack[4][2], gpack[4][2];
  int vact[4];  // DIAG: the row's element
  int nplanes, nruns;
  int run_plane[kMaxRuns], run_len[kMaxRuns], run_dst[kMaxRuns];
  int block_vis;    // consecutive visibilities a CTA takes
  int evict_first;  // the CF table is larger than L2: its lines go first
  int ring_bytes, off_part, off_offs, off_tab, off_ring, tab_taps;
  int dense;  // every element active: no activity tests
  int op;                  // linear operators: 0 D, 1 D^H, 2 G, 3 G^H
  const double2* vals_in;  // D^H, G: [n][npol]
  double2* vals_out;       // D, G^H: [n][npol]
  unsigned* status;
  unsigned long long wait_limit_ns;
  // test hook (ring): the copies for this descriptor are never issued
  const TileDesc* withhold;
};

// shared memory of the ring variant, from its start
struct Fixed {
  static constexpr int kFull = 0;                    // u64 [kSlots]
  static constexpr int kEmpty = kFull + 8 * kSlots;  // u64 [kSlots]
  static constexpr int kReq = kEmpty + 8 * kSlots;   // u64 [kSlots]
  static constexpr int kCtl = kReq + 8 * kSlots;     // WaitCtl
  static constexpr int kDead = kCtl + int(sizeof(ptx::WaitCtl));  // int [kWarps]
  static constexpr int kSlotEnd = kDead + 4 * kWarps;             // u64
  static constexpr int kReqSrc = kSlotEnd + 8 * kSlots;           // u64
  static constexpr int kReqDesc = kReqSrc + 8 * kSlots;           // u64
  static constexpr int kRingOff = kReqDesc + 8 * kSlots;          // int
  static constexpr int kReqPst = kRingOff + 4 * kSlots;           // int
  static constexpr int kIssued = kReqPst + 4 * kSlots;            // int
  static constexpr int kDesc = (kIssued + 4 * kSlots + 127) / 128 * 128;
  static constexpr int kEnd = kDesc + kSlots * int(sizeof(TileDesc));
};

// Row of footprint cell c (cells run along x, taps_x a row), given ch = c +
// 0.5: floor(ch / taps_x) by rounding ch * inv_tx - 0.5 to an integer in the
// mantissa of 1.5 * 2^23, without conversion or division.  Exact: with ch <
// 2^14 and taps_x < 128 the roundings move ch * inv_tx by less than 2^14 /
// taps_x * 2^-22, under its distance to a tie, which is 0.5 / taps_x at
// least.
__device__ __forceinline__ int cell_row(float ch, float inv_tx) {
  const float r = fmaf(ch, inv_tx, -0.5f) + 12582912.0f;
  return __float_as_int(r) - 0x4b400000;
}

// where the cell loops read CF values: the slot in the ring, or the slice in
// global memory; off in elements
template <bool RING>
struct CFRef {
  const float2* at;
  __device__ __forceinline__ CFRef plus(int off) const {
    return CFRef{at + off};
  }
  __device__ __forceinline__ float2 get(int off) const {
    if constexpr (RING)
      return at[off];
    else
      return __ldg(at + off);
  }
};

// a row's CF values at one cell; o: the row's plane offsets (-1: inactive)
template <int N, bool RING>
__device__ __forceinline__ void row_planes(const CFRef<RING>& cf, const int* o,
                                           bool dense, float2 (&v)[N]) {
  const int4 o4 = *reinterpret_cast<const int4*>(o);
  const int off[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (dense || off[k] >= 0) v[k] = cf.plus(off[k]).get(0);
}

// exp(i (phi_x(X) + phi_y(Y))) from the group's table of the two axes'
// phasors: taps_x + taps_y sine-cosine pairs per visibility instead of two
// per cell
__device__ __forceinline__ double2 screen_at(const double2* tab, int tx, int X,
                                             int Y) {
  return cmul_d(tab[X], tab[tx + Y]);
}

// Degridding sums (src/hpg_core.hpp:642-668) of A accumulators: element v of
// the sum over rows, or with one element per row (DIAG) row r.  The sign of
// the CF imaginary part (+1 for w > 0, else -1) is moved onto the model
// value's imaginary part and the sum's: sgn*(cf * m) with cf' = (cr, sgn*ci)
// equals the sum taken with (cr, ci) and (mx, sgn*my), imaginary part times
// sgn.  Mixed form: packed FP32 products, P = sum cf * (mx, mx) and Q = sum
// cf * (my, my) componentwise.  A lane sums up to 127 * 127 / 32 cells of
// every row, so chains end early, in a second pair of sums: after 16 cells
// (18 where six are taken at a time) when each row has its own sums (support
// 64: error against 64 bits 1.7e-7 in one chain, 1.2e-7 in two, 0.95e-7 with
// the warp's sums in FP64 too, which cost nothing: 2 polarizations, supports
// 16 to 64, 300k visibilities 1960 -> 1914 us), after 8 products when all
// rows add into them (4x4 planes, support 36: 64 products 1.04e-7, 8 0.81e-7,
// the tiled kernel 1.01e-7; supports 8 to 16, 300k visibilities, both passes:
// 2580 -> 2605 us).
template <int A, int FORM>
struct Sums {
  using V = typename std::conditional<FORM == kMixed, float2, double2>::type;
  V p[A], q[FORM == kMixed ? A : 1];
  V p2[FORM == kMixed ? A : 1], q2[FORM == kMixed ? A : 1];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < A; ++k) {
      p[k].x = p[k].y = 0;
      if constexpr (FORM == kMixed) {
        q[k].x = q[k].y = 0;
        p2[k].x = p2[k].y = q2[k].x = q2[k].y = 0;
      }
    }
  }
  // ends a chain of additions
  __device__ __forceinline__ void settle() {
    if constexpr (FORM == kMixed)
#pragma unroll
      for (int k = 0; k < A; ++k) {
        p2[k] = __fadd2_rn(p2[k], p[k]);
        q2[k] = __fadd2_rn(q2[k], q[k]);
        p[k] = q[k] = make_float2(0.f, 0.f);
      }
  }
  __device__ __forceinline__ void add(int k, float2 cf, V m, bool pos_w) {
    if constexpr (FORM == kMixed) {
      p[k] = __ffma2_rn(cf, make_float2(m.x, m.x), p[k]);
      q[k] = __ffma2_rn(cf, make_float2(m.y, m.y), q[k]);
    } else {
      const double my = pos_w ? m.y : -m.y;
      const double cr = cf.x, ci = cf.y;
      p[k].x = fma(cr, m.x, fma(-ci, my, p[k].x));
      p[k].y = fma(cr, my, fma(ci, m.x, p[k].y));
    }
  }
  __device__ __forceinline__ double value(int t, bool pos_w) const {
    const int k = t >> 1;
    if constexpr (FORM == kMixed) {
      const double u = (t & 1) ? p2[k].y : q2[k].y;
      return (t & 1) ? double(q2[k].x) + (pos_w ? u : -u)
                     : double(p2[k].x) - (pos_w ? u : -u);
    } else {
      return (t & 1) ? (pos_w ? p[k].y : -p[k].y) : p[k].x;
    }
  }
};

// A gridding value, conjugated when w > 0 (the CF imaginary part is negated
// then: conj(cf)*s*g = conj(cf*conj(s)*conj(g)), bit for bit in the
// reference's FP32 products, so only the sum's imaginary part flips), and the
// products of one row with it (src/hpg_core.hpp:856-873).  Mixed form, with s
// = -1 for w > 0 (else +1): the cell gains (s1.x + s2.y, s1.y + s2.x) for s1
// = sum cf * a, s2 = sum cf * b, a = (gx, s gx), b = (s gy, -gy), packed FP32.
template <int FORM>
struct Value {
  typename std::conditional<FORM == kLinear, double2, float2>::type a;
  float2 b;
  template <typename T>
  __device__ __forceinline__ void set(T g, bool pos_w) {
    if (pos_w) g.y = -g.y;
    if constexpr (FORM == kMixed) {
      const float sg = pos_w ? -1.0f : 1.0f;
      a = make_float2(g.x, sg * g.x);
      b = make_float2(sg * g.y, -g.y);
    } else {
      a = g;
    }
  }
};

template <int FORM>
struct Products {
  double2 s;      // FP64 sums
  float2 s1, s2;  // mixed form
  __device__ __forceinline__ void zero() {
    if constexpr (FORM == kMixed)
      s1 = s2 = make_float2(0.f, 0.f);
    else
      s = make_double2(0.0, 0.0);
  }
  __device__ __forceinline__ void add(float2 cf, const Value<FORM>& g,
                                      bool screen, float2 scf) {
    if constexpr (FORM == kMixed) {
      s1 = __ffma2_rn(cf, g.a, s1);
      s2 = __ffma2_rn(cf, g.b, s2);
    } else if constexpr (FORM == kLinear) {
      const double cr = cf.x, ci = cf.y;
      s.x = fma(cr, g.a.x, fma(-ci, g.a.y, s.x));
      s.y = fma(cr, g.a.y, fma(ci, g.a.x, s.y));
    } else {
      const float2 prod = screen ? cmul_f(cmul_f(cf, scf), g.a) : cmul_f(cf, g.a);
      s.x = __dadd_rn(s.x, double(prod.x));
      s.y = __dadd_rn(s.y, double(prod.y));
    }
  }
  // the cell's increment: of type T, float2 in the mixed form
  using T = typename std::conditional<FORM == kMixed, float2, double2>::type;
  __device__ __forceinline__ T done(bool pos_w, bool screen, double2 sc) const {
    if constexpr (FORM == kMixed) {
      float2 u = make_float2(s1.x + s2.y, s1.y + s2.x);
      if (screen) {
        const float sx = float(sc.x), sy = float(sc.y);
        u = make_float2(u.x * sx - u.y * sy, u.x * sy + u.y * sx);
      }
      return u;
    } else {
      double2 u = make_double2(s.x, pos_w ? -s.y : s.y);
      if constexpr (FORM == kLinear)
        if (screen) u = cmul_d(u, sc);
      return u;
    }
  }
};

// CTAs take a job's blocks in turn (a stretch of the tile order each leaves
// them uneven: measured up to 1.4x slower), each job's first one where the
// last job's ended.

// PASS: 1 degrids, 2 grids, 3 does both (kernels of their own: one with the
// passes as flags keeps the registers of both), 0: as p says.
template <int N, bool DIAG, int FORM, int W, bool RING, int PASS>
__global__ void __launch_bounds__(32 * warps_of(RING, W),
                                  ctas_per_sm(RING, N, W))
stream_kernel(const __grid_constant__ StreamParams p) {
  using V = typename Sums<N, FORM>::V;  // model element
  using G = typename std::conditional<FORM == kLinear, double2, float2>::type;
  constexpr int kCompute = RING ? kWarps - kProducers : warps_of(false, W);
  constexpr int kG = kCompute / W;  // groups
  constexpr int kT = 32 * W;        // threads of a group
  constexpr int NV = 2 * N;
  constexpr int NVP = NV <= 2 ? 2 : NV <= 4 ? 4 : 8;
  static_assert(kCompute % W == 0, "whole groups");
  extern __shared__ __align__(1024) unsigned char sm[];
  using F = Fixed;
  uint64_t* const full = reinterpret_cast<uint64_t*>(sm + F::kFull);
  uint64_t* const empty = reinterpret_cast<uint64_t*>(sm + F::kEmpty);
  uint64_t* const req = reinterpret_cast<uint64_t*>(sm + F::kReq);
  volatile int* const abort = reinterpret_cast<volatile int*>(sm + F::kCtl);
  volatile int* const dead = reinterpret_cast<volatile int*>(sm + F::kDead);
  unsigned long long* const slot_end =
      reinterpret_cast<unsigned long long*>(sm + F::kSlotEnd);
  const float2** const req_src = reinterpret_cast<const float2**>(sm + F::kReqSrc);
  const TileDesc** const req_desc =
      reinterpret_cast<const TileDesc**>(sm + F::kReqDesc);
  int* const ring_off = reinterpret_cast<int*>(sm + F::kRingOff);
  int* const req_pst = reinterpret_cast<int*>(sm + F::kReqPst);
  int* const issued = reinterpret_cast<int*>(sm + F::kIssued);
  TileDesc* const sdescs = reinterpret_cast<TileDesc*>(sm + F::kDesc);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  bool ok = true;
  if constexpr (RING) {
    if (tid == 0) {
      for (int s = 0; s < kSlots; ++s) {
        ptx::mbar_init(&full[s], 1);
        ptx::mbar_init(&empty[s], W);
        ptx::mbar_init(&req[s], 1);
        issued[s] = -1;
      }
      for (int g = 0; g < kWarps; ++g) dead[g] = 0x7fffffff;
      ptx::WaitCtl* ctl =
          reinterpret_cast<ptx::WaitCtl*>(const_cast<int*>(abort));
      ctl->flag = 0;
      ctl->copies = 0;
      ctl->limit_ns = p.wait_limit_ns;
      ptx::fence_mbar_init();
    }
    __syncthreads();
  }
  const bool degrid = PASS == 2 ? false
                      : PASS == 3 ? true
                                  : p.do_degrid && p.has_model;
  const bool do_grid = PASS ? PASS >= 2 : bool(p.do_grid);
  const int njobs = p.jobs ? p.njobs : 1;
  const bool cf_needed = degrid || do_grid;

  if (RING && warp >= kCompute) {
    // ---------------- producer warps ----------------
    // The lead warp reserves a slot and ring room for every visibility and
    // issues the copies of the even ones; the helper those of the odd ones,
    // as the lead requests them (a warp's bulk copies are taken up one after
    // another).
    uint64_t policy = 0;
    if (p.evict_first)
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;"
                   : "=l"(policy));
    auto issue = [&](const TileDesc* desc, const float2* slice, int s, int roff,
                     int pst, uint32_t q) {
      if (desc == p.withhold) return;
      const uint32_t pbytes = uint32_t(pst) * 8u;
      const uint32_t need = cf_needed ? uint32_t(p.nplanes) * pbytes : 0u;
      ring_off[s] = roff;
      ptx::mbar_expect_tx(&full[s], uint32_t(sizeof(TileDesc)) + need);
      ptx::bulk_g2s(&sdescs[s], desc, uint32_t(sizeof(TileDesc)), &full[s]);
      if (cf_needed) {
        unsigned char* dst = sm + p.off_ring + roff;
        for (int u = 0; u < p.nruns; ++u) {
          unsigned char* d = dst + uint32_t(p.run_dst[u]) * pbytes;
          const float2* src = slice + size_t(p.run_plane[u]) * pst;
          const uint32_t bytes = uint32_t(p.run_len[u]) * pbytes;
          if (p.evict_first)
            ptx::bulk_g2s_hint(d, src, bytes, &full[s], policy);
          else
            ptx::bulk_g2s(d, src, bytes, &full[s]);
        }
      }
      issued[s] = int(q);
    };
    uint32_t q = 0;
    uint32_t q_old = 0;           // oldest visibility not yet reclaimed
    unsigned long long head = 0;  // ring bytes allocated (monotonic)
    uint32_t pos = 0;             // head modulo the ring size
    unsigned long long tail = 0;  // ring bytes released (monotonic)
    const uint32_t rb = uint32_t(p.ring_bytes);
    unsigned first = blockIdx.x;
    for (int j = 0; j < njobs; ++j) {
      const StreamJob job = p.jobs ? p.jobs[j] : p.job;
      const unsigned n = *job.num_vis;
      const unsigned bv = unsigned(p.block_vis);
      const unsigned nb = (n + bv - 1) / bv;
      const TileDesc* jdescs = job.descs;
      const SliceRef* jsrefs = job.srefs;
      const float2* jcf = job.cf;
      unsigned b = first;
      // lane k: the slice reference of visibility k of the block, one block
      // ahead
      SliceRef next{};
      if (b < nb && lane < int(bv) && b * bv + lane < n)
        next = jsrefs[b * bv + lane];
      for (; b < nb; b += gridDim.x) {
        const unsigned i0 = b * bv;
        const int count = int(min(bv, n - i0));
        const SliceRef cur = next;
        const unsigned i1 = (b + gridDim.x) * bv;
        next = SliceRef{};
        if (b + gridDim.x < nb && lane < int(bv) && i1 + lane < n)
          next = jsrefs[i1 + lane];
        for (int k = 0; k < count; ++k, ++q) {
          const int s = int(q % uint32_t(kSlots));
          if (warp != kCompute) {
            if (q % kProducers == 0) continue;
            ok &= ptx::mbar_wait(&req[s], (q / kSlots) & 1, abort);
            if (lane == 0 && !*abort)
              issue(req_desc[s], req_src[s], s, ring_off[s], req_pst[s], q);
            __syncwarp();
            continue;
          }
          const long long off = __shfl_sync(0xffffffffu, cur.off, k);
          const int pst = __shfl_sync(0xffffffffu, cur.pstride, k);
          const uint32_t need =
              cf_needed ? uint32_t(p.nplanes) * uint32_t(pst) * 8u : 0u;
          // reclaim the oldest visibilities until a slot is free and the CF
          // part fits (allocations never straddle the ring's end)
          for (;;) {
            unsigned long long h = head;
            uint32_t ps = pos;
            if (need > 0 && ps + need > rb) {
              h += rb - ps;
              ps = 0;
            }
            const bool need_slot = (q - q_old) >= uint32_t(kSlots);
            // (an empty ring takes any part from its start)
            const bool need_space = need > 0 && h + need - tail > rb;
            if (!need_slot && !need_space) {
              head = h;
              pos = ps;
              break;
            }
            if (q_old == q) {
              // everything is released: start over at the ring's beginning
              head += rb - pos;
              pos = 0;
              tail = head;
              break;
            }
            const int so = int(q_old % uint32_t(kSlots));
            ok &= ptx::mbar_wait(&empty[so], (q_old / kSlots) & 1, abort);
            tail = slot_end[so];
            ++q_old;
          }
          // after an abort nothing is copied into slots that may still be read
          if (lane == 0 && !*abort) {
            slot_end[s] = head + need;
            if (q % kProducers == 0) {
              issue(jdescs + i0 + k, jcf + off, s, int(pos), pst, q);
            } else {
              ring_off[s] = int(pos);
              req_src[s] = jcf + off;
              req_pst[s] = pst;
              req_desc[s] = jdescs + i0 + k;
              ptx::mbar_arrive(&req[s]);
            }
          }
          head += need;
          pos += need;
          __syncwarp();
        }
      }
      first = b - nb;
    }
  } else {
    // ---------------- compute groups ----------------
    const int grp = warp / W, wig = warp % W;
    const int gt = wig * 32 + lane;  // thread of the group
    // partial sums of the group's warps
    double* const part =
        reinterpret_cast<double*>(sm + p.off_part) + grp * W * NV;
    double2* const tab =
        reinterpret_cast<double2*>(sm + p.off_tab) + grp * p.tab_taps;
    // plane offsets (elements) of the warp's visibility, [degridding,
    // gridding][row][element], -1 where inactive
    int* const offs = reinterpret_cast<int*>(sm + p.off_offs) + warp * 32;
    auto group_sync = [&]() {
      if constexpr (W == 1)
        __syncwarp();
      else
        ptx::named_sync(1 + grp, kT);
    };
    const int vl = lane < N ? lane : 0;
    uint32_t q = 0;
    unsigned first = blockIdx.x;
    bool live = true;
    for (int j = 0; j < njobs && live; ++j) {
      const StreamJob job = p.jobs ? p.jobs[j] : p.job;
      const unsigned n = *job.num_vis;
      const unsigned bv = unsigned(p.block_vis);
      const unsigned nb = (n + bv - 1) / bv;
      const int nx = job.nx, ny = job.ny;
      const size_t plane = size_t(nx) * ny;
      // grid weights: lane r of the group's first warp holds row r's sum of
      // the visibilities of one grid cube
      double wrow = 0.0;
      int wcube = -1;
      auto flush_weights = [&]() {
        if (wig == 0 && lane < p.nrow && wcube >= 0 && wrow != 0.0)
          atomicAdd(job.weights + size_t(wcube) * p.nrow + lane, wrow);
        wrow = 0.0;
      };
      unsigned b = first;
      for (; b < nb && live; b += gridDim.x) {
        const unsigned i0 = b * bv;
        const int count = int(min(bv, n - i0));
        // (groups take visibilities in turn by q, so that they stay level)
        const int k0 = int((uint32_t(grp) + kG - q % kG) % kG);
        long long next_off = 0;
        for (int k = k0; k < count; k += kG) {
          const uint32_t qq = q + uint32_t(k);
          const int s = int(qq % uint32_t(kSlots));
          const TileDesc* d;
          CFRef<RING> cfb;
          if constexpr (RING) {
            // the slot's previous visibility is released (so its copies have
            // landed, and the phase waited for next is this visibility's)
            bool got = qq < uint32_t(kSlots) ||
                       ptx::mbar_wait(&empty[s], (qq / kSlots - 1) & 1, abort);
            got = got && ptx::mbar_wait(&full[s], (qq / kSlots) & 1, abort);
            // one warp's failed wait ends the group's work, at this
            // visibility, for all its warps (a warp ahead of the others may
            // already have failed at a later one)
            if (!got) dead[grp] = int(qq);
            group_sync();
            if (dead[grp] <= int(qq)) {
              live = false;
              break;
            }
            d = &sdescs[s];
            cfb.at = reinterpret_cast<const float2*>(sm + p.off_ring + ring_off[s]);
          } else {
            group_sync();  // the last visibility's readers of part and tab
            d = job.descs + i0 + k;
            cfb.at = job.cf + (k == k0 ? job.srefs[i0 + k].off : next_off);
            // the group's next visibility of the block: its descriptor, and
            // the start of its CF slice, into L1 meanwhile
            if (k + kG < count) {
              const SliceRef sr = job.srefs[i0 + k + kG];
              next_off = sr.off;
              if (gt < 8)
                ptx::prefetch_l1(reinterpret_cast<const char*>(d + kG) + 32 * gt);
              else if (gt < 32 && 128 * (gt - 8) < p.nplanes * sr.pstride * 8)
                ptx::prefetch_l1(reinterpret_cast<const char*>(job.cf + next_off) +
                                 128 * (gt - 8));
            }
          }
          const int4 head4 = *reinterpret_cast<const int4*>(d);
          const int tx = head4.z & 0xff, ty = (head4.z >> 8) & 0xff;
          const int flags = (head4.z >> 16) & 0xff;
          const bool pos_w = flags & kPosW, screen = flags & kScreen;
          if (flags & kSkip) {  // off the grid
            if constexpr (RING) {
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(&empty[s]);
            }
            continue;
          }
          const int pst = head4.w, ncell = tx * ty;
          const float inv_tx = d->inv_tx;
          const int gx = d->abs_x, gy = d->abs_y, cube = d->cube;
          // cell (0, 0) of the footprint in row 0 of the visibility's cube
          const size_t org =
              (size_t(cube) * p.nrow * ny + size_t(gy)) * nx + size_t(gx);
          {
            const int r = (lane >> 2) & 3, v = lane & 3;
            const uint32_t pk = lane < 16 ? p.dpack[r][pos_w] : p.gpack[r][pos_w];
            const int pp = int(int8_t(pk >> (8 * v)));
            offs[lane] = pp < 0 ? -1 : pp * pst;
            __syncwarp();
          }
          double2 lin_in = make_double2(0.0, 0.0);
          if constexpr (FORM == kLinear)
            if (do_grid)
              lin_in = __ldg(p.vals_in + size_t(head4.x) * N + vl);
          if (screen && cf_needed) {
            for (int i = gt; i < tx + ty; i += kT) {
              const int a = i < tx ? 0 : 1;
              const int X = a ? i - tx : i;
              tab[i] = cphase_d(
                  __dadd_rn(d->phi0[a], __dmul_rn(double(X), d->dphi[a])));
            }
            group_sync();
          }
          double2 num = make_double2(0.0, 0.0);
          if (degrid) {
            const V* model = static_cast<const V*>(job.model) + org;
            Sums<N, FORM> sum;
            sum.zero();
            // kU cells at a time, their model values asked for together (two
            // polarizations, supports 8 to 64, 500k visibilities, mixed: 2.8
            // ms with four, 2.4 with six; asking for the next step's CF values
            // too: 3.4, two steps' registers leave too few)
            constexpr bool kAll = !DIAG && !RING;
            constexpr int kU = DIAG ? (FORM == kMixed && N == 2 ? 6 : 4) : kAll ? 1 : 2;
            constexpr int kRows = DIAG ? N : 4;
            // steps of a chain: 16 cells (18 with six at a time), or with
            // several rows in a sum, 8 products
            const int most =
                DIAG ? (16 + kU - 1) / kU : max(1, 8 / (kU * p.nrow));
            int chain = 0;
#pragma unroll 1
            for (int c0 = gt; c0 < ncell; c0 += kU * kT) {
              if (chain == most) {
                sum.settle();
                chain = 0;
              }
              ++chain;
              V m[kU][kRows];
              bool on[kU];
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                const int c = c0 + u * kT;
                on[u] = c < ncell;
                const int Y = cell_row(float(c) + 0.5f, inv_tx);
                const V* at = model + uint32_t(Y * (nx - tx) + c);
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                  if (on[u] && (DIAG || r < p.nrow))
                    m[u][r] = __ldg(at + size_t(r) * plane);
              }
              if (screen) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                  if (!on[u]) continue;
                  const int c = c0 + u * kT;
                  const int Y = cell_row(float(c) + 0.5f, inv_tx);
                  double2 sc = screen_at(tab, tx, c - Y * tx, Y);
                  sc.y = -sc.y;
#pragma unroll
                  for (int r = 0; r < kRows; ++r) {
                    if constexpr (FORM == kMixed) {
                      const float sx = float(sc.x), sy = float(sc.y);
                      m[u][r] = make_float2(m[u][r].x * sx - m[u][r].y * sy,
                                            m[u][r].x * sy + m[u][r].y * sx);
                    } else {
                      m[u][r] = cmul_d(m[u][r], sc);
                    }
                  }
                }
              }
              const CFRef<RING> cfc = cfb.plus(c0);
              if constexpr (kAll) {
                // a row's CF values ahead of its products
                float2 cf[2][N];
                row_planes<N, RING>(cfc, offs, p.dense, cf[0]);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                  if (r >= p.nrow) break;
                  if (r + 1 < 4 && r + 1 < p.nrow)
                    row_planes<N, RING>(cfc, offs + 4 * (r + 1), p.dense,
                                        cf[(r + 1) & 1]);
#pragma unroll
                  for (int v = 0; v < N; ++v)
                    if (p.dense || offs[4 * r + v] >= 0)
                      sum.add(v, cf[r & 1][v], m[0][r], pos_w);
                }
                continue;
              }
#pragma unroll
              for (int r = 0; r < kRows; ++r) {
                if (!DIAG && r >= p.nrow) break;
                if constexpr (DIAG) {
                  const CFRef<RING> pl = cfc.plus(offs[4 * r]);
#pragma unroll
                  for (int u = 0; u < kU; ++u)
                    if (on[u])
                      sum.add(r, pl.get(u * kT), m[u][r], pos_w);
                } else {
                  const int4 o4 = *reinterpret_cast<const int4*>(offs + 4 * r);
                  const int o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                  for (int v = 0; v < N; ++v) {
                    if (!p.dense && o[v] < 0) continue;
                    const CFRef<RING> pl = cfc.plus(o[v]);
#pragma unroll
                    for (int u = 0; u < kU; ++u)
                      if (on[u])
                        sum.add(v, pl.get(u * kT), m[u][r], pos_w);
                  }
                }
              }
            }
            sum.settle();
            // sums across the warp: halve the values held per lane while
            // there are several, then butterfly; every lane ends with one
            double v[NVP];
#pragma unroll
            for (int t = 0; t < NVP; ++t)
              v[t] = t < NV ? sum.value(t, pos_w) : 0.0;
            int comp = 0, o = 16;
#pragma unroll
            for (int m = NVP / 2; m > 0; m >>= 1, o >>= 1) {
              const bool hi = lane & o;
#pragma unroll
              for (int i = 0; i < m; ++i) {
                const double give = hi ? v[i] : v[i + m];
                const double keep = hi ? v[i + m] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
              }
              comp += hi ? m : 0;
            }
#pragma unroll
            for (int x = 16 / NVP; x > 0; x >>= 1)
              v[0] += __shfl_xor_sync(0xffffffffu, v[0], x);
            // and across the group's warps
            if ((lane & (32 / NVP - 1)) == 0 && comp < NV)
              part[wig * NV + comp] = v[0];
            group_sync();
            double tot = 0.0;
            if (lane < NV)
#pragma unroll
              for (int w = 0; w < W; ++w) tot += part[w * NV + lane];
            if constexpr (DIAG) {
              // row r belongs to element vact[r]
#pragma unroll
              for (int r = 0; r < N; ++r) {
                const double x = __shfl_sync(0xffffffffu, tot, 2 * r);
                const double y = __shfl_sync(0xffffffffu, tot, 2 * r + 1);
                if (p.vact[r] == vl) {
                  num.x += x;
                  num.y += y;
                }
              }
            } else {
              num.x = __shfl_sync(0xffffffffu, tot, 2 * vl);
              num.y = __shfl_sync(0xffffffffu, tot, 2 * vl + 1);
            }
          }
          // the visibility's values, identically in every warp
          const double2 phasor = d->phasor;
          G gout;
          gout.x = gout.y = 0;
          if constexpr (FORM == kLinear) {
            const double wgt = double(d->weights[vl]);
            const double2 wfac = d->wfac[vl];
            if (do_grid) {
              // D^H: phasor / conj(den) = conj(conj(phasor) / den);
              // G: phasor * w
              gout = cmul_d(p.op == 1 ? make_double2(wfac.x, -wfac.y)
                                      : make_double2(phasor.x * wgt,
                                                     phasor.y * wgt),
                            lin_in);
            } else if (wig == 0 && lane < N) {
              // D: conj(phasor) / den;  G^H: conj(phasor) * w
              p.vals_out[size_t(head4.x) * N + lane] =
                  cmul_d(num, p.op == 0 ? wfac
                                        : make_double2(phasor.x * wgt,
                                                       -phasor.y * wgt));
            }
          } else if (lane < N) {
            if (p.do_degrid) {
              float2 pred = make_float2(0.f, 0.f);
              if (degrid) {
                const double2 qv = cmul_d(num, d->wfac[lane]);
                pred = make_float2(__double2float_rn(qv.x),
                                   __double2float_rn(qv.y));
              }
              float2* out = reinterpret_cast<float2*>(
                  job.records + size_t(head4.x) * p.rec_stride);
              if (do_grid) {
                const float2 val = d->vals[lane];
                const float2 rr = make_float2(__fsub_rn(val.x, pred.x),
                                              __fsub_rn(val.y, pred.y));
                if (wig == 0 && p.write_back) out[lane] = rr;
                gout = scale_for_gridding(rr, phasor, d->weights[lane]);
              } else if (wig == 0 && p.write_back) {
                out[lane] = pred;
              }
            } else {
              gout = d->gvis[lane];
            }
          }
          if (do_grid) {
            if (wig == 0) {
              if (cube != wcube) {
                flush_weights();
                wcube = cube;
              }
              if (FORM != kLinear && lane < p.nrow && p.update_weights)
                wrow += d->twgt[lane];
            }
            // the elements' values; with one element per row, the rows'
            Value<FORM> gv[N];
#pragma unroll
            for (int v = 0; v < N; ++v) {
              const int src = DIAG ? p.vact[v] : v;
              G t;
              t.x = __shfl_sync(0xffffffffu, gout.x, src);
              t.y = __shfl_sync(0xffffffffu, gout.y, src);
              gv[v].set(t, pos_w);
            }
            // Lanes work in pairs: of 32 consecutive cells, lanes 2i and 2i + 1
            // form the increments of cells a = i and b = 16 + i; the even lane
            // gives a's imaginary part for b's real part, and the pair reduces
            // a's two words, then b's, so that each time the warp's 32 words
            // are consecutive (up to the footprint's row ends).
            const int h = lane & 1;
            double* const gbase = reinterpret_cast<double*>(job.grid + org) + h;
            // kU steps of 32 cells at a time, their CF values asked for
            // together
            constexpr int kU = DIAG ? (N == 1 ? 4 : N == 2 ? 6 : 2) : (N <= 2 ? 2 : 1);
            constexpr int kRows = DIAG ? N : 4;
#pragma unroll 1
            for (int w0 = wig * 32; w0 < ncell; w0 += kU * kT) {
              uint32_t at_a[kU], at_b[kU];
              float2 cfd[kU][DIAG ? N : 1];
              constexpr bool kAll = !DIAG && !RING;
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                const int ca = w0 + u * kT + (lane >> 1), c = ca + 16 * h;
                const int Ya = cell_row(float(ca) + 0.5f, inv_tx);
                const int Yb = cell_row(float(ca) + 16.5f, inv_tx);
                at_a[u] = uint32_t(Ya * (nx - tx) + ca);
                at_b[u] = uint32_t(Yb * (nx - tx) + ca + 16);
                if constexpr (DIAG)
#pragma unroll
                  for (int r = 0; r < N; ++r) {
                    cfd[u][r] = make_float2(0.f, 0.f);
                    if (c < ncell) cfd[u][r] = cfb.plus(offs[16 + 4 * r]).get(c);
                  }
              }
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                if (w0 + u * kT >= ncell) break;
                const int ca = w0 + u * kT + (lane >> 1), c = ca + 16 * h;
                const bool on_a = ca < ncell, on_b = ca + 16 < ncell;
                const bool on = h ? on_b : on_a;
                double2 sc = make_double2(1.0, 0.0);
                float2 scf = make_float2(1.0f, 0.0f);
                if (screen && on) {
                  const int Y = cell_row(float(c) + 0.5f, inv_tx);
                  sc = screen_at(tab, tx, c - Y * tx, Y);
                  scf = make_float2(__double2float_rn(sc.x),
                                    pos_w ? -__double2float_rn(sc.y)
                                          : __double2float_rn(sc.y));
                }
                float2 cfr[2][N];  // a row's CF values ahead of its products
                if constexpr (kAll)
                  if (on) row_planes<N, RING>(cfb.plus(c), offs + 16, p.dense, cfr[0]);
                double* dst_a = gbase + 2 * size_t(at_a[u]);
                double* dst_b = gbase + 2 * size_t(at_b[u]);
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                  if (!DIAG && r >= p.nrow) break;
                  Products<FORM> pr;
                  pr.zero();
                  if constexpr (DIAG) {
                    pr.add(cfd[u][r], gv[r], screen, scf);
                  } else if constexpr (kAll) {
                    if (on) {
                      if (r + 1 < 4 && r + 1 < p.nrow)
                        row_planes<N, RING>(cfb.plus(c), offs + 20 + 4 * r,
                                            p.dense, cfr[(r + 1) & 1]);
#pragma unroll
                      for (int v = 0; v < N; ++v)
                        if (p.dense || offs[16 + 4 * r + v] >= 0)
                          pr.add(cfr[r & 1][v], gv[v], screen, scf);
                    }
                  } else {
                    const int4 o4 =
                        *reinterpret_cast<const int4*>(offs + 16 + 4 * r);
                    const int o[4] = {o4.x, o4.y, o4.z, o4.w};
                    if (on) {
                      float2 cf[N];
#pragma unroll
                      for (int v = 0; v < N; ++v)
                        if (p.dense || o[v] >= 0) cf[v] = cfb.plus(o[v]).get(c);
#pragma unroll
                      for (int v = 0; v < N; ++v)
                        if (p.dense || o[v] >= 0)
                          pr.add(cf[v], gv[v], screen, scf);
                    }
                  }
                  const auto x = pr.done(pos_w, screen, sc);
                  const auto got =
                      __shfl_xor_sync(0xffffffffu, h ? x.x : x.y, 1);
                  if (on_a) atomicAdd(dst_a, double(h ? got : x.x));
                  if (on_b) atomicAdd(dst_b, double(h ? x.y : got));
                  dst_a += 2 * plane;
                  dst_b += 2 * plane;
                }
              }
            }
          }
          if constexpr (RING) {
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&empty[s]);
          }
        }
        q += uint32_t(count);
      }
      flush_weights();
      first = b - nb;
    }
    ok &= live;
  }
  if constexpr (RING) {
    // bulk copies issued into this CTA's shared memory have landed before it
    // leaves (after an abort the waits above return early)
    __syncthreads();
    if (tid == 0)
      for (int s = 0; s < kSlots; ++s)
        if (issued[s] >= 0)
          ok &= ptx::mbar_drain(&full[s], (uint32_t(issued[s]) / kSlots) & 1,
                                abort);
    if (!ok) atomicOr(p.status, kStatusWaitTimeout);
  }
}

}  // namespace stream
}  // namespace hpgb

// Tiled compositing: forward, adjoint, and the fused forward+loss+adjoint.
//
// Reference kernels restated:
//   forward   crates/rmesh-render/src/wgsl/rasterize_compute.wgsl:92-511
//   loss      crates/rmesh-train/src/wgsl/loss_compute.wgsl:24-72
//   adjoint   crates/rmesh-backward/src/wgsl/backward_tiled_compute.wgsl:154-587
//
// B200 layout.  The unit of work is a strip: SR rows of one tile.  One warp
// owns a strip from its first tet to its last and never meets a block barrier;
// persistent warps pull strips from a queue.  Two or three times as many
// independent instruction streams as one-CTA-per-tile phases, each with work in
// every phase, keep the issue slots busy: the kernel is bound by instruction
// issue, not by memory (see strip_kernel).
//
// Per batch of up to kBatch = 32 tets of the strip (lane = tet):
//
//   gather   the lanes read the next list positions' span words (one 32-bit
//            word: the pixel spans of four rows, pair_spans_kernel) and keep
//            the pairs that cover a pixel of the strip;
//   stage    each kept tet's 96-byte render record (face planes, colour,
//            gradient) comes by asynchronous copies into the warp's shared memory;
//   runs     each tet's covered pixels ("items", row by row) are cut into runs
//            of at most R, numbered tet-major over the batch; a round is the
//            next 32 runs, one per lane.  The batch's coverage bits are
//            transposed by shuffles into one 32-bit tet mask per pixel;
//   phase 0  lane = run: ray-tet intersection and segment integral of the run's
//            items (the tet's record stays in registers);
//   phase 1  lane = pixel (the only order-dependent part, a few instructions per
//            item): the owner walks its mask and composites front to back
//            (forward) or undoes back to front and leaves the restored
//            transmittance and d(logT) with the item (adjoint);
//   phase 2  adjoint only, lane = run again: the gradient of each item, summed
//            over the run into 24 moments, which the warp combines per tet (a
//            tet's runs sit in adjacent lanes) and adds to the entry's moments
//            in global memory; grad_finalize_kernel rebuilds the tet's
//            gradients from them once per step.
// A round may split a tet: a pixel meets a tet in one item only, and rounds
// follow the runs' order, so each pixel still sees its tets in order.
//
// Semantics kept from the reference: the forward includes vertices inside a
// pixel row (rasterize_compute.wgsl:236-242) and skips pixels whose
// log-transmittance fell below -13.8 (:257-262, :338); the adjoint uses edge
// crossings only (backward_tiled_compute.wgsl:241-299), takes the ray origin at
// the camera, undoes every covered tet (clamping log T at 0) and skips the
// gradient when the restored transmittance is below 1e-6 (:424-437).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "project.cuh"
#include "tma.cuh"

namespace rm {

constexpr int kBatch = 32;
constexpr int kSpanWords = 4;  // span words per pair and rule: 16 rows, four per word
// A row's span [lo, hi] (columns < 16) is one byte, lo << 4 | hi; an empty row is 0xF0 (lo > hi).
constexpr uint32_t kEmptySpans = 0xF0F0F0F0u;
__device__ __forceinline__ uint8_t pack_span(short2 sp) {
  return sp.x > sp.y ? (uint8_t)0xF0u : (uint8_t)((sp.x << 4) | sp.y);
}
// Moments per entry, summed over its items (see phase 2): columns 4f..4f+3 hold
// (S, P.x, P.y, P.z) of face f, 16 density, 17..19 colour, 20 the sum of the three
// colour gradients, 21..23 the colour gradient's gradient.
constexpr int kMom = 24;
// error statistics per tet: 10 sums, then two integer words: the pixel count and a maximum
constexpr int kErrMom = 12;
// per-lane rows of the warp's reduction buffers, with strides that spread a column
// of 16-byte accesses over all banks: the 16 face sums (column 16 free), and the
// other 8 sums (in the item area, once the round's items have been read)
constexpr int kRedCols = 20;
constexpr int kSumCols = 12;
constexpr int kStripWarps = 4;  // warps (independent strips) per CTA

constexpr int kAuxShared = 8;   // custom aux channels accumulated in shared memory

enum TileMode : int { kModeForward = 0, kModeBackward = 1, kModeTrain = 2, kModeError = 3 };

struct TileArgs {
  const ViewParams* views;
  int n_views;
  uint32_t n_tiles;
  const uint2* ranges;
  const uint32_t* pair_val;    // index of the pair's per-view tet record
  const TetView* vis_view;     // per-(view, visible tet) records
  const TetRec* rec;           // tet records (the forward's min_t path)
  const float4* color4;
  float* rgba;                 // [pixels][4] (forward output; optional in train mode)
  float* aux;                  // [pixels][8 + aux_dim] (optional, forward only)
  const float* aux_data;       // [M][aux_dim] per-tet custom channels (aux_dim > 0)
  int aux_dim;
  const float* dl_rgba;        // [pixels][4] (backward mode)
  // backward mode with AUX: gradient of the custom aux channels [pixels][aux_dim]
  // and the per-tet aux data gradient [M][aux_dim] (accumulated)
  const float* dl_aux;
  float* d_aux;
  const float* gt_rgb;         // [pixels][3] (train mode)
  const float* pixel_err;      // [pixels] (error mode)
  const float* ssim_err;       // [pixels] (error mode)
  float* mom;                  // [entries][kMom] (adjoint) or [M][kErrMom] (error mode), accumulated
  const float4* vis_color;     // SH colours per entry (the min_t path reads them), or nullptr
  Counters* counters;
  const AdamParams* hp;
  int persistent;
  // span words of the sorted pairs under the forward's rule and the adjoint's:
  // word w of pair i (rows 4w..4w+3) at [w * span_stride + i]
  const uint32_t* spans_fwd;
  const uint32_t* spans_adj;
  unsigned long long span_stride;
  // persistent launches: ticket -> tile (longest lists first); nullptr = identity
  const uint32_t* tile_order;
  // the launch covers global tiles [tile_lo, tile_lo + n_tiles) (the views of
  // one tile configuration); tile_order holds indices relative to tile_lo
  uint32_t tile_lo;
  uint32_t* ticket;  // persistent strip-queue head of this launch (zeroed before it)
};

// Strips of a tile: SR rows (1, 2 or 4) of TS pixels.
template <int TS, int SR>
struct StripCfg {
  static constexpr int S = TS / SR;         // strips per tile
  static constexpr int PX = TS * SR;        // pixels per strip (at most 64)
  static constexpr int NPX = (PX + 31) / 32;  // pixels per lane
  // items per run, as many as leave room for five CTAs per SM (four for 16-pixel
  // tiles); run lengths are odd, so that lanes at the same place of their runs
  // hit distinct banks
  static constexpr int RMAX = SR == 4 ? 5 : 7;
  static constexpr int SLOTS = 32 * RMAX;
  static_assert(TS % SR == 0 && PX <= 64, "strip shape");
  static_assert(RMAX % 2 == 1 && 16 * SLOTS >= 4 * 32 * kSumCols, "run length, room for the sums");
};

// Aux channels' part of a strip's shared memory (empty without them).
template <int SLOTS, int PX, bool AUX>
struct AuxSmem {
  float2 aux[SLOTS];           // forward: (t_min, t_max); backward: (aux_s, d a[tet] weight T_prev alpha)
  float caux[kAuxShared * PX];  // forward: the pixels' first custom channels
  uint32_t bent[kBatch];       // the batch's entries
};
template <int SLOTS, int PX>
struct AuxSmem<SLOTS, PX, false> {};

template <int TS, int SR, bool AUX>
struct __align__(16) StripSmem : AuxSmem<StripCfg<TS, SR>::SLOTS, StripCfg<TS, SR>::PX, AUX> {
  using Cfg = StripCfg<TS, SR>;
  __align__(16) float4 rec[kBatch][6];  // render records: nrm[4], cb, gm
  float4 v0[kBatch];            // adjoint: the tets' first vertices
  // per item slot (a run's items are consecutive).  Forward: (premultiplied rgb, od).  Adjoint
  // and error: .ex = (od, dl.c) -> (t_prev, d_od_state), .tt = (t_min, t_max)
  union {
    float4 item[Cfg::SLOTS];
    struct {
      float2 ex[Cfg::SLOTS];
      float2 tt[Cfg::SLOTS];
    } a;
  };
  __align__(16) float red[32][kRedCols];  // per-lane moment rows of phase 2
  uint16_t pk[Cfg::SLOTS];      // pack_item
  float4 pdir[Cfg::PX];         // pixel ray direction; w: the pixel's dL/dR (adjoint)
  float2 pdl[Cfg::PX];          // the pixel's dL/dG, dL/dB (adjoint); pixel and SSIM error (error mode)
  uint32_t qw[2 * kBatch];      // gathered pairs waiting for a batch: span word
  uint32_t qv[2 * kBatch];      //   and entry
  __align__(8) int16_t rowbase[kBatch][SR];  // per (tet, row): i0 with i0 + column = run * R + index in run
};

__device__ __forceinline__ float4 rec_vertex(const TetRec& r, int i) {
  return i == 0 ? r.a : (i == 1 ? r.b : (i == 2 ? r.c : r.d));
}

// Ray vs the four inward face planes with the reference's rules
// (rasterize_compute.wgsl:355-390): |den| < 1e-20 is parallel (outside if
// num > 0), entry = max t over den > 0 (strict), exit = min t over den < 0.
// Exact arithmetic: t_max - t_min cancels for thin tets.
__device__ __forceinline__ bool intersect4(const float4* nrm, const float* num_override, float dx, float dy, float dz,
                                           float& t_min, float& t_max, int& fmin, int& fmax) {
  t_min = -3.402823e38f;
  t_max = 3.402823e38f;
  fmin = 0;
  fmax = 0;
  bool ok = true;
  int entry = 4;
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const float4 n = nrm[f];
    const float den = dot3x(n.x, n.y, n.z, dx, dy, dz);
    const float num = num_override ? num_override[f] : n.w;
    if (fabsf(den) < 1e-20f) {
      if (num > 0.0f) ok = false;
      continue;
    }
    const float t = fdv(num, den);
    if (den > 0.0f) {
      if (t > t_min) { t_min = t; fmin = f; entry = f; }
    } else {
      if (t < t_max) { t_max = t; fmax = f; }
    }
  }
  if (entry == 4) fmin = 4;  // no entering face (the forward's entry normal is then zero)
  return ok && t_min < t_max;
}

// e^x and 1/x by the hardware approximations (one unit in the last place or
// two; results and arguments below 2^-126 count as zero).  Where they are used,
// that changes nothing: transmittances are compared with 1e-6, 1 - e^-od and the
// series' sums round such an e^-od away, and 1/x of an x above 2^126 is 0 in
// __fdividef too.
__device__ __forceinline__ float exp_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
  return r;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// num / den, correctly rounded, for 1e-20 <= |den| <= 2^60 and num 0 or 2^-60 <= |num|
// <= 2^60, where no intermediate can overflow or lose bits: a Newton step makes y the
// reciprocal to within rounding, and by Markstein's theorem (IBM J. Res. Dev. 34,
// 1990) one fused residual step from q = num * y then rounds the quotient correctly.
__device__ __forceinline__ float plain_quotient(float num, float den) {
  float y = rcp_fast(den);
  y = __fmaf_rn(y, __fmaf_rn(-den, y, 1.0f), y);
  const float q = fm(num, y);
  return __fmaf_rn(__fmaf_rn(-den, q, num), y, q);
}

// The same rules without branches, for planes whose numbers are in range (the
// record's kPlainPlanes bit) and a ray parallel to none of them; `plain` is false
// otherwise and the caller takes intersect4.  FACES: also the faces that gave t_min
// (4: none) and t_max.
template <bool FACES>
__device__ __forceinline__ bool intersect4_plain(const float4* nrm, float dx, float dy, float dz, float& t_min,
                                                 float& t_max, int& fmin, int& fmax, bool& plain) {
  float den[4], q[4];
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    den[f] = dot3x(nrm[f].x, nrm[f].y, nrm[f].z, dx, dy, dz);
    q[f] = plain_quotient(nrm[f].w, den[f]);
  }
  plain = fminf(fminf(fabsf(den[0]), fabsf(den[1])), fminf(fabsf(den[2]), fabsf(den[3]))) >= 1e-20f;
  t_min = -3.402823e38f;
  t_max = 3.402823e38f;
  fmin = 4;
  fmax = 0;
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const bool in = den[f] > 0.0f;
    if (FACES) {
      const bool a = in && q[f] > t_min, b = !in && q[f] < t_max;
      t_min = a ? q[f] : t_min;
      fmin = a ? f : fmin;
      t_max = b ? q[f] : t_max;
      fmax = b ? f : fmax;
    } else {  // (NaN quotients change nothing, as in the comparisons)
      t_min = fmaxf(t_min, in ? q[f] : -3.402823e38f);
      t_max = fminf(t_max, in ? 3.402823e38f : q[f]);
    }
  }
  return t_min < t_max;
}

// Segment integral of one item (rasterize_compute.wgsl:394-410).  The series
// and the quotient are both evaluated and one selected: od >= 1e-8, so the
// quotients are finite and inside the reference's +-1e20 clips.
struct Integral {
  float csr, csg, csb, cer, ceg, ceb;  // ReLU'd colours at entry / exit
  float dist, od_raw, od, alpha_t, rod, w0, w1;
};
__device__ __forceinline__ void integrate(const float4& cb, float dcdt, float t_min, float t_max, Integral& I) {
  I.csr = fmaxf(cb.x + dcdt * t_min, 0.f); I.csg = fmaxf(cb.y + dcdt * t_min, 0.f); I.csb = fmaxf(cb.z + dcdt * t_min, 0.f);
  I.cer = fmaxf(cb.x + dcdt * t_max, 0.f); I.ceg = fmaxf(cb.y + dcdt * t_max, 0.f); I.ceb = fmaxf(cb.z + dcdt * t_max, 0.f);
  I.dist = t_max - t_min;
  I.od_raw = cb.w * I.dist;
  I.od = clipf(I.od_raw, 1e-8f, 88.0f);
  I.alpha_t = exp_fast(-I.od);
  I.rod = rcp_fast(I.od);
  const float series = 1.0f + I.od * (-0.5f + I.od * (1.0f / 6.0f + I.od * (-1.0f / 24.0f)));
  const float ph = I.od < 0.02f ? series : (1.0f - I.alpha_t) * I.rod;
  I.w0 = ph - I.alpha_t;
  I.w1 = 1.0f - ph;
}

// Pixel spans of tile row `row` of one (tile, tet) pair, packed as pack_span:
// fwd under the forward's rule (rasterize_compute.wgsl:170-275: a row is
// reached when an edge crosses its centre line or a vertex lies in the row),
// adj under the adjoint's (backward_tiled_compute.wgsl:241-299: edge crossings
// only).  The vertex projections are taken minus the tile origin; columns past
// valid_cols (outside the image) are dropped, as the reference skips their
// pixels (rasterize_compute.wgsl:332).  The projections use fast arithmetic,
// and spans include pixels up to 0.001 px outside the silhouette, where the
// exact ray test misses anyway, so a last-bit difference in a span end changes
// no pixel value.
__device__ __forceinline__ short2 span_of_cols(float xl, float xr, int valid_cols) {
  short2 sp = make_short2(0, -1);
  if (xl <= xr) {
    // directed-rounding conversions: ceil / floor and the conversion in one step
    const int32_t lo = max(__float2int_ru(xl - 0.5f - 0.001f), 0);
    const int32_t hi = min(__float2int_rd(xr - 0.5f + 0.001f), valid_cols - 1);
    if (lo <= hi) sp = make_short2((short)lo, (short)hi);
  }
  return sp;
}
// One pair's set-up: the four vertices sorted by y and the slopes dx/dy of the
// edges between sorted ranks (an edge without height crosses no centre line, so
// its slope is never used).
struct SpanSetup {
  float x[4], y[4];
  float m01, m02, m03, m12, m13, m23;
  int first_row;   // row of the warp's task t of this pair: first_row + t
  int valid_cols;  // columns of the tile inside the image
};
// An edge crosses the row's centre line yc when its lower end is <= yc < its
// upper end, so with b vertices at or below yc the crossing edges are exactly
// the pairs (i, j) of sorted ranks i < b <= j: three edges for b = 1 or 3, four
// for b = 2, none otherwise.  The adjoint's span comes out empty without
// crossings; its reach (some edge crosses yc) implies the forward's.
__device__ __forceinline__ void row_spans(const SpanSetup& p, int row, bool adjoint, uint8_t& fwd, uint8_t& adj) {
  fwd = 0xF0u;
  adj = 0xF0u;
  const float yc = fa((float)row, 0.5f);
  const float blo = fs(yc, 0.5f), bhi = fa(yc, 0.5f);
  if (!(p.y[3] >= blo && p.y[0] < bhi)) return;
  const int nb = (p.y[0] <= yc ? 1 : 0) + (p.y[1] <= yc ? 1 : 0) + (p.y[2] <= yc ? 1 : 0) + (p.y[3] <= yc ? 1 : 0);
  float xl = 1e10f, xr = -1e10f;
  if (nb >= 1 && nb <= 3) {
    const float d0 = yc - p.y[0], d1 = yc - p.y[1];
    const float a = p.x[0] + d0 * p.m03;  // (0, 3) crosses in every band
    // (0, 1) | (0, 2) | (1, 3) for b = 1 | 2 | 3
    const float b = nb == 3 ? p.x[1] + d1 * p.m13 : p.x[0] + d0 * (nb == 1 ? p.m01 : p.m02);
    // (0, 2) | (1, 2) | (2, 3)
    const float c = nb == 1 ? p.x[0] + d0 * p.m02 : (nb == 2 ? p.x[1] + d1 * p.m12 : p.x[2] + (yc - p.y[2]) * p.m23);
    const float d = nb == 2 ? p.x[1] + d1 * p.m13 : a;  // (1, 3)
    xl = fminf(fminf(a, b), fminf(c, d));
    xr = fmaxf(fmaxf(a, b), fmaxf(c, d));
  }
  if (adjoint) adj = pack_span(span_of_cols(xl, xr, p.valid_cols));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (p.y[q] >= blo && p.y[q] < bhi) {
      xl = fminf(xl, p.x[q]);
      xr = fmaxf(xr, p.x[q]);
    }
  }
  fwd = pack_span(span_of_cols(xl, xr, p.valid_cols));
}

// pk packs the adjoint's entry (0..4) and exit (0..3) faces and the strip pixel (0..63)
__device__ __forceinline__ uint32_t pack_item(int fmin, int fmax, int p) {
  return (uint32_t)fmin | ((uint32_t)fmax << 3) | ((uint32_t)p << 5);
}

// 32 x 32 bit transpose across the warp: bit k of lane p's result is bit p of
// lane k's x (five exchange steps, each swapping the off-diagonal blocks).
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, int lane) {
  uint32_t m = 0x0000FFFFu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

__device__ __forceinline__ int next_bit(uint32_t& m) {
  const int p = __ffs(m) - 1;
  m &= m - 1u;
  return p;
}
__device__ __forceinline__ int next_bit(unsigned long long& m) {
  const int p = __ffsll(m) - 1;
  m &= m - 1ull;
  return p;
}
template <bool WIDE64>
struct PixMask {
  using T = uint32_t;
};
template <>
struct PixMask<true> {
  using T = unsigned long long;
};

// Covered pixels of span rows 0..r-1 in byte r of the result, the word's total in
// `total`: per byte, (hi | 0x80) - lo keeps bit 7 exactly when lo <= hi and holds
// hi - lo below it; the prefix sum of the widths is one multiply by 0x01010101
// (no byte carries: at most 4 x 16 = 64 pixels).  `width` gets the rows' widths.
__device__ __forceinline__ uint32_t span_prefix(uint32_t w, uint32_t& width, int& total) {
  const uint32_t lo = (w >> 4) & 0x0F0F0F0Fu, hi = w & 0x0F0F0F0Fu;
  const uint32_t d = (hi | 0x80808080u) - lo;
  const uint32_t mask = ((d & 0x80808080u) >> 7) * 0xFFu;
  width = ((d & 0x7F7F7F7Fu) + 0x01010101u) & mask;
  const uint32_t incl = width * 0x01010101u;
  total = (int)(incl >> 24);
  return incl - width;
}

// Bound by instruction issue and, at four to five warps per scheduler, by the
// latency between dependent instructions: one 801x603 step (19.8 M crossings,
// 0.57 M pairs) issues 0.74 instructions per cycle and scheduler, DRAM 1 % busy.
// Its tile-kernel time, before strips and after each step: 1.233 ms; strips with
// the branch-free division 1.100; branch-free compositing 0.982; combine in
// pieces, warp-wide copies 0.824; two-row strips 0.784; five CTAs per SM 0.753
// (96 registers, a few spills outside the item loops; shorter runs).  The
// adjoint alone keeps four CTAs: its launches are one view's, where the longest
// strip counts (512x512, 66 k tets, forward + adjoint: 0.418 against 0.444 ms).
// Packed two-float arithmetic (FFMA2) cut the instructions by 2 % and the time
// by nothing.
template <int TS, int SR, int MODE, bool AUX>
__global__ void __launch_bounds__(32 * kStripWarps, AUX ? 3 : (TS == 16 || MODE == kModeBackward ? 4 : 5))
    strip_kernel(TileArgs a) {
  using Cfg = StripCfg<TS, SR>;
  constexpr int S = Cfg::S, PX = Cfg::PX, NPX = Cfg::NPX, RMAX = Cfg::RMAX;
  using PMask = typename PixMask<(PX > 32)>::T;
  constexpr bool kAdjoint = MODE == kModeBackward || MODE == kModeTrain;
  extern __shared__ __align__(16) unsigned char strip_smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  StripSmem<TS, SR, AUX>& s = reinterpret_cast<StripSmem<TS, SR, AUX>*>(strip_smem_raw)[warp];
  const uint32_t n_units = a.n_tiles * (uint32_t)S;
  const uint32_t lanes_le = 0xffffffffu >> (31 - lane);

  uint32_t unit = blockIdx.x * (uint32_t)kStripWarps + (uint32_t)warp;
  while (true) {
    if (a.persistent) {
      if (lane == 0) unit = atomicAdd(a.ticket, 1u);
      unit = __shfl_sync(0xffffffffu, unit, 0);
    }
    if (unit >= n_units) break;
    uint32_t tile = unit / (uint32_t)S;
    const uint32_t strip = unit - tile * (uint32_t)S;
    if (a.persistent && a.tile_order) tile = a.tile_order[tile];
    const uint32_t g = tile + a.tile_lo;  // global tile id
    const int view = view_of_tile(a.views, a.n_views, g);
    const ViewParams& V = a.views[view];
    const uint32_t local_tile = g - V.tile_base;
    const uint32_t tile_y = local_tile / (uint32_t)V.tiles_x;
    const uint32_t tile_x = local_tile - tile_y * (uint32_t)V.tiles_x;
    const uint32_t x0 = tile_x * (uint32_t)TS, y0 = tile_y * (uint32_t)TS + strip * (uint32_t)SR;
    if (y0 >= (uint32_t)V.H) {  // rows below the image
      if (!a.persistent) break;
      continue;
    }
    const uint2 range = a.ranges[g];
    const uint32_t rs = range.x, re = range.y;
    const uint32_t n_list = re > rs ? re - rs : 0u;
    const float camx = V.cam[0], camy = V.cam[1], camz = V.cam[2];
    // forward ray origin cam + dir * min_t (rasterize_compute.wgsl:352); the
    // adjoint keeps the origin at the camera (backward_tiled_compute.wgsl:377)
    const bool has_min_t = V.min_t != 0.0f;

    // image index of strip pixel p
    auto strip_pixel = [&](int p) -> size_t {
      const int row = p / TS, col = p - (p / TS) * TS;
      return (size_t)V.pix_base + (size_t)(y0 + (uint32_t)row) * (size_t)V.W + (size_t)(x0 + (uint32_t)col);
    };

    // this lane's pixels p = 32 q + lane
    bool valid[NPX];
    size_t pix[NPX];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NPX; ++q) {
      const int p = 32 * q + lane;
      const int row = p / TS, col = p - (p / TS) * TS;
      const uint32_t px = x0 + (uint32_t)col, py = y0 + (uint32_t)row;
      valid[q] = p < PX && px < (uint32_t)V.W && py < (uint32_t)V.H;
      pix[q] = (size_t)V.pix_base + (size_t)py * (size_t)V.W + px;
      // pixel ray (rasterize_compute.wgsl:343-349), explicitly rounded: the ray and
      // the plane hits feed t_max - t_min, which cancels for thin tets, so they
      // are evaluated exactly as the reference's left-to-right float math.
      if (p < PX) {
        float ux = fdv(fs(fa((float)px, 0.5f), V.cx), V.fx);
        float uy = fdv(fs(fa((float)py, 0.5f), V.cy), V.fy);
        float uz = 1.0f;
        float l = __fsqrt_rn(dot3x(ux, uy, uz, ux, uy, uz));
        ux = fdv(ux, l); uy = fdv(uy, l); uz = fdv(uz, l);
        const float wx = fa(fa(fm(V.c2w[0], ux), fm(V.c2w[3], uy)), fm(V.c2w[6], uz));
        const float wy = fa(fa(fm(V.c2w[1], ux), fm(V.c2w[4], uy)), fm(V.c2w[7], uz));
        const float wz = fa(fa(fm(V.c2w[2], ux), fm(V.c2w[5], uy)), fm(V.c2w[8], uz));
        l = __fsqrt_rn(dot3x(wx, wy, wz, wx, wy, wz));
        s.pdir[p] = make_float4(fdv(wx, l), fdv(wy, l), fdv(wz, l), 0.0f);
      }
    }
    __syncwarp();

    // ---------------- batch machinery ----------------
    // list walk: the next 32 positions' span words and entries are loaded one
    // step ahead of the gather that uses them
    uint32_t off = 0u, wn = kEmptySpans, vn = 0u;
    int qn = 0;
    auto fetch = [&](bool fwd) {
      const uint32_t i = off + (uint32_t)lane;
      wn = kEmptySpans;
      vn = 0u;
      if (i < n_list) {
        const uint32_t pos = fwd ? re - 1u - i : rs + i;
        const uint32_t* sp = (fwd ? a.spans_fwd : a.spans_adj) + (strip * (uint32_t)SR / 4u) * a.span_stride;
        wn = __ldg(sp + pos);
        vn = __ldg(a.pair_val + pos);
        // the strip's rows of the word
        if (SR < 4) wn = ((wn >> (8u * SR * (strip % (4u / SR)))) & (0xFFFFFFFFu >> (32 - 8 * SR))) | (kEmptySpans << (8 * SR & 31));
      }
    };
    auto start_list = [&](bool fwd) {
      off = 0u;
      qn = 0;
      fetch(fwd);
    };
    // the batch (lane = tet): span word, entry, pixels, pixels of the rows above
    // each row, first run; and its totals
    uint32_t bw = kEmptySpans, bv = 0u, bcum = 0u;
    PMask bmask = 0;
    int bcnt = 0, brun = 0, n_runs = 0, R = 1;
    uint32_t tmask[NPX];     // tets of the batch covering each of this lane's pixels
    // gathers the next batch, starts its record copies and prepares its runs;
    // returns its number of tets (0: list done)
    auto next_batch = [&](bool fwd) -> int {
      while (qn < kBatch && off < n_list) {
        const bool some = wn != kEmptySpans;
        const unsigned bal = __ballot_sync(0xffffffffu, some);
        if (some) {
          const int at = qn + __popc(bal & (lanes_le >> 1));
          s.qw[at] = wn;
          s.qv[at] = vn;
        }
        qn += __popc(bal);
        off += 32u;
        fetch(fwd);
      }
      if (qn == 0) return 0;
      __syncwarp();
      const int nb = min(qn, kBatch);
      bw = lane < nb ? s.qw[lane] : kEmptySpans;
      bv = lane < nb ? s.qv[lane] : 0u;
      qn -= nb;
      const uint32_t w2 = s.qw[kBatch + lane], v2 = s.qv[kBatch + lane];
      __syncwarp();
      if (lane < qn) {
        s.qw[lane] = w2;
        s.qv[lane] = v2;
      }
      if constexpr (AUX) s.bent[lane] = bv;
      // records (the warp has read the previous batch's): six 16-byte pieces each,
      // consecutive lanes on consecutive pieces.  Asynchronous copies of a warp are
      // one instruction for 32 pieces, where a bulk copy per record issues alone.
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const int c = 32 * i + lane, k = c / 6;
        const uint32_t entry = __shfl_sync(0xffffffffu, bv, k);
        if (k < nb) async_copy16(&s.rec[0][0] + c, reinterpret_cast<const float4*>(a.vis_view + entry) + (c - 6 * k));
      }
      if (!fwd && lane < nb) async_copy16(&s.v0[lane], &a.rec[bv / (uint32_t)a.n_views].a);
      // pixels
      uint32_t width;
      bcum = span_prefix(bw, width, bcnt);
      bmask = 0;
#pragma unroll
      for (int r = 0; r < SR; ++r) {
        const uint32_t wr = (width >> (8 * r)) & 255u, lo = (bw >> (8 * r + 4)) & 15u;
        bmask |= (PMask)(((1u << wr) - 1u) << lo) << (r * TS);
      }
      // run length: the cheapest of a few, a round costing about its longest
      // run plus one item's work for the set-up and the combine
      const int cmax = __reduce_max_sync(0xffffffffu, bcnt);
      constexpr int kCand[3] = {RMAX, RMAX > 5 ? 5 : 3, 3};
      int best = 0x7fffffff;
      uint32_t rmul = 0u;
#pragma unroll
      for (int i = 0; i < (RMAX > 5 ? 3 : 2); ++i) {
        const int total = __reduce_add_sync(0xffffffffu, (bcnt + kCand[i] - 1) / kCand[i]);
        const int cost = ((total + 31) >> 5) * (min(kCand[i], cmax) + 1);
        if (cost < best) {
          best = cost;
          R = kCand[i];
          rmul = (65536u + (uint32_t)kCand[i] - 1u) / (uint32_t)kCand[i];  // n / R = n * rmul >> 16 for small n
        }
      }
      const int nr = (int)(((uint32_t)(bcnt + R - 1) * rmul) >> 16);
      int x = nr;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      brun = x - nr;
      n_runs = __shfl_sync(0xffffffffu, x, 31);
      {
        const int i0 = brun * R;
        int b[SR];
#pragma unroll
        for (int r = 0; r < SR; ++r)
          b[r] = i0 + (int)((bcum >> (8 * r)) & 255u) - (int)((bw >> (8 * r + 4)) & 15u);
#pragma unroll
        for (int r = 0; r < SR; ++r) s.rowbase[lane][r] = (int16_t)b[r];
      }
#pragma unroll
      for (int q = 0; q < NPX; ++q) tmask[q] = warp_transpose_bits((uint32_t)(bmask >> (q ? 32 : 0)), lane);
      async_copy_wait();
      __syncwarp();
      return nb;
    };

    // the round's run of this lane: tet slot, first pixels, number of items;
    // heads: lanes > 0 whose run is the first of its tet (or past the last run)
    int rk = 0, rk0 = 0, rklast = 0, rlen = 0;
    uint32_t rentry = 0u;
    PMask rmask = 0;
    unsigned heads = 0u;
    auto take_runs = [&](int base) {
      rk0 = __popc(__ballot_sync(0xffffffffu, brun <= base)) - 1;  // tet of run `base`
      const int d = brun - base;
      heads = __reduce_or_sync(0xffffffffu, d > 0 && d < 32 ? 1u << d : 0u);
      rk = min(rk0 + __popc(heads & lanes_le), kBatch - 1);
      rklast = __shfl_sync(0xffffffffu, rk, 31);
      const int run0 = __shfl_sync(0xffffffffu, brun, rk);
      const int cnt = __shfl_sync(0xffffffffu, bcnt, rk);
      const uint32_t w = __shfl_sync(0xffffffffu, bw, rk);
      const uint32_t cum = __shfl_sync(0xffffffffu, bcum, rk);
      rmask = __shfl_sync(0xffffffffu, bmask, rk);
      rentry = __shfl_sync(0xffffffffu, bv, rk);
      const int n0 = (base + lane - run0) * R;
      rlen = base + lane < n_runs ? min(R, cnt - n0) : 0;
      int row = 0;
#pragma unroll
      for (int r = 1; r < SR; ++r) row += n0 >= (int)((cum >> (8 * r)) & 255u) ? 1 : 0;
      const int col = (int)((w >> (8 * row + 4)) & 15u) + n0 - (int)((cum >> (8 * row)) & 255u);
      rmask &= ~(PMask)0 << ((row * TS + col) & (8 * (int)sizeof(PMask) - 1));
    };
    // phase 0: intersection + integral of the run's items.  Colours are clipped
    // at 0 in the forward (rasterize_compute.wgsl:409), at -1e20 in the adjoint (:411).
    auto phase0 = [&](auto forward) {
      constexpr bool fwd = decltype(forward)::value;
      if (rlen > 0) {
        float4 nrm[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) nrm[f] = s.rec[rk][f];
        const float4 cb0 = s.rec[rk][4], gg = s.rec[rk][5];
        const bool moved = fwd && has_min_t;  // rays start at min_t
        const bool in_range = (__float_as_uint(gg.w) & kPlainPlanes) && !moved;
        int slot = lane * R;
        PMask m = rmask;
#pragma unroll 1
        for (int j = 0; j < rlen; ++j, ++slot) {
          const int p = next_bit(m);
          const float4 d = s.pdir[p];
          float4 cb = cb0;
          float t_min, t_max;
          int fmin, fmax;
          bool plain;
          bool hit = intersect4_plain<(AUX || !fwd)>(nrm, d.x, d.y, d.z, t_min, t_max, fmin, fmax, plain);
          if (!(plain && in_range)) {
            float numo[4] = {nrm[0].w, nrm[1].w, nrm[2].w, nrm[3].w};
            if (moved) {
              // origin cam + d*min_t: num = dot(n, va - o), base offset dot(g, o - v0)
              const float oxp = fa(camx, fm(d.x, V.min_t)), oyp = fa(camy, fm(d.y, V.min_t)),
                          ozp = fa(camz, fm(d.z, V.min_t));
              const uint32_t tet = rentry / (uint32_t)a.n_views;
              const TetRec rr = a.rec[tet];
#pragma unroll
              for (int f = 0; f < 4; ++f) {
                const float4 v = rec_vertex(rr, kFacesH[f][0]);
                numo[f] = dot3x(nrm[f].x, nrm[f].y, nrm[f].z, fs(v.x, oxp), fs(v.y, oyp), fs(v.z, ozp));
              }
              const float bo = dot3x(gg.x, gg.y, gg.z, fs(oxp, rr.a.x), fs(oyp, rr.a.y), fs(ozp, rr.a.z));
              const float4 cc = a.vis_color ? a.vis_color[rentry] : a.color4[tet];
              cb = make_float4(fa(cc.x, bo), fa(cc.y, bo), fa(cc.z, bo), cb0.w);
            }
            hit = intersect4(nrm, numo, d.x, d.y, d.z, t_min, t_max, fmin, fmax);
          }
          // a ray that misses leaves od < 0
          const float dcdt = gg.x * d.x + gg.y * d.y + gg.z * d.z;
          Integral I;
          integrate(cb, dcdt, t_min, t_max, I);
          const float lo = fwd ? 0.f : kMinVal;
          const float4 out = make_float4(clipf(I.cer * I.w0 + I.csr * I.w1, lo, kMaxVal),
                                         clipf(I.ceg * I.w0 + I.csg * I.w1, lo, kMaxVal),
                                         clipf(I.ceb * I.w0 + I.csb * I.w1, lo, kMaxVal), hit ? I.od : -1.0f);
          const float2 out_t = make_float2(t_min, t_max);
          const uint32_t out_p = pack_item(fmin, fmax, p);
          if (MODE == kModeError) {
            s.a.ex[slot] = make_float2(out.w, 0.0f);
            s.a.tt[slot] = out_t;
            s.pk[slot] = (uint16_t)out_p;
          } else if (fwd) {
            s.item[slot] = out;
            if constexpr (AUX) {
              s.aux[slot] = out_t;
              s.pk[slot] = (uint16_t)out_p;
            }
          } else {
            const float2 dgb = s.pdl[p];
            float dlc = d.w * out.x + dgb.x * out.y + dgb.y * out.z;
            if constexpr (AUX && MODE == kModeBackward) {
              // custom aux channels (aux += T alpha a[tet], rasterize_compute.wgsl:458-462)
              // continue the transmittance chain like a colour alpha a[tet]:
              // aux_s = sum_ai dl_aux[pixel][ai] a[tet][ai]
              const float* dla = a.dl_aux + strip_pixel(p) * (size_t)a.aux_dim;
              const float* ad = a.aux_data + (size_t)(rentry / (uint32_t)a.n_views) * a.aux_dim;
              float aux_s = 0.0f;
              for (int ai = 0; ai < a.aux_dim; ++ai) aux_s += dla[ai] * ad[ai];
              dlc += (1.0f - I.alpha_t) * aux_s;
              s.aux[slot] = make_float2(aux_s, 0.0f);
            }
            s.a.ex[slot] = make_float2(out.w, dlc);
            s.a.tt[slot] = out_t;
            s.pk[slot] = (uint16_t)out_p;
          }
        }
      }
    };
    // phase 1: the round's tets of pixel q (taken out of tmask).  Only the tet of
    // the round's last run may continue in the next round: its item at this pixel
    // is looked up once.
    auto take_tets = [&](int q, int base, bool on) -> uint32_t {
      const int row = (32 * q + lane) / TS & (SR - 1), col = (32 * q + lane) % TS;
      uint32_t m = on ? tmask[q] & ((2u << rklast) - 1u) : 0u;
      if ((m >> rklast) & 1u) {
        if ((int)s.rowbase[rklast][row] + col >= (base + 32) * R) m ^= 1u << rklast;
      }
      tmask[q] &= ~m;
      return m;
    };
    // slot of (tet k, this lane's pixel q) in the round that starts at run `base`
    auto slot_of = [&](int k, int q, int base) -> int {
      const int row = (32 * q + lane) / TS & (SR - 1), col = (32 * q + lane) % TS;
      return (int)s.rowbase[k][row] + (col - base * R);
    };
    // adds the lanes' rows (one per run) to `dst` per tet.  The rows are cut into
    // pieces of one tet and at most eight rows; six lanes (four columns each) take
    // a piece, five pieces at a time, and add its sums with 16-byte atomics.
    auto combine = [&](int base, float* dst) {
      static_assert(kMom == 24, "six lanes of four columns");
      const int n_rows = min(32, n_runs - base);
      const unsigned cuts = (heads | 0x01010101u) & (0xffffffffu >> (32 - n_rows));
      const int n_pieces = __popc(cuts);
      // piece i's first row and tet slot, in a padding column of row i
      if ((cuts >> lane) & 1u) s.red[__popc(cuts & (lanes_le >> 1))][16] = __int_as_float(lane | (rk << 8));
      __syncwarp();
      const int sub = lane / 6, col = 4 * (lane - 6 * sub);
      const float* src = col < 16 ? &s.red[0][col] : reinterpret_cast<const float*>(&s.item[0]) + (col - 16);
      const int stride = col < 16 ? kRedCols : kSumCols;
      for (int i0 = 0; i0 < n_pieces; i0 += 5) {
        const int i = i0 + sub;
        const bool on = lane < 30 && i < n_pieces;
        const int pc = on ? __float_as_int(s.red[i][16]) : 0;
        const uint32_t entry = __shfl_sync(0xffffffffu, bv, pc >> 8);
        if (on) {
          const int r1 = i + 1 < n_pieces ? __float_as_int(s.red[i + 1][16]) & 255 : n_rows;
          int r = pc & 255;
          float4 sum = *reinterpret_cast<const float4*>(src + r * stride);
          for (++r; r < r1; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(src + r * stride);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
          if (sum.x != 0.0f || sum.y != 0.0f || sum.z != 0.0f || sum.w != 0.0f)
            atomicAdd(reinterpret_cast<float4*>(dst + (size_t)entry * kMom + col), sum);
        }
      }
    };
    // the same for the error statistics: lane c sums column c over each tet's
    // adjacent rows; the last two columns are integers, a sum (exact at any image
    // size) and a maximum
    auto combine_error = [&](int base, float* dst) {
      const int n_rows = min(32, n_runs - base);
      int k = rk0;
      for (int r0 = 0; r0 < n_rows; ++k) {  // one tet's rows [r0, r1) at a time
        const unsigned later = heads & ~((2u << r0) - 1u);
        const int r1 = later ? min(__ffs(later) - 1, n_rows) : n_rows;
        const uint32_t entry = __shfl_sync(0xffffffffu, bv, k);
        if (lane < kErrMom) {
          float* at = dst + (size_t)entry * kErrMom + lane;
          float sum = 0.0f;
          uint32_t count = 0u;
          int mx = 0;
          for (int r = r0; r < r1; ++r) {  // one walk for the three kinds of column
            const float v = s.red[r][lane];
            sum += v;
            count += __float_as_uint(v);
            mx = max(mx, __float_as_int(v));
          }
          if (lane < kErrMom - 2) {
            if (sum != 0.0f) atomicAdd(at, sum);
          } else if (lane == kErrMom - 2) {
            if (count != 0u) atomicAdd(reinterpret_cast<uint32_t*>(at), count);
          } else {
            if (mx > 0) atomicMax(reinterpret_cast<int*>(at), mx);
          }
        }
        r0 = r1;
      }
    };

    float Cr[NPX], Cg[NPX], Cb[NPX], logT[NPX];
#pragma unroll
    for (int q = 0; q < NPX; ++q) Cr[q] = Cg[q] = Cb[q] = logT[q] = 0.0f;

    // =============== forward (front to back) ===============
    if (MODE == kModeForward || MODE == kModeTrain) {
      float nd[AUX ? NPX : 1][4], en[AUX ? NPX : 1][4];
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        if constexpr (AUX) {
#pragma unroll
          for (int i = 0; i < 4; ++i) nd[q][i] = en[q][i] = 0.0f;
          // custom aux channels (rasterize_compute.wgsl:458-462): the first accumulate
          // in shared memory, the others in place in the pixel's output row
          if (valid[q]) {
            for (int ai = 0; ai < kAuxShared; ++ai) s.caux[ai * PX + 32 * q + lane] = 0.0f;
            for (int ai = kAuxShared; ai < a.aux_dim; ++ai) a.aux[pix[q] * (size_t)(8 + a.aux_dim) + 8 + ai] = 0.0f;
          }
        }
      }
      start_list(true);
      while (true) {
        const int nb = next_batch(true);
        if (nb == 0) break;
        for (int base = 0; base < n_runs; base += 32) {
          take_runs(base);
          phase0(std::true_type{});
          __syncwarp();
          // phase 1: composite each pixel's items nearest first.  The lane's pixels
          // advance together (two chains in flight) and without branches: an item
          // that does not count (ray miss, T below the cut) has weight 0.
          uint32_t m[NPX], any = 0u;
#pragma unroll
          for (int q = 0; q < NPX; ++q) {
            m[q] = take_tets(q, base, true);
            if (logT[q] < -13.8f) m[q] = 0u;
            any |= m[q];
          }
          while (any) {
            any = 0u;
#pragma unroll
            for (int q = 0; q < NPX; ++q) {
              const bool has = m[q] != 0u;
              const int k = (__ffs(m[q]) - 1) & 31;
              const int slot = has ? slot_of(k, q, base) : 0;
              m[q] &= m[q] - 1u;
              const float4 c = s.item[slot];
              const float Tj = exp_fast(fmaxf(logT[q], -88.0f));
              const bool on = has && c.w >= 0.0f && Tj >= 1e-6f;
              const float w = on ? Tj : 0.0f;
              Cr[q] += c.x * w; Cg[q] += c.y * w; Cb[q] += c.z * w;
              logT[q] -= on ? c.w : 0.0f;
              if (logT[q] < -13.8f) m[q] = 0u;  // saturated: the rest is skipped
              any |= m[q];
              if constexpr (AUX) {
                if (!on) continue;
                const float2 c2 = s.aux[slot];
                const float t_min = c2.x, t_max = c2.y;
                const int entry = (int)(s.pk[slot] & 7u);
                const float od = c.w;
                const float alpha_t = exp_fast(-od);  // as the intersection phase computed it
                const float ph = fabsf(od) < 0.02f
                                     ? 1.0f + od * (-0.5f + od * (1.0f / 6.0f + od * (-1.0f / 24.0f)))
                                     : clipf(__fdividef(1.0f - alpha_t, od), kMinVal, kMaxVal);
                const float w0 = ph - alpha_t, w1 = 1.0f - ph;
                const float alpha = 1.0f - alpha_t;
                float enx = 0.f, eny = 0.f, enz = 0.f;
                if (entry < 4) {
                  const float4 n = s.rec[k][entry];
                  // (the root and the quotients correctly rounded: an output of its own)
                  const float l = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
                  enx = -n.x / l; eny = -n.y / l; enz = -n.z / l;
                }
                const float ta = Tj * alpha;
                nd[q][0] += ta * enx; nd[q][1] += ta * eny; nd[q][2] += ta * enz;
                nd[q][3] += Tj * (w0 * t_max + w1 * t_min);
                const float wt = alpha * Tj;
                const float cmid = (t_min + t_max) * 0.5f;
                const float wc = wt * cmid;
                en[q][0] += wt;
                en[q][1] += wt > 1e-20f ? wt * logf(wt) : 0.0f;
                en[q][2] += wt * cmid;
                en[q][3] += wc > 1e-20f ? wc * logf(wc) : 0.0f;
                if (a.aux_dim > 0) {
                  const float* ad = a.aux_data + (size_t)(s.bent[k] / (uint32_t)a.n_views) * a.aux_dim;
                  float* aux_px = a.aux + pix[q] * (size_t)(8 + a.aux_dim) + 8;
                  const int n_sh = min(a.aux_dim, kAuxShared);
                  for (int ai = 0; ai < n_sh; ++ai) s.caux[ai * PX + 32 * q + lane] += ta * ad[ai];
                  for (int ai = kAuxShared; ai < a.aux_dim; ++ai) aux_px[ai] += ta * ad[ai];
                }
              }
            }
          }
          __syncwarp();
        }
        // all pixels saturated: the remaining tets would all be skipped
        bool more = false;
#pragma unroll
        for (int q = 0; q < NPX; ++q) more = more || (valid[q] && logT[q] >= -13.8f);
        if (!__any_sync(0xffffffffu, more)) break;
      }
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        if (valid[q] && (MODE == kModeForward || a.rgba != nullptr)) {
          const float A = 1.0f - safe_exp(logT[q]);
          reinterpret_cast<float4*>(a.rgba)[pix[q]] = make_float4(Cr[q], Cg[q], Cb[q], A);
          if constexpr (AUX) {
          if (a.aux_dim == 0) {
            reinterpret_cast<float4*>(a.aux)[2 * pix[q]] = make_float4(nd[q][0], nd[q][1], nd[q][2], nd[q][3]);
            reinterpret_cast<float4*>(a.aux)[2 * pix[q] + 1] = make_float4(en[q][0], en[q][1], en[q][2], en[q][3]);
          } else {  // [normal.xyz, depth, entropy.4, custom...] (:486-500)
            float* o = a.aux + pix[q] * (size_t)(8 + a.aux_dim);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              o[i] = nd[q][i];
              o[4 + i] = en[q][i];
            }
            for (int ai = 0; ai < min(a.aux_dim, kAuxShared); ++ai) o[8 + ai] = s.caux[ai * PX + 32 * q + lane];
          }
          }
        }
      }
    }

    // =============== error statistics (front to back) ===============
    // crates/rmesh-error/src/wgsl/error_tiled_compute.wgsl:90-373: the forward's
    // walk with a -5.5 log-transmittance cut; each covered pixel with T >= 1e-6
    // gives its tet the weight w = T * od.  Phase 1 (per pixel, in order) sets
    // the item to (w, 1); phase 2 sums per tet (w, w pe, w pe^2, w se,
    // w entry, w exit, count, max 65535 w); error_finalize_kernel spreads the sums
    // to tet_err / tet_count.
    if (MODE == kModeError) {
      bool alive[NPX];
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        alive[q] = valid[q];
        if (32 * q + lane < PX)
          s.pdl[32 * q + lane] = valid[q] ? make_float2(a.pixel_err[pix[q]], a.ssim_err[pix[q]]) : make_float2(0.f, 0.f);
      }
      start_list(true);
      while (true) {
        const int nb = next_batch(true);
        if (nb == 0) break;
        for (int base = 0; base < n_runs; base += 32) {
          take_runs(base);
          phase0(std::true_type{});
          __syncwarp();
#pragma unroll
          for (int q = 0; q < NPX; ++q) {
            uint32_t m = take_tets(q, base, alive[q]);
            while (m) {
              if (logT[q] < -5.5f) break;
              const int k = __ffs(m) - 1;
              const int slot = slot_of(k, q, base);
              m &= m - 1u;
              const float od = s.a.ex[slot].x;
              if (od < 0.0f) continue;  // ray miss
              const float Tj = exp_fast(clipf(logT[q], -88.0f, kLogMax));
              if (Tj >= 1e-6f) {
                s.a.ex[slot] = make_float2(Tj * od, 1.0f);
                logT[q] -= od;
              }
            }
            if (logT[q] < -5.5f) alive[q] = false;
          }
          __syncwarp();
          // phase 2: the run's sums, then the warp combine
          float acc[kErrMom];
#pragma unroll
          for (int i = 0; i < kErrMom; ++i) acc[i] = 0.0f;
          int count = 0, mx = 0;
          for (int j = 0, slot = lane * R; j < rlen; ++j, ++slot) {
            const float2 st = s.a.ex[slot];
            if (!(st.y > 0.5f)) continue;
            const float2 ix = s.a.tt[slot];
            const int p = (int)(s.pk[slot] >> 5);
            const float w = st.x;
            const float4 d = s.pdir[p];
            const float2 e = s.pdl[p];
            const float ox = camx + d.x * V.min_t, oy = camy + d.y * V.min_t, oz = camz + d.z * V.min_t;
            acc[0] += w;
            acc[1] += w * e.x;
            acc[2] += w * e.x * e.x;
            acc[3] += w * e.y;
            acc[4] += w * (ox + d.x * ix.x); acc[5] += w * (oy + d.y * ix.x); acc[6] += w * (oz + d.z * ix.x);
            acc[7] += w * (ox + d.x * ix.y); acc[8] += w * (oy + d.y * ix.y); acc[9] += w * (oz + d.z * ix.y);
            ++count;
            mx = max(mx, __float2int_rz(65535.0f * w));
          }
          acc[10] = __int_as_float(count);
          acc[11] = __int_as_float(mx);
#pragma unroll
          for (int i = 0; i < kErrMom; ++i) s.red[lane][i] = acc[i];
          __syncwarp();
          combine_error(base, a.mom);
          __syncwarp();
        }
        bool more = false;
#pragma unroll
        for (int q = 0; q < NPX; ++q) more = more || alive[q];
        if (!__any_sync(0xffffffffu, more)) break;  // every pixel below the cut
      }
    }

    // =============== adjoint (back to front) ===============
    if (kAdjoint) {
      float dlogT[NPX];
      float lsum = 0.f;
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        float dlr = 0.f, dlg = 0.f, dlb = 0.f;
        dlogT[q] = 0.0f;
        if (MODE == kModeTrain) {
          if (valid[q]) {
            const float A = 1.0f - safe_exp(logT[q]);
            const float* gt = a.gt_rgb + 3 * pix[q];
            const float er = Cr[q] - gt[0], eg = Cg[q] - gt[1], eb = Cb[q] - gt[2];
            if (a.hp->loss_type == 0) {
              dlr = (er > 0.f ? 1.f : (er < 0.f ? -1.f : 0.f)) / V.n_pixels;
              dlg = (eg > 0.f ? 1.f : (eg < 0.f ? -1.f : 0.f)) / V.n_pixels;
              dlb = (eb > 0.f ? 1.f : (eb < 0.f ? -1.f : 0.f)) / V.n_pixels;
              lsum += fabsf(er) + fabsf(eg) + fabsf(eb);
            } else {
              dlr = 2.0f * er / V.n_pixels;
              dlg = 2.0f * eg / V.n_pixels;
              dlb = 2.0f * eb / V.n_pixels;
              lsum += er * er + eg * eg + eb * eb;
            }
            logT[q] = logf(fmaxf(1.0f - A, 1e-20f));
            dlogT[q] = -0.0f * (1.0f - A);  // the loss has no alpha term (loss_compute.wgsl:71)
          }
        } else if (valid[q]) {
          const float4 img = reinterpret_cast<const float4*>(a.rgba)[pix[q]];
          const float4 dl = reinterpret_cast<const float4*>(a.dl_rgba)[pix[q]];
          logT[q] = logf(fmaxf(1.0f - img.w, 1e-20f));
          dlogT[q] = -dl.w * (1.0f - img.w);
          dlr = dl.x; dlg = dl.y; dlb = dl.z;
        }
        const int p = 32 * q + lane;
        if (p < PX) {
          s.pdir[p].w = dlr;
          s.pdl[p] = make_float2(dlg, dlb);
        }
      }
      if (MODE == kModeTrain) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if (lane == 0) atomicAdd(&a.counters->loss[view], (double)lsum);
      }
      __syncwarp();
      start_list(false);
      while (true) {
        // adjoint: edge crossings only (backward_tiled_compute.wgsl:241-299)
        const int nb = next_batch(false);
        if (nb == 0) break;
        for (int base = 0; base < n_runs; base += 32) {
          take_runs(base);
          phase0(std::false_type{});
          __syncwarp();
          // phase 1: undo each pixel's items farthest first, the lane's pixels
          // together; the item gets (t_prev, d_od_state), with t_prev 0 where it has
          // no gradient, and a ray miss changes nothing
          uint32_t m[NPX], any = 0u;
#pragma unroll
          for (int q = 0; q < NPX; ++q) {
            m[q] = take_tets(q, base, true);
            any |= m[q];
          }
          while (any) {
            any = 0u;
#pragma unroll
            for (int q = 0; q < NPX; ++q) {
              const bool has = m[q] != 0u;
              const int k = (__ffs(m[q]) - 1) & 31;
              const int slot = slot_of(k, q, base);
              m[q] &= m[q] - 1u;
              any |= m[q];
              float2 c = make_float2(-1.0f, 0.0f);
              if (has) c = s.a.ex[slot];
              const bool hit = c.x >= 0.0f;
              const float prev_logT = fminf(logT[q] + c.x, 0.0f);
              const float t_prev = exp_fast(fmaxf(prev_logT, -88.0f));
              logT[q] = hit ? prev_logT : logT[q];
              const bool on = hit && t_prev >= 1e-6f;
              if (has) s.a.ex[slot] = make_float2(on ? t_prev : 0.0f, -dlogT[q]);
              const float next = clipf(dlogT[q] + c.y * t_prev, kMinVal, kMaxVal);
              dlogT[q] = on ? next : dlogT[q];
            }
          }
          __syncwarp();
          // phase 2: per-item adjoint over the run.
          // Vertex gradients enter through moments: for a face (a, b, c) with
          // unflipped normal n, hit h = cam + d t and s = dT / (n.d), the item
          // adds s (a-h) x (c-a) to vertex b, s (a-h) x (a-b) to c and
          // s ((a-h) x (b-c) + n) to a (backward_tiled_compute.wgsl:506-533).
          // The sum over a tet's items needs only S = sum s and P = sum s (h - v0) per
          // face (v0: the tet's first vertex, so that the differences are taken item
          // by item and nothing large cancels in the sums, whatever their order);
          // grad_finalize_kernel rebuilds the vertex gradients from them.  The
          // face sums live in the lane's row of the warp buffer, so the item's
          // entry / exit face is an address (one 16-byte read and write), not a
          // 16-way select; the other 8 sums stay in registers.
          float acc[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
          float4* fac = reinterpret_cast<float4*>(&s.red[lane][0]);
#pragma unroll
          for (int f = 0; f < 4; ++f) fac[f] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (rlen > 0) {
            const float4 cb = s.rec[rk][4], gg = s.rec[rk][5];
            const uint32_t flips = __float_as_uint(gg.w);
            const float4 v0 = s.v0[rk];
            const float rx = V.cam[0] - v0.x, ry = V.cam[1] - v0.y, rz = V.cam[2] - v0.z;
            int slot = lane * R;
#pragma unroll 1
            for (int j = 0; j < rlen; ++j, ++slot) {
              // (t_prev, d_od_state); ray misses and items below the transmittance
              // cut have no positive t_prev
              const float2 st = s.a.ex[slot];
              if (!(st.x > 0.0f)) continue;
              const float2 ix = s.a.tt[slot];
              const uint32_t pk = s.pk[slot];
              const int p = (int)(pk >> 5);
              int fmin = (int)(pk & 7u);
              const int fmax = (int)((pk >> 3) & 3u);
              if (fmin == 4) fmin = 0;  // reference keeps min_face = 0 when no face enters
              const float t_min = ix.x, t_max = ix.y;
              const float t_prev = st.x, d_od_state = st.y;
              const float4 d = s.pdir[p];
              const float2 dgb = s.pdl[p];
              const float dcdt = gg.x * d.x + gg.y * d.y + gg.z * d.z;
              Integral I;
              integrate(cb, dcdt, t_min, t_max, I);
              const float dcpr = clipf(d.w * t_prev, kMinVal, kMaxVal);
              const float dcpg = clipf(dgb.x * t_prev, kMinVal, kMaxVal);
              const float dcpb = clipf(dgb.y * t_prev, kMinVal, kMaxVal);
              const float dseries = -0.5f + I.od * (1.0f / 3.0f + I.od * (-1.0f / 8.0f + I.od * (1.0f / 30.0f)));
              // one quotient (rcp(od)^2 would round twice: rms error 1.05 against 0.64 units
              // of 2^-24 at od 47..87; __fdividef's range scaling costs 1 % of a step)
              const float dph = I.od < 0.02f ? dseries : (I.alpha_t * (I.od + 1.0f) - 1.0f) * rcp_fast(I.od * I.od);
              const float dw0 = dph + I.alpha_t, dw1 = -dph;
              const float d_od_int = dcpr * (I.cer * dw0 + I.csr * dw1) + dcpg * (I.ceg * dw0 + I.csg * dw1) +
                                     dcpb * (I.ceb * dw0 + I.csb * dw1);
              float d_od_aux = 0.0f;
              if constexpr (AUX && MODE == kModeBackward) {
                // the aux channels' own terms: d od += T_prev alpha_t aux_s (d alpha / d od =
                // alpha_t); d a[tet][ai] += dl_aux[pixel][ai] T_prev alpha, below
                // (__expf: this is the one use of exp(-od) to which values below 2^-126,
                // od > 87.3, can matter)
                d_od_aux = t_prev * __expf(-I.od) * s.aux[slot].x;
                s.aux[slot].y = t_prev * (1.0f - I.alpha_t);
              }
              const float d_od = clipf(d_od_state + d_od_int + d_od_aux, kMinVal, kMaxVal);
              const bool active = (I.od_raw >= 1e-8f) && (I.od_raw <= 88.0f);
              const float d_od_raw = active ? d_od : 0.0f;
              const float d_dist = clipf(d_od_raw * cb.w, kMinVal, kMaxVal);
              float d_tmin = -d_dist, d_tmax = d_dist;
              const float dsr = I.csr > 0.f ? dcpr * I.w1 : 0.f, dsg = I.csg > 0.f ? dcpg * I.w1 : 0.f,
                          dsb = I.csb > 0.f ? dcpb * I.w1 : 0.f;
              const float der = I.cer > 0.f ? dcpr * I.w0 : 0.f, deg = I.ceg > 0.f ? dcpg * I.w0 : 0.f,
                          deb = I.ceb > 0.f ? dcpb * I.w0 : 0.f;
              const float dbr = dsr + der, dbg = dsg + deg, dbb = dsb + deb;
              const float ss = dsr + dsg + dsb, se = der + deg + deb;
              // hits relative to v0
              const float3 hi = make_float3(rx + d.x * t_min, ry + d.y * t_min, rz + d.z * t_min);
              const float3 ho = make_float3(rx + d.x * t_max, ry + d.y * t_max, rz + d.z * t_max);
              d_tmin += ss * dcdt;
              d_tmax += se * dcdt;
              acc[0] += clipf(d_od_raw * I.dist, kMinVal, kMaxVal);
              // (|dbr| <= |dcpr| (w0 + w1) is inside the reference's +-1e20 clip)
              acc[1] += dbr;
              acc[2] += dbg;
              acc[3] += dbb;
              acc[4] += dbr + dbg + dbb;
              acc[5] += ss * hi.x + se * ho.x;
              acc[6] += ss * hi.y + se * ho.y;
              acc[7] += ss * hi.z + se * ho.z;
#pragma unroll
              for (int side = 0; side < 2; ++side) {
                const int f = side == 0 ? fmin : fmax;
                const float dt = side == 0 ? d_tmin : d_tmax;
                const float3 h = side == 0 ? hi : ho;
                const float4 nf = s.rec[rk][f];
                const float den = (((flips >> f) & 1u) ? -1.0f : 1.0f) * (nf.x * d.x + nf.y * d.y + nf.z * d.z);
                const float inv_den = fabsf(den) < kTiny ? 1.0f / kTiny : clipf(rcp_fast(den), kMinVal, kMaxVal);
                const float sv = dt * inv_den;
                float4 v = fac[f];
                v.x += sv;
                v.y += sv * h.x;
                v.z += sv * h.y;
                v.w += sv * h.z;
                fac[f] = v;
              }
            }
          }
          if constexpr (AUX && MODE == kModeBackward) {
            // the run's aux data gradient, four channels at a time
            float* dst = a.d_aux + (size_t)(rentry / (uint32_t)a.n_views) * a.aux_dim;
            for (int a0 = 0; a0 < a.aux_dim; a0 += 4) {
              float sum[4] = {0.f, 0.f, 0.f, 0.f};
              for (int j = 0, slot = lane * R; j < rlen; ++j, ++slot) {
                const float wa = s.aux[slot].y;
                const float* dla = a.dl_aux + strip_pixel((int)(s.pk[slot] >> 5)) * (size_t)a.aux_dim + a0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (a0 + i < a.aux_dim) sum[i] += dla[i] * wa;
              }
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (a0 + i < a.aux_dim && sum[i] != 0.0f) atomicAdd(dst + a0 + i, sum[i]);
            }
          }
          __syncwarp();  // every lane has read its items
          {
            float4* sums = reinterpret_cast<float4*>(&s.item[0]) + (kSumCols / 4) * lane;
            sums[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
            sums[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
          }
          __syncwarp();
          combine(base, a.mom);
          __syncwarp();
        }
      }
    }
    if (!a.persistent) break;
  }
}

// Span words of every sorted (tile, tet) pair, one set per rule: a byte per tile
// row (pack_span, row_spans), four rows per 32-bit word, over the rows its tet
// reaches; a strip of the tile kernel reads the word of its rows.  Other rows and
// sentinel slots get empty spans.  Each
// warp takes 32 consecutive pairs; lane l sets up pair l (sorted vertices, edge
// slopes) in shared memory, and the warp's (pair, row) tasks are spread over its
// lanes through a prefix of the row counts, so lanes stay busy whatever the rows
// per tet.  The rows go to shared memory; the owner lane then stores the pair's
// words, each word array coalesced.
//
// The same pass over the keys finds the tiles' [start, end): it restates
// tile_ranges_compute.wgsl:10-45 per view, where the end of a view's last
// non-empty tile is only written when the view had no sentinel slots (in the
// reference the sentinels follow that tile and the idx == count-1 rule never
// fires for it, leaving end = 0 from the clear).  ranges must be zeroed beforehand.
struct PairSpanArgs {
  const ViewParams* views;
  int n_views;
  const uint32_t* keys;              // sorted global tile ids
  const uint32_t* vals;              // the pairs' entry indices (per-view tet records)
  const unsigned long long* n_ptr;   // pair count
  unsigned long long cap;
  const TetView* vis_view;
  uint32_t* spans_fwd;  // word w of pair i at [w * stride + i]
  uint32_t* spans_adj;  // nullptr: a run without an adjoint
  unsigned long long stride;
  uint2* ranges;
  const Counters* counters;
};

__global__ void __launch_bounds__(256) pair_spans_kernel(PairSpanArgs a) {
  __shared__ __align__(16) uint8_t s_fwd[256][4 * kSpanWords];
  __shared__ __align__(16) uint8_t s_adj[256][4 * kSpanWords];
  __shared__ __align__(16) SpanSetup s_set[256];
  static_assert(sizeof(SpanSetup) == 64, "four 16-byte reads");
  const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
  const unsigned long long n = *a.n_ptr < a.cap ? *a.n_ptr : a.cap;
  const bool adjoint = a.spans_adj != nullptr;
  const uint4 empty = make_uint4(kEmptySpans, kEmptySpans, kEmptySpans, kEmptySpans);
  for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < n;
       base += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long p = base + threadIdx.x;
    *reinterpret_cast<uint4*>(s_fwd[threadIdx.x]) = empty;
    *reinterpret_cast<uint4*>(s_adj[threadIdx.x]) = empty;
    SpanSetup st;
    st.valid_cols = 0;
    int r0 = 0, nrows = 0;
    int words = kSpanWords;  // words of the pair's tile size
    const uint32_t key = p < n ? a.keys[p] : kSentinel;
    uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1), next = __shfl_down_sync(0xffffffffu, key, 1);
    if (key != kSentinel) {
      if (lane == 0) prev = p > 0 ? a.keys[p - 1] : kSentinel;
      if (lane == 31) next = p + 1 < n ? a.keys[p + 1] : kSentinel;
      const int view = view_of_tile(a.views, a.n_views, key);
      if (key != prev) a.ranges[key].x = (uint32_t)p;
      if (key != next) {
        const bool last_of_view = next == kSentinel || view_of_tile(a.views, a.n_views, next) != view;
        if (!(last_of_view && a.counters->shortfall[view])) a.ranges[key].y = (uint32_t)(p + 1);
      }
      const ViewParams& V = a.views[view];
      const int TS = V.TS;
      words = (TS + 3) / 4;
      const uint32_t local = key - V.tile_base;
      const uint32_t ty = local / (uint32_t)V.tiles_x, tx = local - ty * (uint32_t)V.tiles_x;
      st.valid_cols = min(TS, V.W - (int)(tx * (uint32_t)TS));
      const int valid_rows = min(TS, V.H - (int)(ty * (uint32_t)TS));
      const TetView* tv = a.vis_view + a.vals[p];
      {  // (a tet with a vertex behind the camera has no pairs)
        const float4 gx4 = __ldg(&tv->px), gy4 = __ldg(&tv->py);
        const float tile_ox = (float)(tx * (uint32_t)TS), tile_oy = (float)(ty * (uint32_t)TS);
        st.x[0] = gx4.x - tile_ox; st.x[1] = gx4.y - tile_ox; st.x[2] = gx4.z - tile_ox; st.x[3] = gx4.w - tile_ox;
        st.y[0] = gy4.x - tile_oy; st.y[1] = gy4.y - tile_oy; st.y[2] = gy4.z - tile_oy; st.y[3] = gy4.w - tile_oy;
        // sorted by y (five compare-exchanges)
        auto cx = [&](int i, int j) {
          if (st.y[j] < st.y[i]) {
            const float ty = st.y[i], tx = st.x[i];
            st.y[i] = st.y[j]; st.x[i] = st.x[j];
            st.y[j] = ty; st.x[j] = tx;
          }
        };
        cx(0, 1); cx(2, 3); cx(0, 2); cx(1, 3); cx(1, 2);
        auto slope = [&](int i, int j) { return __fdividef(st.x[j] - st.x[i], st.y[j] - st.y[i]); };
        st.m01 = slope(0, 1); st.m02 = slope(0, 2); st.m03 = slope(0, 3);
        st.m12 = slope(1, 2); st.m13 = slope(1, 3); st.m23 = slope(2, 3);
        // rows r with floor(ylo) <= r <= floor(yhi), clipped to the image: the
        // only rows the forward's reach rule can accept
        const float flo = fmaxf(floorf(st.y[0]), 0.0f);
        const float fhi = fminf(floorf(st.y[3]), (float)(valid_rows - 1));
        if (flo <= fhi) {
          r0 = (int)flo;
          nrows = (int)fhi - r0 + 1;
        }
      }
    }
    int pre = nrows;  // inclusive prefix of the row counts over the warp's lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += y;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    st.first_row = r0 - (pre - nrows);
    if (nrows > 0) s_set[threadIdx.x] = st;
    __syncwarp();  // the set-ups and the records' empty rows, before any task
    for (int t0 = 0; t0 < total; t0 += 32) {  // warp-uniform trip count
      const int t = t0 + lane;
      int k = 0;  // the lane whose pair owns task t: first inclusive prefix > t
#pragma unroll
      for (int st2 = 16; st2 > 0; st2 >>= 1) {
        const int pv = __shfl_sync(0xffffffffu, pre, k + st2 - 1);
        if (pv <= t) k += st2;
      }
      if (t < total) {
        const SpanSetup q = s_set[wbase + k];
        const int row = q.first_row + t;
        row_spans(q, row, adjoint, s_fwd[wbase + k][row], s_adj[wbase + k][row]);
      }
    }
    __syncwarp();
    if (p < n) {
      const uint32_t* vf = reinterpret_cast<const uint32_t*>(s_fwd[threadIdx.x]);
      const uint32_t* va = reinterpret_cast<const uint32_t*>(s_adj[threadIdx.x]);
      for (int w = 0; w < words; ++w) {
        a.spans_fwd[w * a.stride + p] = vf[w];
        if (adjoint) a.spans_adj[w * a.stride + p] = va[w];
      }
    }
    __syncwarp();  // the stores' reads before the next chunk's rows are reset
  }
}

// Per tet: rebuilds the gradients of every view's moments (see phase 2 of the
// adjoint) and adds their sum to the tet's slot; one thread per tet, no
// atomics.  The colour moments of SH colours stay where sh_backward_kernel
// reads them.
struct GradFinalizeArgs {
  int M;
  int n_views;
  const TetRec* rec;
  const uint32_t* vis_cnt;  // [M * n_views] tiles touched by the entry
  const float* mom;         // [M * n_views][kMom]
  float* grad_slot;         // [M][kGradSlot], accumulated
  int sh;                   // colours come from SH coefficients
};

__global__ void __launch_bounds__(128) grad_finalize_kernel(GradFinalizeArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.M) return;
  float o[kGradSlot];
#pragma unroll
  for (int i = 0; i < kGradSlot; ++i) o[i] = 0.0f;
  bool any = false;
  const TetRec r = a.rec[t];
  const float4 vs[4] = {r.a, r.b, r.c, r.d};
  for (int v = 0; v < a.n_views; ++v) {
    const size_t j = (size_t)t * a.n_views + v;
    if (a.vis_cnt[j] == 0u) continue;
    const float4* m4 = reinterpret_cast<const float4*>(a.mom + j * kMom);
    const float4 fs4[4] = {m4[0], m4[1], m4[2], m4[3]};
    const float4 dc = m4[4], sd = m4[5];
    const bool inner = dc.x != 0.f || dc.y != 0.f || dc.z != 0.f || dc.w != 0.f || sd.x != 0.f || sd.y != 0.f ||
                       sd.z != 0.f || sd.w != 0.f;
    float dv[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) dv[q] = 0.0f;
    bool faces = false;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const float S = fs4[f].x, Px = fs4[f].y, Py = fs4[f].z, Pz = fs4[f].w;
      if (S != 0.0f || Px != 0.0f || Py != 0.0f || Pz != 0.0f) {
        faces = true;
        const int ia = kFacesH[f][0], ib = kFacesH[f][1], ic = kFacesH[f][2];
        const float4 va = vs[ia], vb = vs[ib], vc = vs[ic];
        const float e1x = vc.x - va.x, e1y = vc.y - va.y, e1z = vc.z - va.z;  // c - a
        const float e2x = va.x - vb.x, e2y = va.y - vb.y, e2z = va.z - vb.z;  // a - b
        // the unflipped normal cross(c - a, b - a), rounded as the record's
        const float nx = fs(fm(e1z, e2y), fm(e1y, e2z)), ny = fs(fm(e1x, e2z), fm(e1z, e2x)),
                    nz = fs(fm(e1y, e2x), fm(e1x, e2y));
        // w = sum s (a - h) = (a - v0) S - P
        const float wx = (va.x - r.a.x) * S - Px, wy = (va.y - r.a.y) * S - Py, wz = (va.z - r.a.z) * S - Pz;
        const float bx = wy * e1z - wz * e1y, by = wz * e1x - wx * e1z, bz = wx * e1y - wy * e1x;
        const float cx = wy * e2z - wz * e2y, cy = wz * e2x - wx * e2z, cz = wx * e2y - wy * e2x;
        dv[3 * ia] += nx * S - bx - cx; dv[3 * ia + 1] += ny * S - by - cy; dv[3 * ia + 2] += nz * S - bz - cz;
        dv[3 * ib] += bx; dv[3 * ib + 1] += by; dv[3 * ib + 2] += bz;
        dv[3 * ic] += cx; dv[3 * ic + 1] += cy; dv[3 * ic + 2] += cz;
      }
    }
    if (!inner && !faces) continue;
    any = true;
    const float sb = sd.x;
    o[0] += dc.x;
    if (!a.sh) {
      o[1] += dc.y; o[2] += dc.z; o[3] += dc.w;
    }
    o[4] += clipf(sd.y, kMinVal, kMaxVal);
    o[5] += clipf(sd.z, kMinVal, kMaxVal);
    o[6] += clipf(sd.w, kMinVal, kMaxVal);
    dv[0] -= r.b.w * sb; dv[1] -= r.c.w * sb; dv[2] -= r.d.w * sb;
#pragma unroll
    for (int q = 0; q < 12; ++q) o[7 + q] += clipf(dv[q], kMinVal, kMaxVal);
  }
  if (!any) return;
  float4* dst = reinterpret_cast<float4*>(a.grad_slot + (size_t)t * kGradSlot);
#pragma unroll
  for (int c = 0; c < kGradSlot / 4; ++c) {
    float4 v = dst[c];
    v.x += o[4 * c]; v.y += o[4 * c + 1]; v.z += o[4 * c + 2]; v.w += o[4 * c + 3];
    dst[c] = v;
  }
}

// Per tet: the error statistics (tet_err [M][16], tet_count [M][2]) from the
// error mode's sums.
__global__ void __launch_bounds__(256) error_finalize_kernel(int M, const float* __restrict__ mom,
                                                             const TetRec* __restrict__ rec, float* __restrict__ tet_err,
                                                             int* __restrict__ tet_count) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= M) return;
  const float4* m4 = reinterpret_cast<const float4*>(mom + (size_t)t * kErrMom);
  const float4 a = m4[0], b = m4[1], c = m4[2];  // (w, w pe, w pe^2, w se), (entry, exit.x), (exit.yz, count, max)
  float4* e = reinterpret_cast<float4*>(tet_err + 16 * (size_t)t);
  const TetRec r = rec[t];
  const float cx = (r.a.x + r.b.x + r.c.x + r.d.x) * 0.25f, cy = (r.a.y + r.b.y + r.c.y + r.d.y) * 0.25f,
              cz = (r.a.z + r.b.z + r.c.z + r.d.z) * 0.25f;
  const int count = __float_as_int(c.z);
  const bool some = count != 0;
  e[0] = make_float4(a.x, a.y, a.z, 0.0f);
  e[1] = make_float4(0.0f, a.w, b.x, b.y);
  e[2] = make_float4(b.z, b.w, c.x, c.y);
  e[3] = some ? make_float4(a.x, a.x * cx, a.x * cy, a.x * cz) : make_float4(0.f, 0.f, 0.f, 0.f);
  tet_count[2 * (size_t)t] = count;
  tet_count[2 * (size_t)t + 1] = __float_as_int(c.w);
}

}  // namespace rm

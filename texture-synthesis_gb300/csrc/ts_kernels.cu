// ts_kernels.cu — sm_103a kernels of the texture-synthesis hot loop.
//
// One batch step of a synthesis stage is five parts, a launch each where the
// step makes its own neighbour lists; with the lists made ahead, a chunk of
// steps at a time on other streams (k_tree_append, then knn_list or knn_walk,
// knn_exhaustive and mean_ahead), the step is its resolve launch alone:
//   knn_walk        warp per work item: the k nearest resolved points under
//                   the (d2, y, x) order, by walking a table of lattice offsets
//                   sorted in that order and testing a resolved-point bitmap
//                   (replaces TreeGrid::get_k_nearest_neighbors, ms.rs:1363-1530)
//   knn_exhaustive  CTA per item the walk could not finish (sparse regions):
//                   radix-select over the resolved list
//   mean            thread per item: the mean of the 4x-duplicated distance
//                   list (ms.rs:417-423), the in-order f64 sum, one item per
//                   lane (large batches); for whole small batches the
//                   exhaustive k-NN computes it on one thread
//   resolve         warp per item (a CTA in small steps): neighbour weights (ms.rs:1198-1203) in
//                   double-f32 arithmetic with an exact f64 fallback,
//                   coherence + random candidates (ms.rs:478-602), own
//                   pattern (ms.rs:1151-1181), candidate cost and first-min
//                   argmin (ms.rs:1184-1288), lanes over candidates
// The k-NN kernels also write each neighbour's exact squared normalised
// distance (ms.rs:410-415), one f64 fused multiply-add from per-pixel tables.
//   commit          thread per item: update + flush_resolved (ms.rs:296-377)
// Every item of a batch reads the state as it was when the batch started;
// commit runs after all of them.  Per stage, random_candidates precomputes the
// m random candidates of every item (they depend only on the seed), and
// level_switch recolours the resolved pixels (ms.rs:687-700).
//
// Floating point follows the reference operation by operation: f32 sums are
// sequential, multiplies and adds are never fused (the file is compiled with
// --fmad=false and uses __fadd_rn/__fmul_rn where it matters), and the f64
// distances use an explicit fused multiply-add exactly where ms.rs:415 calls
// mul_add.
#include <float.h>
#include <stdint.h>

#include <cuda_pipeline.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "tsgpu.h"
#include "ts_common.h"
#include "ts_kernels.cuh"

namespace ts {

namespace {

constexpr int kWarp = 32;
constexpr int kResolveWarps = 4;
constexpr int kWalkWarps = 8;
constexpr int kExhThreads = 256;
constexpr int kTeamThreads = 128;
constexpr int kTeamFullThreads = 256;  // the full-evaluation form: batches of at most ~1000 items
constexpr int kStepWideThreads = 512;  // the fused small-step kernel on steps of at most one item per SM
constexpr int kExhCap = 2048;      // keys kept by the exhaustive k-NN at the cut distance
constexpr int kExhAllKeys = 8192;  // keys the exhaustive k-NN sorts in shared memory directly
constexpr int kExhSortAll = 256;   // at most this many keys are sorted without a select
constexpr uint32_t kMaxDraws = TS_MAX_SAMPLE_DRAWS;  // (x, y) pairs per random candidate
constexpr uint32_t kRcandFailed = 0x7fffu;              // map field of a random candidate whose draws ran out

__device__ const double g_exp2_64[64] = {TS_EXP2_TABLE_VALUES};
__device__ const float g_exp2_ff[128] = {TS_EXP2_FF_TABLE_VALUES};

__device__ __forceinline__ void set_err(int *err, int code) {
  if (*err == 0) atomicCAS(err, 0, code);
}

__device__ __forceinline__ int off_dx(int32_t off) { return (int)(int16_t)(off & 0xffff); }
__device__ __forceinline__ int off_dy(int32_t off) { return off >> 16; }
__device__ __forceinline__ int32_t pack_off(int dx, int dy) { return (int32_t)((uint32_t)(dx & 0xffff) | ((uint32_t)dy << 16)); }

// a in [-n, 2n) wrapped into [0, n): every tree point and its tiling mirrors
// lie there (the mirror bands are 5% of a side).
__device__ __forceinline__ int wrap1(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// (x, y) of a pixel index below 2^28: y = p / W by the host's multiplier
// (SessionDev::w_mul, exact), not an integer division.
__device__ __forceinline__ void pixel_xy(const SessionDev &s, uint32_t p, int &x, int &y) {
  const uint32_t q = (uint32_t)(((uint64_t)p * s.w_mul) >> s.w_sh);
  y = (int)q;
  x = (int)(p - q * s.W);
}

// Tree membership of an output-plane point, tiling mirrors included
// (flush_resolved, ms.rs:296-331).
__device__ __forceinline__ bool occupied(const SessionDev &s, int x, int y) {
  const bool inx = (unsigned)x < s.W, iny = (unsigned)y < s.H;
  if (inx && iny) return (__ldg(&s.occ[(size_t)y * s.wpr + (x >> 5)]) >> (x & 31)) & 1u;
  if (!s.tiling || (!inx && !iny)) return false;
  int xs = x, ys = y;
  if (!inx) {
    if (x >= (int)s.W) {
      xs = x - (int)s.W;
      if (xs >= s.x_l) return false;
    } else {
      xs = x + (int)s.W;
      if (xs < 0 || xs <= s.x_r) return false;
    }
  } else {
    if (y >= (int)s.H) {
      ys = y - (int)s.H;
      if (ys >= s.y_b) return false;
    } else {
      ys = y + (int)s.H;
      if (ys < 0 || ys <= s.y_t) return false;
    }
  }
  return (__ldg(&s.mir[(size_t)ys * s.wpr + (xs >> 5)]) >> (xs & 31)) & 1u;
}

// Whether pixel p is in a tree of n points (SessionDev::rank); always true
// when the bitmap is the tree itself.
__device__ __forceinline__ bool in_tree(const SessionDev &s, uint32_t p, uint32_t n) {
  return !s.rank || __ldg(&s.rank[p]) - 1u < n;
}

// occupied() against the tree of an item whose batch starts with n points:
// with SessionDev::rank the bitmap may hold later points too, so a set bit
// is checked against the tree position of the pixel it stands for.
__device__ __forceinline__ bool occupied_n(const SessionDev &s, int x, int y, uint32_t n) {
  if (!occupied(s, x, y)) return false;
  if (!s.rank) return true;
  const int xs = wrap1(x, (int)s.W), ys = wrap1(y, (int)s.H);  // a mirror stands for its wrapped pixel
  return in_tree(s, (uint32_t)ys * s.W + (uint32_t)xs, n);
}

// Resolved-list length at the start of the batch of stage item `item`
// (BatchDev::btab), else the launch's own.
__device__ __forceinline__ uint32_t item_nres(const BatchDev &b, uint32_t item) {
  if (!b.btab) return b.n_res;
  uint32_t lo = 0, hi = b.nbt;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&b.btab[mid].x) <= item)
      lo = mid;
    else
      hi = mid;
  }
  return __ldg(&b.btab[lo].y);
}

__device__ __forceinline__ bool mir_bit(const SessionDev &s, uint32_t x, uint32_t y) {
  return (s.mir[(size_t)y * s.wpr + (x >> 5)] >> (x & 31)) & 1u;
}

// check_coord_validity (ms.rs:1534-1549)
__device__ __forceinline__ bool coord_valid(const SessionDev &s, const MapDesc &md, int x, int y) {
  if (x < 0 || y < 0 || x >= (int)md.w || y >= (int)md.h) return false;
  if (md.mask_off < 0) return true;
  return __ldg(&s.masks[md.mask_off + (size_t)y * md.w + x]) != 0;
}

// ---------------------------------------------------------------------------
// Random candidates of every item of a stage (ms.rs:549-599): the stream is
// Pcg32::seed_from_u64(stage_seed + item + 1); per candidate a map
// (usize range), then (x, y) redrawn until valid.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void random_candidates_body(const SessionDev &s, const StageDev &st, uint32_t vb) {
  const uint32_t item = vb * blockDim.x + threadIdx.x;
  if (item >= st.n_items) return;
  Pcg32 g = pcg_from_u64(st.stage_seed + (uint64_t)item + 1ULL);
  uint2 *out = st.rcand + (size_t)item * s.m;
  for (uint32_t t = 0; t < s.m; ++t) {
    uint64_t map64 = 0;
    bool ok = gen_range_u64_bounded(g, s.n_maps, 256, map64);
    const uint32_t map = ok ? (uint32_t)map64 : 0u;
    const MapDesc md = s.maps[map];
    uint32_t x = 0, y = 0;
    if (ok) {
      ok = false;
      for (uint32_t tries = 0; tries < kMaxDraws; ++tries) {
        if (!gen_range_u32_bounded(g, md.w, 256, x) || !gen_range_u32_bounded(g, md.h, 256, y)) break;
        if (coord_valid(s, md, (int)x, (int)y)) {
          ok = true;
          break;
        }
      }
    }
    if (!ok) {
      // Only an item with resolved neighbours uses its random candidates
      // (an item without any resolves at random, ms.rs:1002-1010), so the
      // failure is left for the resolve kernel to report when it reads one.
      for (; t < s.m; ++t) out[t] = make_uint2(0u, kRcandFailed);
      return;
    }
    out[t] = make_uint2(x | (y << 16), map);
  }
}

// A random candidate as the resolve kernels store it: {x | y<<16, map}.  A
// failed draw (kRcandFailed) reports TS_ERR_NO_VALID_SAMPLE and is replaced
// by texel (0, 0) of map 0, so that nothing reads past the map table; the
// run's result is discarded.
__device__ __forceinline__ uint2 use_rcand(const SessionDev &s, uint2 v) {
  if (v.y == kRcandFailed) {
    set_err(s.err, kDevErrNoSample);
    v = make_uint2(0u, 0u);
  }
  return v;
}

// Exact squared normalised distance of a neighbour at offset (dx, dy).
__device__ __forceinline__ double neighbour_dist(const SessionDev &s, int px, int py, int dx, int dy) {
  const int R = s.dtab_r;
  if (dx >= -R && dx <= R && dy >= -R && dy <= R) {
    const double ddx = __ldg(&s.dxt[(size_t)px * (2 * R + 1) + dx + R]);
    return __fma_rn(ddx, ddx, __ldg(&s.dy2t[(size_t)py * (2 * R + 1) + dy + R]));
  }
  const double ddx = __dsub_rn(__ldg(&s.xdiv[px + dx + s.xdiv_off]), __ldg(&s.xdiv[px + s.xdiv_off]));
  const double ddy = __dsub_rn(__ldg(&s.ydiv[py + dy + s.ydiv_off]), __ldg(&s.ydiv[py + s.ydiv_off]));
  return __fma_rn(ddx, ddx, __dmul_rn(ddy, ddy));
}

// The same from the per-pixel tables only, for offsets within their radius
// (every offset the walk's table holds): one f64 instruction, and no
// predicated far-offset path beside it.
__device__ __forceinline__ double neighbour_dist_near(const SessionDev &s, int px, int py, int dx, int dy) {
  const int R = s.dtab_r;
  const double ddx = __ldg(&s.dxt[(size_t)px * (2 * R + 1) + dx + R]);
  return __fma_rn(ddx, ddx, __ldg(&s.dy2t[(size_t)py * (2 * R + 1) + dy + R]));
}

// ---------------------------------------------------------------------------
// The mean of a distance list whose sums are exact (SessionDev::exact_sum):
// the in-order sum of the 4x-duplicated list (ms.rs:417-421) never rounds,
// so it equals 4 * (the list's sum in any order of exact adds), and the mean
// is that divided by 4n, rounded once, as the reference divides.
// ---------------------------------------------------------------------------
// A neighbour's distance in units of SessionDev::exact_q: an integer (the
// distances are exact), summed in integers instead of f64 adds.
__device__ __forceinline__ unsigned long long exact_units(const SessionDev &s, int dx, int dy) {
  return ((unsigned long long)(uint32_t)(dx * dx) << s.exact_sx) + ((unsigned long long)(uint32_t)(dy * dy) << s.exact_sy);
}
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ unsigned long long warp_sum_units(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// A neighbour's distance from its packed offset, for sessions with exact
// sums: its units, converted (exact below 2^53) and scaled by the power of
// two exact_q, equal fma(dx, dx, dy * dy) of get_distances_to_k_neighs
// (ms.rs:405-425) bit for bit.
__device__ __forceinline__ double exact_dist(const SessionDev &s, int32_t off) {
  return __dmul_rn(__ull2double_rn(exact_units(s, off_dx(off), off_dy(off))), s.exact_q);
}
// The mean from the list's sum in units: below 2^53, so its conversion and
// the scaling by the power of two exact_q are exact; 4 * that is the
// reference's in-order sum, divided by 4n and rounded once.
// Integer arithmetic only (ts_units_bits, ts_div_int_rn): GB300's FP64 pipe
// is narrow, and an f64 division takes it for a whole warp.
__device__ __forceinline__ double exact_mean(const SessionDev &s, unsigned long long units, uint32_t n) {
  return bits_dbl(ts_div_int_rn(ts_units_bits(units, s.exact_qe), n));
}

__device__ __forceinline__ unsigned long long nb_key(uint32_t d2, int x, int y) {
  return ((unsigned long long)d2 << 32) | ((uint32_t)(y + 32768) << 16) | (uint32_t)(x + 32768);
}

// ---------------------------------------------------------------------------
// k-NN by walking the sorted offset table.  The table holds every lattice
// offset with d2 <= its radius^2, in (d2, dy, dx) order, so the first k
// occupied entries are exactly the k nearest points under the tie rule.
// Items for which the table holds fewer than k points (sparse steps, image
// edges) go to the exhaustive k-NN; sparse steps send every item there.
// ---------------------------------------------------------------------------
// Walk window: the bitmap square [-R, R]^2 around an item (R the table
// radius), kWinWords 32-bit words per row, bit i of word w of row r = point
// (px - R + 32w + i, py - R + r).
constexpr int kWinRows = 2 * kKnnTabRadius + 1;
constexpr int kWinWords = (2 * kKnnTabRadius + 1 + 31) / 32;
constexpr uint32_t kWalkDirect = 128;  // expected entries still to scan above which the window is built

// Bits of bitmap row `row` for x in [x0, x0 + 32) (bit i = x0 + i), zero
// outside [0, W).
__device__ __forceinline__ uint32_t row_bits(const uint32_t *row, int x0, const SessionDev &s) {
  const int W = (int)s.W;
  if (x0 >= W || x0 + 32 <= 0) return 0u;
  const int q = x0 >> 5, sh = x0 & 31;  // floor division
  const uint32_t lo = (q >= 0 && q < (int)s.wpr) ? __ldg(&row[q]) : 0u;
  const uint32_t hi = (sh && q + 1 >= 0 && q + 1 < (int)s.wpr) ? __ldg(&row[q + 1]) : 0u;
  uint32_t v = sh ? (lo >> sh) | (hi << (32 - sh)) : lo;
  if (x0 < 0) v &= ~0u << (-x0);
  if (x0 + 32 > W) v &= (1u << (W - x0)) - 1u;
  return v;
}

// Bits i with lo <= i < hi of a 32-bit word (lo, hi clamped to [0, 32]).
__device__ __forceinline__ uint32_t bit_range(int lo, int hi) {
  lo = max(lo, 0);
  hi = min(hi, 32);
  if (hi <= lo) return 0u;
  const uint32_t upto_hi = hi >= 32 ? ~0u : ((1u << hi) - 1u);
  return upto_hi & (~0u << lo);
}

// occupied() for the 32 points (x0 + i, y), i = 0..31, as a word.
__device__ __forceinline__ uint32_t window_word(const SessionDev &s, int x0, int y) {
  const int W = (int)s.W, H = (int)s.H;
  if ((unsigned)y < s.H) {
    uint32_t v = row_bits(s.occ + (size_t)y * s.wpr, x0, s);
    if (s.tiling) {
      const uint32_t *mr = s.mir + (size_t)y * s.wpr;
      // x >= W: mirror of xs = x - W when xs < x_l
      v |= row_bits(mr, x0 - W, s) & bit_range(0, s.x_l - (x0 - W));
      // x < 0: mirror of xs = x + W when xs > x_r
      v |= row_bits(mr, x0 + W, s) & bit_range(s.x_r + 1 - (x0 + W), 32);
    }
    return v;
  }
  if (!s.tiling) return 0u;
  if (y >= H) {
    const int ys = y - H;
    return ys < s.y_b ? row_bits(s.mir + (size_t)ys * s.wpr, x0, s) : 0u;
  }
  const int ys = y + H;
  return (ys >= 0 && ys > s.y_t) ? row_bits(s.mir + (size_t)ys * s.wpr, x0, s) : 0u;
}

// Bound on |dx| and |dy| of the first c table entries: a disc of radius r holds
// at least pi (r - 0.71)^2 lattice points.
__device__ __forceinline__ int walk_reach(uint32_t c) {
  return min(kKnnTabRadius, (int)(sqrtf((float)c * 0.31830989f) + 0.71f) + 1);
}

constexpr int kWalkPend = 3 * kWarp;  // hits of a window walk waiting for their tree check
constexpr size_t kWalkWinBytes = (size_t)kWalkWarps * (kWinRows * kWinWords + kWalkPend) * 4;  // dynamic shared memory
// A warp takes a run of consecutive items (as many as spread the launch over
// its warps, at most 32): their pixels are one load, their batch follows from
// the one before, and their means are divided together at the end, one per
// lane (the 64-bit integer division is some 300 instructions, whatever the
// active lanes).  A round looks 64 table entries up, two per lane.  Items
// whose round stays inside the image, nearly all of them, need no bounds or
// wrapping: with the k-NN made ahead one load and one comparison of the tree
// position per entry, else one bitmap word.  The last stage of a 2048^2 output
// (2^22 items, beside its resolves): 11.6 -> 6.3 ms.
//
// kWin: launches of small (latency-bound) steps, or of a chunk that begins
// with one, whose sparse items switch to a window in dynamic shared memory
// (kWalkWinBytes) once the hits so far say more than two further rounds are
// needed.  With the k-NN made ahead the
// window holds later points too: its hits wait in a list and are checked 32
// at a time, so that a round without a full list waits for no load.
template <bool kWin>
__device__ __forceinline__ void knn_walk_body(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t vb,
                                              uint32_t vg) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t nb = b.i1 - b.i0, warps = vg * kWalkWarps;
  const uint32_t per = min(32u, (nb + warps - 1) / warps);
  const uint32_t tab_n = b.grid_first ? 0u : s.knn_tab_n;
  const bool ahead = s.rank != nullptr;
  int32_t head[4];  // the first two rounds' entries
#pragma unroll
  for (int u = 0; u < 4; ++u) head[u] = (uint32_t)(u * kWarp + lane) < tab_n ? __ldg(&s.knn_tab[u * kWarp + lane]) : 0;
  for (uint32_t base = (vb * kWalkWarps + (threadIdx.x >> 5)) * per; base < nb; base += warps * per) {
    const uint32_t n = min(per, nb - base);
    const uint32_t pixels = (uint32_t)lane < n ? st.items[b.i0 + base + lane] : 0u;
    uint64_t my_units = 0;  // lane q: the units of item base + q, when its list is complete
    bool mine = false;
    uint32_t n_tree = b.n_res, bt = 0, bt_end = 0xffffffffu;  // item base + q's tree, its batch, the batch's last item + 1
    if (b.btab) {
      uint32_t hi = b.nbt;
      while (hi - bt > 1) {
        const uint32_t mid = (bt + hi) >> 1;
        if (__ldg(&b.btab[mid].x) <= b.i0 + base)
          bt = mid;
        else
          hi = mid;
      }
      n_tree = __ldg(&b.btab[bt].y);
      bt_end = bt + 1 < b.nbt ? __ldg(&b.btab[bt + 1].x) : 0xffffffffu;
    }
    for (uint32_t q = 0; q < n; ++q) {
      const uint32_t local = base + q, pixel = __shfl_sync(0xffffffffu, pixels, q);
      while (b.i0 + local >= bt_end) {
        ++bt;
        n_tree = __ldg(&b.btab[bt].y);
        bt_end = bt + 1 < b.nbt ? __ldg(&b.btab[bt + 1].x) : 0xffffffffu;
      }
      int px, py;
      pixel_xy(s, pixel, px, py);
      int32_t *nbo = b.nbuf + (size_t)local * s.k;
      uint32_t count = 0, ux = 0, uy = 0;  // hits; the sums of dx^2 and dy^2 over this lane's kept hits
      auto keep = [&](bool h, uint32_t r, int32_t o) {
        if (h && r < s.k) {
          nbo[r] = o;
          ux += (uint32_t)(off_dx(o) * off_dx(o));
          uy += (uint32_t)(off_dy(o) * off_dy(o));
        }
      };
      auto take = [&](bool h0, bool h1, int32_t o0, int32_t o1) {
        const uint32_t b0 = __ballot_sync(0xffffffffu, h0), b1 = __ballot_sync(0xffffffffu, h1);
        keep(h0, count + __popc(b0 & lt), o0);
        keep(h1, count + __popc(b0) + __popc(b1 & lt), o1);
        count += __popc(b0) + __popc(b1);
      };
      // rounds look the tree up directly while the hits so far say that two
      // more rounds or fewer will do (dense steps end here)
      uint32_t c = 0;
      while (c < tab_n) {
        const uint32_t i0 = c + lane, i1 = i0 + kWarp;
        const bool on0 = i0 < tab_n, on1 = i1 < tab_n;
        const int32_t o0 = c == 0 ? head[0] : (c == 2 * kWarp ? head[2] : (on0 ? __ldg(&s.knn_tab[i0]) : 0));
        const int32_t o1 = c == 0 ? head[1] : (c == 2 * kWarp ? head[3] : (on1 ? __ldg(&s.knn_tab[i1]) : 0));
        const int reach = walk_reach(c + 2 * kWarp);
        const bool inside = px >= reach && py >= reach && px + reach < (int)s.W && py + reach < (int)s.H;
        bool h0, h1;
        if (inside) {
          if (ahead) {
            const uint32_t r0 = __ldg(&s.rank[pixel + (uint32_t)(off_dy(o0) * (int)s.W + off_dx(o0))]);
            const uint32_t r1 = __ldg(&s.rank[pixel + (uint32_t)(off_dy(o1) * (int)s.W + off_dx(o1))]);
            h0 = on0 && r0 - 1u < n_tree;
            h1 = on1 && r1 - 1u < n_tree;
          } else {
            const int x0 = px + off_dx(o0), x1 = px + off_dx(o1);
            const uint32_t w0 = __ldg(&s.occ[(uint32_t)(py + off_dy(o0)) * s.wpr + (uint32_t)(x0 >> 5)]);
            const uint32_t w1 = __ldg(&s.occ[(uint32_t)(py + off_dy(o1)) * s.wpr + (uint32_t)(x1 >> 5)]);
            h0 = on0 && ((w0 >> (x0 & 31)) & 1u);
            h1 = on1 && ((w1 >> (x1 & 31)) & 1u);
          }
        } else {
          h0 = on0 && occupied_n(s, px + off_dx(o0), py + off_dy(o0), n_tree);
          h1 = on1 && occupied_n(s, px + off_dx(o1), py + off_dy(o1), n_tree);
        }
        take(h0, h1, o0, o1);
        c += 2 * kWarp;
        if (count >= s.k) break;
        if (kWin && (count == 0 || (uint64_t)(s.k - count) * c > (uint64_t)count * kWalkDirect)) break;
      }
      if (kWin && count < s.k && c < tab_n) {
        // sparse: the membership bits of the whole table's square, built in
        // one pass of independent loads, then the rest of the walk from
        // shared memory
        extern __shared__ uint32_t walk_win[];
        uint32_t *win = walk_win + (threadIdx.x >> 5) * (kWinRows * kWinWords + kWalkPend);
        int32_t *pend = (int32_t *)(win + kWinRows * kWinWords);
        uint32_t n_pend = 0;
        for (uint32_t wi = lane; wi < kWinRows * kWinWords; wi += kWarp) {
          const int row = (int)(wi / kWinWords), word = (int)(wi - row * kWinWords);
          win[wi] = window_word(s, px - kKnnTabRadius + 32 * word, py - kKnnTabRadius + row);
        }
        __syncwarp();
        auto bit = [&](int32_t o) {
          const int i = off_dx(o) + kKnnTabRadius;
          return ((win[(off_dy(o) + kKnnTabRadius) * kWinWords + (i >> 5)] >> (i & 31)) & 1u) != 0u;
        };
        // the first 32 waiting hits (or all, at the end) against the tree
        auto check = [&]() {
          const bool on = (uint32_t)lane < n_pend;
          const int32_t o = on ? pend[lane] : 0;
          const uint32_t p = (uint32_t)wrap1(py + off_dy(o), (int)s.H) * s.W + (uint32_t)wrap1(px + off_dx(o), (int)s.W);
          const bool h = on && __ldg(&s.rank[p]) - 1u < n_tree;
          const uint32_t bal = __ballot_sync(0xffffffffu, h);
          keep(h, count + __popc(bal & lt), o);
          count += __popc(bal);
          const int32_t m0 = pend[kWarp + lane], m1 = pend[2 * kWarp + lane];
          __syncwarp();
          pend[lane] = m0;
          pend[kWarp + lane] = m1;
          n_pend -= min(n_pend, (uint32_t)kWarp);
          __syncwarp();
        };
        for (; c < tab_n && count < s.k; c += 2 * kWarp) {
          const uint32_t i0 = c + lane, i1 = i0 + kWarp;
          const int32_t o0 = i0 < tab_n ? __ldg(&s.knn_tab[i0]) : 0, o1 = i1 < tab_n ? __ldg(&s.knn_tab[i1]) : 0;
          const bool h0 = i0 < tab_n && bit(o0), h1 = i1 < tab_n && bit(o1);
          if (!ahead) {
            take(h0, h1, o0, o1);
            continue;
          }
          const uint32_t b0 = __ballot_sync(0xffffffffu, h0), b1 = __ballot_sync(0xffffffffu, h1);
          if (h0) pend[n_pend + __popc(b0 & lt)] = o0;
          if (h1) pend[n_pend + __popc(b0) + __popc(b1 & lt)] = o1;
          n_pend += __popc(b0) + __popc(b1);
          __syncwarp();
          while (n_pend >= kWarp && count < s.k) check();
        }
        while (n_pend && count < s.k) check();
        __syncwarp();  // the window is rebuilt for the warp's next item
      }
      if (count >= s.k) {
        if (s.exact_sum) {
          // (sessions with exact sums store no distances: the resolve derives
          // each one from its offset, exact_dist)
          const uint64_t units = ((uint64_t)__reduce_add_sync(0xffffffffu, ux) << s.exact_sx) +
                                 ((uint64_t)__reduce_add_sync(0xffffffffu, uy) << s.exact_sy);
          if ((uint32_t)lane == q) {
            my_units = units;
            mine = true;
          }
        } else if (b.dist) {
          // the distances once the k offsets are known, 32 per f64 warp
          // instruction (lists made ahead leave them to k_mean_ahead and the
          // resolve)
          __syncwarp();
          for (uint32_t j = lane; j < s.k; j += kWarp) {
            const int32_t o = nbo[j];
            b.dist[(size_t)j * nb + local] = neighbour_dist_near(s, px, py, off_dx(o), off_dy(o));
          }
        }
      }
      if (lane == 0) {
        if (count >= s.k)
          b.ncnt[local] = s.k;
        else
          b.fb_list[atomicAdd(b.fb_count, 1u)] = local;
      }
    }
    if (mine) b.mean[base + lane] = exact_mean(s, my_units, s.k);
  }
}

// ---------------------------------------------------------------------------
// Exhaustive k-NN (one CTA per item): radix-select the k-th smallest d2 over
// every resolved point and its mirrors, keep the points at or below it, sort
// them by (d2, y, x) and emit the first k.
// ---------------------------------------------------------------------------
// The mean of a neighbour distance list on one thread (ms.rs:417-423, as
// k_mean_staged computes it): the 4n-long chain of f64 adds in order, then
// / (4n).  Where one thread runs it alone this is shorter than the integer
// form of the four adds (ts_add4_fast): 14.1k against 16.8k cycles for
// n = 50 on GB300.
__device__ __forceinline__ double mean_chain(const double *d, uint32_t n) {
  double sum = 0.0;
  for (uint32_t i = 0; i < n; ++i) {
    const double v = d[i];
    sum = __dadd_rn(sum, v);
    sum = __dadd_rn(sum, v);
    sum = __dadd_rn(sum, v);
    sum = __dadd_rn(sum, v);
  }
  return __ddiv_rn(sum, (double)(n * 4u));
}

struct ExhShared {
  double dist[256];  // the item's neighbour distances, when the kernel also computes the mean
  unsigned long long wsum[16];  // per-warp distance sums in units (SessionDev::exact_sum), up to 512 threads
  int32_t nbo[256];  // and their offsets
  uint32_t hist[256];
  unsigned long long keys[kExhCap];
  uint32_t nkeys;
  uint32_t total;
  uint32_t prefix;
  uint32_t rank;
  int overflow;
  uint32_t flag, cnt;  // cell-grid search: a ring cell lies in the grid; keys below the bound
  uint32_t below, le;  // select: keys below the selected digit's range; at or below it
};

constexpr uint32_t kExhGridFrom = 4096;  // resolved points from which the cell grid is searched

__device__ __forceinline__ void ring_cell(int r, int i, int &dx, int &dy) {
  if (r == 0) {
    dx = dy = 0;
  } else if (i < 2 * r + 1) {
    dx = -r + i;
    dy = -r;
  } else if (i < 4 * r + 2) {
    dx = -r + (i - (2 * r + 1));
    dy = r;
  } else if (i < 6 * r + 1) {
    dx = -r;
    dy = -r + 1 + (i - (4 * r + 2));
  } else {
    dx = r;
    dy = -r + 1 + (i - (6 * r + 1));
  }
}

template <typename F>
__device__ __forceinline__ void for_points(const SessionDev &s, uint32_t n_res, F &&f) {
  for (uint32_t e = threadIdx.x; e < n_res; e += blockDim.x) {
    const uint32_t p = s.resolved[e];
    const int x = (int)(p % s.W), y = (int)(p / s.W);
    f(x, y);
    if (s.tiling && mir_bit(s, (uint32_t)x, (uint32_t)y)) {
      if (x < s.x_l)
        f(x + (int)s.W, y);
      else if (x > s.x_r)
        f(x - (int)s.W, y);
      if (y < s.y_b)
        f(x, y + (int)s.H);
      else if (y > s.y_t)
        f(x, y - (int)s.H);
    }
  }
}

__device__ uint32_t knn_exhaustive_item(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                        ExhShared &sh, unsigned long long *all, uint32_t cap, bool with_mean,
                                        bool use_grid = true, bool mean_here = true);

// One CTA per item.  `all` (dynamic shared memory, kExhAllKeys entries)
// receives every point's key in one pass over the resolved list; when they
// fit, a bitonic sort of them gives the answer directly, otherwise a
// radix select over further passes finds the cut distance first.
__device__ __forceinline__ void knn_exhaustive_body(const SessionDev &s, const StageDev &st, const BatchDev &b,
                                                    int all_items, uint32_t cap, uint32_t vb, uint32_t vg,
                                                    bool use_grid = true) {
  __shared__ ExhShared sh;
  extern __shared__ unsigned long long all_keys[];
  const uint32_t n = all_items ? b.i1 - b.i0 : *b.fb_count;
  for (uint32_t e = vb; e < n; e += vg) {
    const uint32_t local = all_items ? e : b.fb_list[e];
    knn_exhaustive_item(s, st, b, local, sh, all_keys, cap, all_items != 0, use_grid);
    __syncthreads();
  }
}

// Bitonic sort of keys[0, np2) ascending (np2 a power of two), whole CTA.
__device__ __forceinline__ void block_bitonic(unsigned long long *keys, uint32_t np2) {
  for (uint32_t size = 2; size <= np2; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) {
        const uint32_t j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const unsigned long long a = keys[i], c = keys[j];
          if ((a > c) == up) {
            keys[i] = c;
            keys[j] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

// The first `nout` of the n distinct keys in keys[] in ascending order.
// Up to kExhRankSort keys: each key's rank is the count of smaller keys (all
// threads read the same key at a time), and the key lands at out[rank] when
// the rank is below nout; more keys: a bitonic sort in place.  Returns the
// sorted array.
constexpr uint32_t kExhRankSort = 512;
__device__ __forceinline__ const unsigned long long *sort_first(unsigned long long *keys, uint32_t n, uint32_t nout,
                                                                unsigned long long *out) {
  if (n <= kExhRankSort) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned long long key = keys[i];
      uint32_t r = 0;
#pragma unroll 8
      for (uint32_t q = 0; q < n; ++q) r += keys[q] < key ? 1u : 0u;
      if (r < nout) out[r] = key;
    }
    __syncthreads();
    return out;
  }
  uint32_t np2 = 1;
  while (np2 < n) np2 <<= 1;
  for (uint32_t i = n + threadIdx.x; i < np2; i += blockDim.x) keys[i] = ~0ull;
  __syncthreads();
  block_bitonic(keys, np2);
  return keys;
}

// Radix select over keys[0, total), total > k: the cut D such that at least k
// keys have d2 <= D, in digits of up to 8 bits from the highest significant
// bit of any d2 (`bits`) down, until no more than `fit` keys lie at or below
// the selected digit's range or the digits are used up (for points spread
// over an area d2 is near uniform, so the first digit usually suffices).
// Whole CTA; every thread gets D.
__device__ uint32_t block_cut(const unsigned long long *keys, uint32_t total, uint32_t k, int bits, uint32_t fit,
                              ExhShared &sh) {
  const int lane = threadIdx.x & 31;
  __syncthreads();
  if (threadIdx.x == 0) {
    sh.prefix = 0;
    sh.rank = k;
    sh.below = 0;
  }
  int hi = bits;  // the bits at and above hi are fixed by the prefix
  for (;;) {
    const int lo = max(hi - 8, 0);
    const uint32_t dmask = (1u << (hi - lo)) - 1u;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) sh.hist[i] = 0;
    __syncthreads();
    const uint32_t prefix = sh.prefix;
    for (uint32_t i0 = 0; i0 < total; i0 += blockDim.x) {
      const uint32_t i = i0 + threadIdx.x;
      uint32_t bin = 0xffffffffu;
      if (i < total) {
        const uint32_t d2 = (uint32_t)(keys[i] >> 32);
        if (hi >= 32 || (d2 >> hi) == (prefix >> hi)) bin = (d2 >> lo) & dmask;
      }
      // one shared atomic per distinct digit of the warp
      const uint32_t peers = __match_any_sync(0xffffffffu, bin);
      if (bin != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&sh.hist[bin], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // warp 0: inclusive scan of 256 bins, 8 per lane
      uint32_t v[8], acc = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        acc += sh.hist[lane * 8 + q];
        v[q] = acc;
      }
      uint32_t off = acc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, off, o);
        if (lane >= o) off += t;
      }
      off -= acc;  // exclusive prefix of this lane's 8 bins
      const uint32_t rank = sh.rank, below = sh.below;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t lo_c = off + (q ? v[q - 1] : 0u), hi_c = off + v[q];
        if (lo_c < rank && rank <= hi_c) {
          sh.prefix = prefix | ((uint32_t)(lane * 8 + q) << lo);
          sh.rank = rank - lo_c;
          sh.le = below + hi_c;  // keys at or below the digit's range
          sh.below = below + lo_c;
        }
      }
    }
    __syncthreads();
    if (lo == 0 || sh.le <= fit) return sh.prefix | ((1u << lo) - 1u);
    hi = lo;
  }
}

// The points of the cells in rings around the item's cell, as keys in
// all[], until k keys lie below the rings' reach: after rings 0..r every
// point with d2 < (r * kCell + 1)^2 has been seen (the cells beyond are that
// far away in x or y), so the k smallest collected keys are then the k
// nearest points under the tie rule; a ring wholly outside the grid means
// every point has been seen.  The cells of consecutive rings are numbered
// 0, 1.. (ring r starts at 4r(r-1) + 1) and taken up to blockDim.x at a time,
// as many as surely fit the buffer; the bound is tested after each such round
// for the last ring it completed.  Once kCutFrom keys are held only the ones
// up to the k-th smallest's cut stay, and no point beyond it enters: an item
// in a hole of a dense image meets thousands of points per ring at its rim
// (before, they overflowed the buffer and sent it to five passes over the
// whole resolved list; 2756 such items of a 512^2 inpainting: 3.4 -> 0.19 ms).
// Leaves the count in sh.total (above cap: the buffer overflowed) and the OR
// of the d2 in sh.prefix.
__device__ __forceinline__ uint32_t ring_base(uint32_t r) { return r == 0 ? 0u : 4u * r * (r - 1u) + 1u; }
constexpr uint32_t kCutFrom = 512;

__device__ void grid_collect(const SessionDev &s, int px, int py, uint32_t k, uint32_t n_tree, ExhShared &sh,
                             unsigned long long *all, uint32_t cap) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    sh.total = 0;
    sh.cnt = 0;
  }
  uint32_t dor = 0, cut = 0xffffffffu;
  __syncthreads();
  const int qcx = (px - s.cox) / kCell, qcy = (py - s.coy) / kCell;
  // rings wholly outside the grid start beyond the farthest grid edge
  const uint32_t r_max = (uint32_t)max(max(qcx, (int)s.cgw - 1 - qcx), max(qcy, (int)s.cgh - 1 - qcy));
  const uint32_t f_end_all = ring_base(r_max + 1);
  for (uint32_t f0 = 0; f0 < f_end_all;) {
    const uint32_t f = f0 + threadIdx.x;
    const uint32_t held = sh.total;
    int gx = -1, gy = -1;
    uint32_t cnt = 0;
    if (f < f_end_all) {
      // ring r of cell number f: 4r(r-1) + 1 <= f < 4r(r+1) + 1
      uint32_t r = f == 0 ? 0u : (uint32_t)(sqrtf((float)(f - 1) * 0.25f + 0.25f) + 0.5f);
      while (r > 0 && ring_base(r) > f) --r;
      while (ring_base(r + 1) <= f) ++r;
      ring_cell((int)r, (int)(f - ring_base(r)), gx, gy);
      gx += qcx;
      gy += qcy;
      cnt = ((unsigned)gx < s.cgw && (unsigned)gy < s.cgh) ? __ldg(&s.cells[(size_t)gy * s.cgw + gx]) : 0u;
    }
    // the round's cells: the first ones whose points fit beside the held keys
    // (all of them once a cut keeps most points out)
    uint32_t f1 = min(f0 + blockDim.x, f_end_all);
    if (cut == 0xffffffffu) {
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) sh.hist[warp] = incl;
      if (threadIdx.x == 0) sh.flag = 0;
      __syncthreads();
      for (int q = 0; q < warp; ++q) incl += sh.hist[q];
      const uint32_t fits = __ballot_sync(0xffffffffu, held + incl <= cap);
      if (lane == 0 && fits) atomicMax(&sh.flag, (uint32_t)(warp * kWarp + 32 - __clz(fits)));
      __syncthreads();
      f1 = min(f1, f0 + max(1u, sh.flag));
    }
    if (f < f1 && cnt) {
      const int x0 = s.cox + gx * kCell, y0 = s.coy + gy * kCell;
      uint32_t found = 0;
      for (int yy = 0; yy < kCell && found < cnt; ++yy) {
        const int y = y0 + yy, dy = y - py;
        uint32_t bits;
        if ((unsigned)y < s.H && x0 >= 0 && x0 + kCell <= (int)s.W) {
          const uint32_t wi = (uint32_t)x0 >> 5, sh5 = (uint32_t)x0 & 31u;
          const uint32_t *row = s.occ + (size_t)y * s.wpr;
          uint64_t wv = __ldg(&row[wi]);
          if (sh5 + kCell > 32) wv |= (uint64_t)__ldg(&row[wi + 1]) << 32;
          bits = (uint32_t)(wv >> sh5) & ((1u << kCell) - 1u);
          found += __popc(bits);
          for (uint32_t t = bits; t;) {
            const int bp = __ffs(t) - 1;
            t &= t - 1u;
            const int dx = x0 + bp - px;
            // beyond the cut, or (k-NN made ahead) a later point
            if ((uint32_t)(dx * dx + dy * dy) > cut || !in_tree(s, (uint32_t)y * s.W + (uint32_t)(x0 + bp), n_tree))
              bits &= ~(1u << bp);
          }
        } else {
          bits = 0;
          for (int xx = 0; xx < kCell; ++xx)
            if (occupied_n(s, x0 + xx, y, n_tree)) bits |= 1u << xx;
          found += __popc(bits);
        }
        while (bits) {
          const int bp = __ffs(bits) - 1;
          bits &= bits - 1u;
          const int x = x0 + bp, dx = x - px;
          const uint32_t d2 = (uint32_t)(dx * dx + dy * dy);
          if (d2 > cut) continue;
          dor |= d2;
          const uint32_t slot = atomicAdd(&sh.total, 1u);
          if (slot < cap) all[slot] = nb_key(d2, x, y);
        }
      }
    }
    __syncthreads();
    const uint32_t n = sh.total;
    if (n > cap) break;
    // the last ring this round completed
    const uint32_t f_done = f1;
    f0 = f1;
    uint32_t r_done = 0;
    while (ring_base(r_done + 2) <= f_done) ++r_done;
    const uint32_t lim = ring_base(r_done + 1) > f_done ? 0u : (uint32_t)(r_done * kCell + 1) * (uint32_t)(r_done * kCell + 1);
    uint32_t c = 0;
    for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) c += (uint32_t)(all[e] >> 32) < lim ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0 && c) atomicAdd(&sh.cnt, c);
    __syncthreads();
    const uint32_t below = sh.cnt;
    __syncthreads();  // every thread has read cnt
    if (below >= k) break;
    if (threadIdx.x == 0) sh.cnt = 0;
    if (n >= kCutFrom && n > k) {
      // the keys up to the k-th smallest's cut, compacted in place
      // (the points seen lie within r_done + 2 cells in x and y)
      const uint32_t far = (r_done + 2) * kCell;
      cut = min(cut, block_cut(all, n, k, 32 - __clz(2 * far * far), max(k, kCutFrom / 2), sh));
      uint32_t kept = 0;
      for (uint32_t e0 = 0; e0 < n; e0 += blockDim.x) {
        const uint32_t e = e0 + threadIdx.x;
        const unsigned long long key = e < n ? all[e] : ~0ull;
        const bool in = (uint32_t)(key >> 32) <= cut && e < n;
        const uint32_t bal = __ballot_sync(0xffffffffu, in);
        if (lane == 0) sh.hist[warp] = __popc(bal);
        __syncthreads();
        uint32_t at = kept + __popc(bal & ((1u << lane) - 1u)), all_in = 0;
        for (uint32_t q = 0; q < blockDim.x / kWarp; ++q) {
          if (q < (uint32_t)warp) at += sh.hist[q];
          all_in += sh.hist[q];
        }
        if (in) all[at] = key;  // (at <= e: every key of this round has been read)
        kept += all_in;
        __syncthreads();
      }
      if (threadIdx.x == 0) sh.total = kept;
    }
    __syncthreads();
  }
  // the OR of the keys' d2 (an upper bound on their bits)
  __syncthreads();
  if (threadIdx.x == 0) sh.prefix = 0;
  __syncthreads();
  dor = __reduce_or_sync(0xffffffffu, dor);
  if (lane == 0 && dor) atomicOr(&sh.prefix, dor);
  __syncthreads();
}

__device__ uint32_t knn_exhaustive_item(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                        ExhShared &sh, unsigned long long *all, uint32_t cap, bool with_mean,
                                        bool use_grid, bool mean_here) {
  const uint32_t pixel = st.items[b.i0 + local];
  int px, py;
  pixel_xy(s, pixel, px, py);
  const uint32_t k = s.k;
  const uint32_t n_res = item_nres(b, b.i0 + local);
  auto d2of = [&](int x, int y) -> uint32_t {
    const int dx = x - px, dy = y - py;
    return (uint32_t)(dx * dx + dy * dy);
  };
  if (threadIdx.x == 0) {
    sh.nkeys = 0;
    sh.total = 0;
    sh.prefix = 0;
    sh.rank = k;
    sh.overflow = 0;
  }
  __syncthreads();
  // pass 1: every key into shared memory while it fits, and the count; one
  // shared atomic per warp and round.  Many points: the cell grid's rings
  // instead, which hold the k nearest.
  const int lane = threadIdx.x & 31;
  const bool grid = use_grid && s.cells != nullptr && n_res > kExhGridFrom;
  if (grid) grid_collect(s, px, py, k, n_res, sh, all, cap);
  // kPts points per thread and round: their loads (the point, then its
  // mirror bit) are all in flight together
  constexpr int kPts = 4;
  for (uint32_t e0 = 0; e0 < (grid ? 0u : n_res); e0 += kPts * blockDim.x) {
    uint32_t pt[kPts];
#pragma unroll
    for (int u = 0; u < kPts; ++u) {
      const uint32_t e = e0 + (uint32_t)u * blockDim.x + threadIdx.x;
      pt[u] = e < n_res ? __ldg(&s.resolved[e]) : 0xffffffffu;
    }
    // up to three keys per point in fixed slots (the point, its mirror
    // across x, its mirror across y), compacted through a bit mask
    int xs[3 * kPts], ys[3 * kPts];
    uint32_t vm = 0;
#pragma unroll
    for (int u = 0; u < kPts; ++u) {
      const int x = (int)(pt[u] % s.W), y = (int)(pt[u] / s.W);
      const bool mb = pt[u] != 0xffffffffu && s.tiling && mir_bit(s, (uint32_t)x, (uint32_t)y);
      xs[3 * u] = x;
      ys[3 * u] = y;
      xs[3 * u + 1] = x < s.x_l ? x + (int)s.W : x - (int)s.W;
      ys[3 * u + 1] = y;
      xs[3 * u + 2] = x;
      ys[3 * u + 2] = y < s.y_b ? y + (int)s.H : y - (int)s.H;
      if (pt[u] != 0xffffffffu) vm |= 1u << (3 * u);
      if (mb && (x < s.x_l || x > s.x_r)) vm |= 2u << (3 * u);
      if (mb && (y < s.y_b || y > s.y_t)) vm |= 4u << (3 * u);
    }
    const uint32_t cnt = (uint32_t)__popc(vm);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&sh.total, incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - cnt;
    uint32_t dor = 0;
#pragma unroll
    for (int i = 0; i < 3 * kPts; ++i) {
      if ((vm >> i) & 1u) {
        const uint32_t d2 = d2of(xs[i], ys[i]);
        dor |= d2;
        const uint32_t slot = base + (uint32_t)__popc(vm & ((1u << i) - 1u));
        if (slot < cap) all[slot] = nb_key(d2, xs[i], ys[i]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dor |= __shfl_xor_sync(0xffffffffu, dor, o);
    if (lane == 0 && dor) atomicOr(&sh.prefix, dor);  // prefix holds the OR of all d2 until the select
  }
  __syncthreads();
  uint32_t total = sh.total;
  if (use_grid && !grid && total > cap && s.cells != nullptr) {
    __syncthreads();
    grid_collect(s, px, py, k, n_res, sh, all, cap);
    total = sh.total;
  }
  const unsigned long long *sorted;
  uint32_t n;
  if (total <= k || total <= cap) {
    // radix select over the shared keys, digits of up to 8 bits from the
    // highest significant bit of any d2 down, until the keys at or below the
    // selected digit's range fit the sort buffer (for points spread over an
    // area d2 is near uniform, so the first digit usually suffices); few
    // keys are sorted whole
    const uint32_t dor_all = sh.prefix;
    const int bits = dor_all ? 32 - __clz(dor_all) : 1;
    if (total > k && total > (uint32_t)kExhSortAll) {
      const uint32_t D = block_cut(all, total, k, bits, (uint32_t)kExhCap, sh);
      // keys at or below the cut, into the small buffer
      if (threadIdx.x == 0) sh.nkeys = 0;
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
        const unsigned long long key = all[i];
        if ((uint32_t)(key >> 32) <= D) {
          const uint32_t slot = atomicAdd(&sh.nkeys, 1u);
          if (slot < (uint32_t)kExhCap)
            sh.keys[slot] = key;
          else
            sh.overflow = 1;
        }
      }
    } else {
      if (threadIdx.x == 0) sh.nkeys = total;
      for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) sh.keys[i] = all[i];
    }
    __syncthreads();
    if (sh.overflow) {
      if (threadIdx.x == 0) {
        set_err(s.err, kDevErrLimit);
        b.ncnt[local] = 0;
      }
      return 0;
    }
    n = sh.nkeys;
    sorted = sort_first(sh.keys, n, n < k ? n : k, all);
  } else {
    if (threadIdx.x == 0) {
      sh.prefix = 0;
      sh.rank = k;
    }
    __syncthreads();
    // radix select of the k-th smallest d2 over further passes
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      for (int i = threadIdx.x; i < 256; i += blockDim.x) sh.hist[i] = 0;
      __syncthreads();
      const uint32_t prefix = sh.prefix;
      for_points(s, n_res, [&](int x, int y) {
        const uint32_t d2 = d2of(x, y);
        const bool match = pass == 0 || ((d2 ^ prefix) >> (shift + 8)) == 0;
        if (match) atomicAdd(&sh.hist[(d2 >> shift) & 255u], 1u);
      });
      __syncthreads();
      if (threadIdx.x == 0) {
        uint32_t cum = 0, rank = sh.rank;
        for (int bk = 0; bk < 256; ++bk) {
          const uint32_t h = sh.hist[bk];
          if (cum + h >= rank) {
            sh.prefix = prefix | ((uint32_t)bk << shift);
            sh.rank = rank - cum;
            break;
          }
          cum += h;
        }
      }
      __syncthreads();
    }
    const uint32_t D = sh.prefix;
    for_points(s, n_res, [&](int x, int y) {
      const uint32_t d2 = d2of(x, y);
      if (d2 <= D) {
        const uint32_t slot = atomicAdd(&sh.nkeys, 1u);
        if (slot < (uint32_t)kExhCap)
          sh.keys[slot] = nb_key(d2, x, y);
        else
          sh.overflow = 1;
      }
    });
    __syncthreads();
    if (sh.overflow) {
      if (threadIdx.x == 0) {
        set_err(s.err, kDevErrLimit);
        b.ncnt[local] = 0;
      }
      return 0;
    }
    n = sh.nkeys;
    sorted = sort_first(sh.keys, n, n < k ? n : k, all);
  }
  const uint32_t nout = n < k ? n : k;
  int32_t *nbo = b.nbuf + (size_t)local * k;
  const uint32_t nb = b.i1 - b.i0;
  // the f64 distances from the coordinate tables, where something reads
  // them: the stored lists of an inexact session, and the caller's weights
  // when the mean is not made here (exact sums derive the rest from the
  // offsets, lists made ahead leave theirs to k_mean_ahead)
  const bool ahead = s.rank != nullptr;
  const bool want_d = (!s.exact_sum && !ahead) || (with_mean && !mean_here);
  unsigned long long part = 0;
  for (uint32_t i = threadIdx.x; i < nout; i += blockDim.x) {
    const unsigned long long key = sorted[i];
    const int x = (int)(key & 0xffffu) - 32768, y = (int)((key >> 16) & 0xffffu) - 32768;
    nbo[i] = pack_off(x - px, y - py);
    const double d = !want_d ? 0.0
                     : s.exact_sum ? exact_dist(s, pack_off(x - px, y - py))
                                   : neighbour_dist(s, px, py, x - px, y - py);
    if (s.exact_sum)
      part += exact_units(s, x - px, y - py);
    else if (!ahead)
      b.dist[(size_t)i * nb + local] = d;
    if (with_mean) {
      sh.dist[i] = d;
      sh.nbo[i] = pack_off(x - px, y - py);
    }
  }
  if (s.exact_sum && mean_here) {
    // every item of the launch, fallback items included, gets its mean here
    part = warp_sum_units(part);
    if ((threadIdx.x & 31) == 0) sh.wsum[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0 && nout > 0) {
      unsigned long long sum = 0;
      for (uint32_t w = 0; w < blockDim.x / 32; ++w) sum += sh.wsum[w];
      b.mean[local] = exact_mean(s, sum, nout);
    }
  } else if (with_mean && mean_here && !ahead) {
    __syncthreads();
    if (threadIdx.x == 0 && nout > 0) b.mean[local] = mean_chain(sh.dist, nout);
  }
  if (threadIdx.x == 0) b.ncnt[local] = nout;
  return nout;
}

// ---------------------------------------------------------------------------
// k-NN over a short resolved list (the sparse first steps, up to kListMax
// points), lists made ahead: a warp per item.  One pass over the tree's points
// keeps the keys within a squared radius chosen from the density so that some
// 1.5 k points are expected; too few or too many and the radius is bisected
// (the count grows with it).  The keys' ranks among each other are their
// places.  A CTA per item with a radix select over every key (the exhaustive
// form, which still takes the items whose radius does not settle and those
// the walk could not finish) took 74 us for a launch of a few thousand items
// and held the first stage's steps up; this one takes 30.
// ---------------------------------------------------------------------------
constexpr uint32_t kListWarps = 4;
constexpr uint32_t kListMax = 4096;
__host__ __device__ __forceinline__ uint32_t list_cap(uint32_t k) { return 2u * k + 96u; }

__device__ __forceinline__ void knn_list_body(const SessionDev &s, const StageDev &st, const BatchDev &b) {
  extern __shared__ unsigned long long list_keys[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u, cap = list_cap(s.k), nb = b.i1 - b.i0;
  unsigned long long *keys = list_keys + (size_t)warp * cap;
  for (uint32_t local = blockIdx.x * kListWarps + warp; local < nb; local += gridDim.x * kListWarps) {
    const uint32_t pixel = st.items[b.i0 + local], n_tree = item_nres(b, b.i0 + local);
    int px, py;
    pixel_xy(s, pixel, px, py);
    // squared radius of a disc that holds 1.5 k + 8 of n points spread over the image
    const float want = 1.5f * (float)s.k + 8.0f;
    const float r2 = want * (float)s.W * (float)s.H / (3.1415927f * (float)max(n_tree, 1u));
    uint32_t lo = 0, hi = 0xffffffffu;  // counts: at lo (if > 0) below k, at hi (if found) above cap
    uint32_t lim = r2 < 2.0e9f ? (uint32_t)r2 : 2000000000u;
    if (n_tree <= s.k) lim = 0xfffffffeu;
    uint32_t n = 0;
    bool settled = false;
    for (int pass = 0; pass < 24 && !settled; ++pass) {
      n = 0;
      auto add = [&](bool in, int x, int y) {
        const int dx = x - px, dy = y - py;
        const uint32_t d2 = (uint32_t)(dx * dx + dy * dy);
        in = in && d2 <= lim;
        const uint32_t bal = __ballot_sync(0xffffffffu, in);
        const uint32_t at = n + __popc(bal & lt);
        if (in && at < cap) keys[at] = nb_key(d2, x, y);
        n += __popc(bal);
      };
      for (uint32_t e0 = 0; e0 < n_tree; e0 += 4 * kWarp) {
        uint32_t pt[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t e = e0 + (uint32_t)u * kWarp + lane;
          pt[u] = e < n_tree ? __ldg(&s.resolved[e]) : 0xffffffffu;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool on = pt[u] != 0xffffffffu;
          int x = 0, y = 0;
          if (on) pixel_xy(s, pt[u], x, y);
          add(on, x, y);
          if (s.tiling) {
            // its mirrors (flush_resolved, ms.rs:306-328)
            const int mx = x < s.x_l ? (int)s.W : (x > s.x_r ? -(int)s.W : 0);
            const int my = y < s.y_b ? (int)s.H : (y > s.y_t ? -(int)s.H : 0);
            const bool mb = on && (mx | my) != 0 && mir_bit(s, (uint32_t)x, (uint32_t)y);
            if (__any_sync(0xffffffffu, mb)) {
              add(mb && mx != 0, x + mx, y);
              add(mb && my != 0, x, y + my);
            }
          }
        }
      }
      if (n > cap) {
        hi = lim;
        if (hi - lo <= 1) break;  // more points at one distance than there is room for
        lim = lo + (hi - lo) / 2;
      } else if (n < s.k && lim < 0xfffffffeu && hi - lo > 1) {
        lo = lim;
        // grow the area; between a too small and a too large one, halve
        lim = hi == 0xffffffffu ? (lim < 1000000000u ? lim * 2u + 2u : 0xfffffffeu) : lo + (hi - lo) / 2;
      } else {
        settled = n >= s.k || lim == 0xfffffffeu;
        if (!settled) break;
      }
    }
    __syncwarp();
    if (!settled) {
      if (lane == 0) b.fb_list[atomicAdd(b.fb_count, 1u)] = local;
      continue;
    }
    // each key's place: the number of smaller ones (keys are distinct)
    const uint32_t nout = min(n, s.k);
    int32_t *nbo = b.nbuf + (size_t)local * s.k;
    // 64-bit: a lane holds up to (2 k + 96) / 32 keys, whose squared offsets
    // reach 2^28 each (a cluster at the other end of a 16384-wide output)
    unsigned long long units = 0;
    for (uint32_t e0 = 0; e0 < n; e0 += kWarp) {
      const uint32_t e = e0 + lane;
      const unsigned long long key = e < n ? keys[e] : ~0ull;
      uint32_t r = 0;
#pragma unroll 4
      for (uint32_t q = 0; q < n; ++q) r += keys[q] < key ? 1u : 0u;
      if (e < n && r < nout) {
        const int dx = (int)(key & 0xffffu) - 32768 - px, dy = (int)((key >> 16) & 0xffffu) - 32768 - py;
        nbo[r] = pack_off(dx, dy);
        units += exact_units(s, dx, dy);
      }
    }
    if (s.exact_sum) {
      units = warp_sum_units(units);
      if (lane == 0 && nout) b.mean[local] = exact_mean(s, units, nout);
    }
    if (lane == 0) b.ncnt[local] = nout;
    __syncwarp();  // the keys are rebuilt for the warp's next item
  }
}

// ---------------------------------------------------------------------------
// mean: thread per item (get_distances_to_k_neighs, ms.rs:417-423): the sum
// of the 4x-duplicated distance list in order, then / (4k).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mean_body(const SessionDev &s, const BatchDev &b, uint32_t vb) {
  const uint32_t nb = b.i1 - b.i0;
  const uint32_t local = vb * blockDim.x + threadIdx.x;
  if (local >= nb) return;
  const uint32_t nk = b.ncnt[local];
  if (nk == 0) return;
  // one item per lane: 32 chains share each f64 warp instruction, which on
  // GB300 costs the same whatever its active-lane count
  double sum = 0.0;
#pragma unroll 8
  for (uint32_t j = 0; j < nk; ++j) {
    const double d = b.dist[(size_t)j * nb + local];
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
  }
  b.mean[local] = __ddiv_rn(sum, (double)(nk * 4u));
}

// ---------------------------------------------------------------------------
// resolve: warp per item.
// ---------------------------------------------------------------------------
// Per-item shared memory: one 16-byte record per neighbour {its texel offset
// on the padded planes (dy * ppitch + dx), own pattern texel, target-guide
// texel, weight bits}, its packed offset, and the candidates {x | y<<16,
// map | neg flag | source index << 16}.
struct WarpSmem {
  uint4 *nbr;
  uint2 *cand;
  float *term;   // candidate 0's neighbour terms
  int32_t *off;  // packed neighbour offsets
};

__device__ __forceinline__ size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }

__host__ __device__ __forceinline__ size_t warp_smem_bytes(uint32_t k, uint32_t m) {
  const size_t kk = k ? k : 1;
  size_t b = kk * 16;                        // nbr
  b += ((kk + m) * 8 + 15) & ~(size_t)15;    // cand
  b += (kk * 4 + 15) & ~(size_t)15;          // term
  b += (kk * 4 + 15) & ~(size_t)15;          // off
  return b;
}

__device__ __forceinline__ WarpSmem carve(unsigned char *base, uint32_t k, uint32_t m) {
  const size_t kk = k ? k : 1;
  WarpSmem w;
  unsigned char *p = base;
  w.nbr = (uint4 *)p;
  p += kk * 16;
  w.cand = (uint2 *)p;
  p += align16((kk + m) * 8);
  w.term = (float *)p;
  p += align16(kk * 4);
  w.off = (int32_t *)p;
  return w;
}

constexpr uint32_t kAuxNeg = 0x8000u;  // random candidate: neighbourhood c + (p - n)

// Random candidate t of an item's list as a candidate record.
__device__ __forceinline__ uint2 random_candidate(const SessionDev &s, uint2 v, uint32_t t) {
  v = use_rcand(s, v);
  return make_uint2(v.x, v.y | kAuxNeg | (t << 16));
}
__device__ __forceinline__ uint2 random_candidate(const SessionDev &s, const uint2 *rc, uint32_t t) {
  return random_candidate(s, __ldg(&rc[t]), t);
}

__device__ __forceinline__ uint32_t texel(const uint32_t *lv, const MapDesc &md, int x, int y) {
  if ((unsigned)x < md.w && (unsigned)y < md.h) return __ldg(&lv[(size_t)y * md.w + x]);
  return kOutside;
}

// Sum of the four channel LUT terms in channel order, starting from acc.
// The byte offsets of the four entries come straight from the packed
// differences (d >> (8c - 2)) & 0x3fc.  kOpaque (StageDev::opaque): the
// alpha difference is always 0 and its term +-0, which leaves the sum as it
// is, so only the colour channels are looked up.
template <bool kOpaque = false>
__device__ __forceinline__ float lut4(const float *lut, uint32_t d, float acc) {
  const char *lb = (const char *)lut;
  acc = __fadd_rn(acc, *(const float *)(lb + ((d << 2) & 0x3fcu)));
  acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 6) & 0x3fcu)));
  acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 14) & 0x3fcu)));
  if (!kOpaque) acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 22) & 0x3fcu)));
  return acc;
}
// The same with the stage's flag at run time (the alpha lookup predicated).
__device__ __forceinline__ float lut4r(const float *lut, uint32_t d, float acc, int opaque) {
  const char *lb = (const char *)lut;
  acc = __fadd_rn(acc, *(const float *)(lb + ((d << 2) & 0x3fcu)));
  acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 6) & 0x3fcu)));
  acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 14) & 0x3fcu)));
  if (!opaque) acc = __fadd_rn(acc, *(const float *)(lb + ((d >> 22) & 0x3fcu)));
  return acc;
}

// Cost of candidate c (better_match, ms.rs:1225-1288), abandoning once the
// partial sum reaches `bound`; bounds-checked gathers (out-of-bounds texels
// read Rgba(0,0,0,255)), issued four neighbours ahead.  Returns false when
// abandoned.  The terms are never negative, so partial sums never decrease
// and testing every fourth one, and the total, decides as the reference's
// test after every term does.
// kG = false compiles the guide terms out (sessions without guides).
template <bool kG = true>
__device__ __forceinline__ bool candidate_cost(const SessionDev &s, const StageDev &st, const WarpSmem &w,
                                               const float *lc, const float *lg, uint32_t nk, uint32_t cxy,
                                               uint32_t aux, float bound, float &out) {
  const uint32_t map = aux & 0x7fffu;
  const int sg = (aux & kAuxNeg) ? -1 : 1;
  const MapDesc md = s.maps[map];
  const uint32_t *lv = s.levels + md.off + (size_t)st.level * md.w * md.h;
  const int cx = (int)(cxy & 0xffffu), cy = (int)(cxy >> 16);
  const uint32_t *gv = nullptr;
  GuideDesc gd;
  if (kG && s.guided) {
    gd = s.gdesc[map];
    gv = s.guides + gd.off + (size_t)st.level * gd.w * gd.h;
  }
  float score = 0.0f;
  for (uint32_t j0 = 0; j0 < nk; j0 += 4) {
    uint4 nr[4];
    uint32_t t[4], gt[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      t[u] = kOutside;
      gt[u] = kOutside;
      if (j0 + u < nk) {
        nr[u] = w.nbr[j0 + u];
        const int32_t o = w.off[j0 + u];
        const int qx = cx + sg * off_dx(o), qy = cy + sg * off_dy(o);
        if ((unsigned)qx < md.w && (unsigned)qy < md.h) t[u] = __ldg(&lv[(size_t)qy * md.w + qx]);
        if (kG && s.guided && (unsigned)qx < gd.w && (unsigned)qy < gd.h) gt[u] = __ldg(&gv[(size_t)qy * gd.w + qx]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u >= nk) break;
      float nps = lut4(lc, __vabsdiffu4(nr[u].y, t[u]), 0.0f);
      if (kG && s.guided) nps = lut4(lg, __vabsdiffu4(nr[u].z, gt[u]), nps);
      score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr[u].w)));
    }
    if (score >= bound) return false;
  }
  out = score;
  return true;
}

// Terms [j, j + C) of a guided candidate, their gathers in flight together
// (the records are read again for the terms instead of held in registers).
template <int C, bool kOpaque>
__device__ __forceinline__ float guided_chunk(const WarpSmem &w, const float *lc, const float *lg, const char *base,
                                              const char *gbase, int sg, uint32_t j, float score) {
  uint32_t t[C], gt[C];
#pragma unroll
  for (int u = 0; u < C; ++u) {
    const int64_t at = (int64_t)sg * (int32_t)w.nbr[j + u].x;
    t[u] = __ldg((const uint32_t *)(base + at));
    gt[u] = __ldg((const uint32_t *)(gbase + at));
  }
#pragma unroll
  for (int u = 0; u < C; ++u) {
    const uint4 nr = w.nbr[j + u];
    float nps = lut4<kOpaque>(lc, __vabsdiffu4(nr.y, t[u]), 0.0f);
    nps = lut4<kOpaque>(lg, __vabsdiffu4(nr.z, gt[u]), nps);
    score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr.w)));
  }
  return score;
}

// The same on the padded images, for items whose neighbour offsets all lie
// within kPad: no bounds checks, gathers issued four neighbours ahead; with a
// guide, whose evaluations are twice as long, six once a candidate has passed
// its first four, where most random ones end (512^2, k = m = 50: 6.30 -> 5.95
// ms; with four, five, seven, eight, twelve 6.10, 6.11, 6.08, 6.15, 6.6;
// without a guide six cost 2048^2 3%).
// centre: texel index of the candidate's centre on the padded planes.
template <bool kGuided, bool kOpaque>
__device__ __forceinline__ bool candidate_cost_padded_v(const SessionDev &s, const WarpSmem &w, const float *lc,
                                                      const float *lg, uint32_t nk, uint64_t centre, bool neg,
                                                      float bound, float &out) {
  const int sg = neg ? -4 : 4;  // bytes per texel, signed: the gather address is one multiply-add
  const char *base = (const char *)(s.plevels + centre);
  const char *gbase = kGuided ? (const char *)(s.pguides + centre) : nullptr;
  float score = 0.0f;
  uint32_t j = 0;
  if (kGuided && nk >= 10) {
    score = guided_chunk<4, kOpaque>(w, lc, lg, base, gbase, sg, 0, score);
    if (score >= bound) return false;
    for (j = 4; j + 6 <= nk; j += 6) {
      score = guided_chunk<6, kOpaque>(w, lc, lg, base, gbase, sg, j, score);
      if (score >= bound) return false;
    }
  }
  for (; j + 4 <= nk; j += 4) {
    uint4 nr[4];
    uint32_t t[4], gt[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      nr[u] = w.nbr[j + u];
      const int64_t at = (int64_t)sg * (int32_t)nr[u].x;
      t[u] = __ldg((const uint32_t *)(base + at));
      if (kGuided) gt[u] = __ldg((const uint32_t *)(gbase + at));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float nps = lut4<kOpaque>(lc, __vabsdiffu4(nr[u].y, t[u]), 0.0f);
      if (kGuided) nps = lut4<kOpaque>(lg, __vabsdiffu4(nr[u].z, gt[u]), nps);
      score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr[u].w)));
    }
    if (score >= bound) return false;
  }
  for (; j < nk; ++j) {
    const uint4 nr = w.nbr[j];
    const int64_t at = (int64_t)sg * (int32_t)nr.x;
    float nps = lut4<kOpaque>(lc, __vabsdiffu4(nr.y, __ldg((const uint32_t *)(base + at))), 0.0f);
    if (kGuided) nps = lut4<kOpaque>(lg, __vabsdiffu4(nr.z, __ldg((const uint32_t *)(gbase + at))), nps);
    score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr.w)));
  }
  if (score >= bound) return false;
  out = score;
  return true;
}

// The loop in two versions, chosen per stage (a uniform branch).
template <bool kGuided>
__device__ __forceinline__ bool candidate_cost_padded(const SessionDev &s, const StageDev &st, const WarpSmem &w,
                                                      const float *lc, const float *lg, uint32_t nk, uint64_t centre,
                                                      bool neg, float bound, float &out) {
  if (st.opaque) return candidate_cost_padded_v<kGuided, true>(s, w, lc, lg, nk, centre, neg, bound, out);
  return candidate_cost_padded_v<kGuided, false>(s, w, lc, lg, nk, centre, neg, bound, out);
}

// Texel index of (x, y) of a map's level on the padded planes.
__device__ __forceinline__ uint64_t padded_centre(const MapDesc &md, uint32_t level, uint32_t cxy) {
  return md.poff + (uint64_t)level * md.pw * md.ph + (uint64_t)((cxy >> 16) + kPad) * md.pw + ((cxy & 0xffffu) + kPad);
}

// Per-neighbour set-up of an item: weight (find_best_match, ms.rs:1198-1203,
// w = (f32) exp(-(d / mean))), own pattern texel and target-guide texel
// (ms.rs:1151-1181, wrapped when tiling), the record in shared memory, and
// the neighbour's coherence candidate (ms.rs:497-547): its source plus the
// shift to the centre, kept if valid.  Returns true for a valid candidate.
// The weight alone, w = (f32) exp(-(d / mean)) (find_best_match,
// ms.rs:1198-1203): the double-f32 path when it decides, else the exact f64
// one (about one weight in 2^15; the empty asm keeps the reciprocal from
// being computed ahead for every item, on an FP64 pipe that takes 18 cycles
// of an SM per instruction).
__device__ __forceinline__ float weight_exact(double dj, double avg) {
  asm volatile("" : "+d"(avg));
  return __double2float_rn(ts_exp64(-1.0 * ts_div_markstein(dj, avg, __drcp_rn(avg)), g_exp2_64));
}
__device__ __forceinline__ float neighbour_weight(double dj, double avg, const float *tab_ff) {
  float wv;
  if (!ts_weight_ff(dj, avg, tab_ff, wv)) wv = weight_exact(dj, avg);
  return wv;
}

// Batch-start colour and state of output pixel p: the image, unless the
// previous batch step left its commit to this launch (BatchDev::prev_tag)
// and p is one of its pixels, whose values the shadow holds.  All loads are
// issued together.  Tags of this launch's own deferred pixels never equal
// prev_tag.
__device__ __forceinline__ void start_pixel(const SessionDev &s, const BatchDev &b, uint32_t p, bool want_colour,
                                            uint32_t &colour, uint4 &state) {
  colour = want_colour ? s.color[p] : 0u;
  state = s.state[p];
  if (b.prev_tag) {
    const uint4 h0 = s.shadow[2 * (size_t)p], h1 = s.shadow[2 * (size_t)p + 1];
    if (h0.x == b.prev_tag) {
      colour = want_colour ? h0.y : 0u;
      state = h1;
    }
  }
}

// Everything of neighbour_setup but the weight, which the record gets as wv.
// A neighbour is a tree point, so it or the pixel it mirrors lies in the
// image (wrap1).
template <bool kG = true>
__device__ __forceinline__ bool neighbour_records(const SessionDev &s, const StageDev &st, const BatchDev &b, int px,
                                                  int py, uint32_t j, int32_t off, float wv, const WarpSmem &w,
                                                  uint32_t &cxy, uint32_t &aux, int &maxoff, bool &bad_map) {
  const int dx = off_dx(off), dy = off_dy(off);
  maxoff = max(maxoff, max(abs(dx), abs(dy)));
  const uint32_t p = (uint32_t)wrap1(py + dy, (int)s.H) * s.W + (uint32_t)wrap1(px + dx, (int)s.W);
  uint32_t pat;
  uint4 sv;
  start_pixel(s, b, p, true, pat, sv);
  uint32_t gpat = 0;
  if (kG && s.guided) gpat = __ldg(&s.tguide[(size_t)st.level * s.W * s.H + p]);
  w.nbr[j] = make_uint4((uint32_t)(dy * (int)s.ppitch + dx), pat, gpat, __float_as_uint(wv));
  w.off[j] = off;
  const uint32_t map = sv.z;
  if (map >= s.n_maps) {
    bad_map = true;
    return false;
  }
  const int ccx = (int)(sv.x & 0xffffu) - dx;
  const int ccy = (int)(sv.x >> 16) - dy;
  if (!coord_valid(s, s.maps[map], ccx, ccy)) return false;
  cxy = (uint32_t)ccx | ((uint32_t)ccy << 16);
  aux = map | (j << 16);
  return true;
}

// The weight of an item's neighbour j at offset off (fm = ts_ff_mean(avg)).
// Sessions with exact sums and equal sides: the distance is dx^2 + dy^2 units,
// an f32 pair (below 2^24 units a single f32).
// Other sessions: the stored list, or (made ahead) the coordinate tables.
__device__ __forceinline__ double item_dist(const SessionDev &s, const BatchDev &b, uint32_t local, uint32_t nb,
                                            int px, int py, uint32_t j, int32_t off) {
  if (s.exact_sum) return exact_dist(s, off);
  if (!s.rank) return b.dist[(size_t)j * nb + local];
  return neighbour_dist(s, px, py, off_dx(off), off_dy(off));
}
__device__ __forceinline__ float item_weight(const SessionDev &s, const BatchDev &b, uint32_t local, uint32_t nb,
                                             int px, int py, uint32_t j, int32_t off, double avg, const FfMean &fm,
                                             const float *tab_ff) {
  float d_hi = 0.0f, d_lo = 0.0f, wv;
  bool split = true;
  if (s.exact_sum && (s.exact_sx | s.exact_sy) == 0u) {
    const int dx = off_dx(off), dy = off_dy(off);
    const uint32_t u = (uint32_t)(dx * dx + dy * dy);
    const float hi = (float)u;
    d_hi = __fmul_rn(hi, s.exact_qf);
    d_lo = __fmul_rn((float)(int32_t)(u - (uint32_t)hi), s.exact_qf);
  } else {
    const double d = s.exact_sum ? bits_dbl(ts_units_bits(exact_units(s, off_dx(off), off_dy(off)), s.exact_qe))
                                 : item_dist(s, b, local, nb, px, py, j, off);
    split = dbl_bits(d) == 0 || ff_split_rn(d, d_hi, d_lo);
  }
  if (!(split && ts_weight_ff_pair(d_hi, d_lo, fm, tab_ff, wv)))
    wv = weight_exact(item_dist(s, b, local, nb, px, py, j, off), avg);
  return wv;
}

template <bool kG = true>
__device__ __forceinline__ bool neighbour_setup(const SessionDev &s, const StageDev &st, const BatchDev &b,
                                                uint32_t local, uint32_t nb, int px, int py, uint32_t j, int32_t off,
                                                double avg, const FfMean &fm, const float *tab_ff,
                                                const WarpSmem &w, uint32_t &cxy, uint32_t &aux, bool &nan_w,
                                                int &maxoff, bool &bad_map) {
  const float wv = item_weight(s, b, local, nb, px, py, j, off, avg, fm, tab_ff);
  nan_w |= (wv != wv);
  return neighbour_records<kG>(s, st, b, px, py, j, off, wv, w, cxy, aux, maxoff, bad_map);
}

// Candidate 0's exact score (better_match, ms.rs:1225-1288, with no bound):
// lane j of a group of G lanes (a warp, or a CTA's warp) computes the terms
// nps_j * w_j of neighbours j, j + G, ..., then every lane sums them in
// order.
template <int G, bool kG = true>
__device__ __forceinline__ float candidate0_score(const SessionDev &s, const StageDev &st, const WarpSmem &w,
                                                  const float *lc, const float *lg, uint32_t nk, int gl,
                                                  uint32_t gmask) {
  const uint32_t cxy0 = w.cand[0].x, aux0 = w.cand[0].y;
  const uint32_t map = aux0 & 0x7fffu;
  const bool neg = (aux0 & kAuxNeg) != 0;
  const MapDesc md = s.maps[map];
  const uint32_t *lv = s.levels + md.off + (size_t)st.level * md.w * md.h;
  const int cx = (int)(cxy0 & 0xffffu), cy = (int)(cxy0 >> 16);
  for (uint32_t j = gl; j < nk; j += G) {
    const uint4 nr = w.nbr[j];
    int dx = off_dx(w.off[j]), dy = off_dy(w.off[j]);
    if (neg) {
      dx = -dx;
      dy = -dy;
    }
    const int qx = cx + dx, qy = cy + dy;
    float nps = lut4(lc, __vabsdiffu4(nr.y, texel(lv, md, qx, qy)), 0.0f);
    if (kG && s.guided) {
      const GuideDesc gd = s.gdesc[map];
      const uint32_t *gv = s.guides + gd.off + (size_t)st.level * gd.w * gd.h;
      uint32_t gt = kOutside;
      if ((unsigned)qx < gd.w && (unsigned)qy < gd.h) gt = __ldg(&gv[(size_t)qy * gd.w + qx]);
      nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
    }
    w.term[j] = __fmul_rn(nps, __uint_as_float(nr.w));
  }
  __syncwarp(gmask);
  float sc = 0.0f;
  uint32_t j = 0;
  for (; j + 4 <= nk; j += 4) {
    const float4 t4 = *(const float4 *)(w.term + j);
    sc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sc, t4.x), t4.y), t4.z), t4.w);
  }
  for (; j < nk; ++j) sc = __fadd_rn(sc, w.term[j]);
  return sc;
}

// The reference's sequential find_best_match (ms.rs:1184-1221), for stages or
// items with non-finite costs, where early exit and argmin need its exact
// comparison sequence.  One thread.  Candidates from n_coh on lie
// `gap` records further.
template <bool kG = true>
__device__ void sequential_best(const SessionDev &s, const StageDev &st, const WarpSmem &w, const float *lc,
                                const float *lg, uint32_t nk, uint32_t nc, float &best_s, uint32_t &best_i,
                                uint32_t n_coh = 0, uint32_t gap = 0) {
  best_s = FLT_MAX;
  best_i = 0;
  for (uint32_t c = 0; c < nc; ++c) {
    const uint2 cd = w.cand[c < n_coh ? c : c + gap];
    const uint32_t aux = cd.y;
    const uint32_t map = aux & 0x7fffu;
    const bool neg = (aux & kAuxNeg) != 0;
    const MapDesc md = s.maps[map];
    const uint32_t *lv = s.levels + md.off + (size_t)st.level * md.w * md.h;
    const int cx = (int)(cd.x & 0xffffu), cy = (int)(cd.x >> 16);
    float score = 0.0f;
    bool better = true;
    for (uint32_t j = 0; j < nk; ++j) {
      const uint4 nr = w.nbr[j];
      int dx = off_dx(w.off[j]), dy = off_dy(w.off[j]);
      if (neg) {
        dx = -dx;
        dy = -dy;
      }
      const int qx = cx + dx, qy = cy + dy;
      float nps = lut4(lc, __vabsdiffu4(nr.y, texel(lv, md, qx, qy)), 0.0f);
      if (kG && s.guided) {
        const GuideDesc gd = s.gdesc[map];
        const uint32_t *gv = s.guides + gd.off + (size_t)st.level * gd.w * gd.h;
        uint32_t gt = kOutside;
        if ((unsigned)qx < gd.w && (unsigned)qy < gd.h) gt = gv[(size_t)qy * gd.w + qx];
        nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
      }
      score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr.w)));
      if (score >= best_s) {
        better = false;
        break;
      }
    }
    if (better) {
      best_s = score;
      best_i = c;
    }
  }
}

// Which cost tables a copy of a resolve body takes.  The single-session kernels
// come in two copies: in order (kLutSigned) and the rest, whose registers and
// code the former would cost guided runs 1%.
enum CostMode { kCostPlain, kCostSigned, kCostAny };
template <int kMode>
__device__ __forceinline__ bool costs_in_order(const StageDev &st) {
  return kMode == kCostSigned || (kMode == kCostAny && st.slow_lut == kLutSigned);
}
template <int kMode>
__device__ __forceinline__ bool costs_exact(const StageDev &st) {
  return kMode == kCostPlain ? st.slow_lut != 0 : kMode == kCostAny && st.slow_lut == kLutExact;
}

// A warp's candidates in index order (lane l: candidate first + l), each taken
// where its largest partial sum lies below the best score so far (why:
// best_in_order).
__device__ __forceinline__ void take_signed(float sum, float peak, uint32_t first, float &best_s, uint32_t &best_i) {
  uint32_t later = 0xffffffffu;
  for (;;) {
    const uint32_t below = __ballot_sync(0xffffffffu, peak < best_s) & later;
    if (below == 0) return;
    const int l = __ffs(below) - 1;
    best_s = __shfl_sync(0xffffffffu, sum, l);
    best_i = first + (uint32_t)l;
    later = 0xfffffffeu << l;
  }
}

// find_best_match for finite tables with negative entries (kLutSigned), where a
// partial sum can fall again: a whole warp, a candidate per lane.  The
// reference rejects a candidate at the first partial sum that reaches the best
// score so far, so it takes one exactly when its largest partial sum lies below
// that score, which its own then replaces.  The score only falls, so a
// candidate may be left once it reaches the one at the start of its round, and
// a repeat of an earlier candidate is never taken (that one was rejected by a
// best that was no lower, or its sum, no more than its largest partial sum,
// became the best).  Guided inpainting, k = m = 50, one lane going through all
// candidates against this, device time: 256^2 2.61 against 0.51 ms, 512^2 3.39
// against 0.88, 1024^2 6.75 against 2.19.
template <bool kG = true>
__device__ void best_in_order(const SessionDev &s, const StageDev &st, const WarpSmem &w, const float *lc,
                              const float *lg, uint32_t nk, uint32_t nc, float &best_s, uint32_t &best_i) {
  const uint32_t lane = threadIdx.x & 31u;
  // candidate 0 is always taken (its sums are finite): its terms on all lanes
  best_s = candidate0_score<kWarp, kG>(s, st, w, lc, lg, nk, (int)lane, 0xffffffffu);
  best_i = 0;
  for (uint32_t base = 1; base < nc; base += kWarp) {
    const uint32_t c = base + lane;
    float score = 0.0f, peak = __builtin_huge_valf();
    if (c < nc) {
      peak = -FLT_MAX;
      const uint2 cd = w.cand[c];
      const uint32_t map = cd.y & 0x7fffu;
      const int sg = (cd.y & kAuxNeg) ? -1 : 1;
      const MapDesc md = s.maps[map];
      const uint32_t *lv = s.levels + md.off + (size_t)st.level * md.w * md.h;
      const int cx = (int)(cd.x & 0xffffu), cy = (int)(cd.x >> 16);
      for (uint32_t j = 0; j < nk && peak < best_s; ++j) {
        const uint4 nr = w.nbr[j];
        const int qx = cx + sg * off_dx(w.off[j]), qy = cy + sg * off_dy(w.off[j]);
        float nps = lut4(lc, __vabsdiffu4(nr.y, texel(lv, md, qx, qy)), 0.0f);
        if (kG && s.guided) {
          const GuideDesc gd = s.gdesc[map];
          const uint32_t *gv = s.guides + gd.off + (size_t)st.level * gd.w * gd.h;
          uint32_t gt = kOutside;
          if ((unsigned)qx < gd.w && (unsigned)qy < gd.h) gt = gv[(size_t)qy * gd.w + qx];
          nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
        }
        score = __fadd_rn(score, __fmul_rn(nps, __uint_as_float(nr.w)));
        peak = fmaxf(peak, score);
      }
    }
    __syncwarp();
    take_signed(score, peak, base, best_s, best_i);
  }
}

__device__ __forceinline__ void add_cell_point(const SessionDev &s, int x, int y) {
  atomicAdd(&s.cells[(size_t)((y - s.coy) / kCell) * s.cgw + (x - s.cox) / kCell], 1u);
}

// A tree point in the cell counts, with its mirror copies where it has them
// (flush_resolved, ms.rs:306-328).
__device__ __forceinline__ void add_cells(const SessionDev &s, int x, int y, bool mirrors) {
  add_cell_point(s, x, y);
  if (!mirrors) return;
  if (x < s.x_l)
    add_cell_point(s, x + (int)s.W, y);
  else if (x > s.x_r)
    add_cell_point(s, x - (int)s.W, y);
  if (y < s.y_b)
    add_cell_point(s, x, y + (int)s.H);
  else if (y > s.y_t)
    add_cell_point(s, x, y - (int)s.H);
}

// update + flush_resolved of one item (ms.rs:296-377): its colour and state,
// its place in the resolved list, the bitmap, mirrors and cell counts.
__device__ __forceinline__ void commit_item(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                            const Result &r, bool count_evals = true) {
  const uint32_t p = r.pixel;
  if ((r.flags & kResBad) || p >= s.W * s.H) {
    set_err(s.err, kDevErrIndex);
    return;
  }
  s.state[p] = make_uint4(r.srcxy, r.idp, r.idm, r.idm);
  s.color[p] = r.color;
  if (count_evals && r.ncand) atomicAdd(s.evals, (unsigned long long)r.ncand);
  if (r.flags & kResAppend) {
    const uint32_t item = b.i0 + local;
    const uint32_t pos = b.n_res + (item - b.append_from);
    s.rscore[pos] = r.score;
    if (s.rank) return;  // k-NN made ahead: k_tree_append entered the point already
    s.resolved[pos] = p;
    int x, y;
    pixel_xy(s, p, x, y);
    atomicOr(&s.occ[(size_t)y * s.wpr + (x >> 5)], 1u << (x & 31));
    const bool mirrors = s.tiling && (r.flags & kResMirrors);
    if (mirrors) atomicOr(&s.mir[(size_t)y * s.wpr + (x >> 5)], 1u << (x & 31));
    add_cells(s, x, y, mirrors);
  }
}

// An item's result: committed at once when the batch holds only new items
// (b.fused_commit: no item of the batch is in the tree, so no other item
// reads its pixel, state or bit during the batch), else kept for k_commit.
__device__ __forceinline__ void emit_result(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                            const Result &r, bool count_evals = true) {
  if (b.fused_commit) {
    commit_item(s, st, b, local, r, count_evals);
  } else {
    b.res[local] = r;
    if (b.defer_tag && !(r.flags & kResBad) && r.pixel < s.W * s.H) {
      // what the commit will write, for the next step's readers (start_pixel)
      s.shadow[2 * (size_t)r.pixel] = make_uint4(b.defer_tag, r.color, 0u, 0u);
      s.shadow[2 * (size_t)r.pixel + 1] = make_uint4(r.srcxy, r.idp, r.idm, r.idm);
    }
  }
}

// The colour of a candidate's centre at the stage's level (its coordinates
// are valid).
__device__ __forceinline__ uint32_t centre_colour(const SessionDev &s, const StageDev &st, uint32_t map, uint32_t cxy) {
  const MapDesc md = s.maps[map];
  return __ldg(&s.levels[md.off + (size_t)st.level * md.w * md.h + (size_t)(cxy >> 16) * md.w + (cxy & 0xffffu)]);
}

// The winning candidate as an update (ms.rs:976-1001): source coordinate and
// map, patch id (the neighbour's for coherence candidates, the example flat
// index for random ones), score.
__device__ void write_result(const SessionDev &s, const StageDev &st, const WarpSmem &w, const BatchDev &b,
                             uint32_t local, uint32_t pixel, int px, int py, bool is_new, uint32_t nc, float best_s,
                             uint32_t best_i, bool count_evals = true) {
  const uint32_t aux = w.cand[best_i].y;
  const uint32_t map = aux & 0x7fffu;
  const uint32_t cxy = w.cand[best_i].x;
  uint32_t idp;
  if (aux & kAuxNeg) {
    idp = (cxy >> 16) * s.maps[map].w + (cxy & 0xffffu);
  } else {
    const uint32_t j = aux >> 16;
    const int32_t off = w.off[j];
    const int wx = wrap1(px + off_dx(off), (int)s.W), wy = wrap1(py + off_dy(off), (int)s.H);
    uint32_t unused;
    uint4 sv;
    start_pixel(s, b, (uint32_t)wy * s.W + (uint32_t)wx, false, unused, sv);
    idp = sv.y;
  }
  Result r;
  r.pixel = pixel;
  r.srcxy = cxy;
  r.idp = idp;
  r.idm = map;
  r.color = centre_colour(s, st, map, cxy);
  r.flags = (is_new ? kResAppend : 0u) | kResMirrors;
  r.score = best_s;
  r.ncand = nc;
  emit_result(s, st, b, local, r, count_evals);
}

// Result for an item with no resolved neighbour: resolve_at_random with the
// stage seed, appended without tiling mirrors (ms.rs:1002-1010, 473).
__device__ void write_random_result(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                    uint32_t pixel) {
  Pcg32 g = pcg_from_u64(st.stage_seed);
  uint64_t map64 = 0;
  uint32_t x = 0, y = 0;
  bool ok = gen_range_u64_bounded(g, s.n_maps, 256, map64);
  const uint32_t map = ok ? (uint32_t)map64 : 0u;
  const MapDesc md = s.maps[map];
  g = pcg_from_u64(st.stage_seed);
  ok = ok && gen_range_u32_bounded(g, md.w, 256, x);
  g = pcg_from_u64(st.stage_seed);
  ok = ok && gen_range_u32_bounded(g, md.h, 256, y);
  if (!ok) set_err(s.err, kDevErrNoSample);
  Result r;
  r.pixel = pixel;
  r.srcxy = x | (y << 16);
  r.idp = pixel;
  r.idm = map;
  r.color = centre_colour(s, st, map, r.srcxy);
  r.flags = kResAppend;
  r.score = 0.0f;
  r.ncand = 0;
  emit_result(s, st, b, local, r);
}

// A result that commit skips (an invalid map id was met; the reference
// panics there).
__device__ void write_bad_result(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t local,
                                 uint32_t pixel) {
  set_err(s.err, kDevErrIndex);
  Result r;
  r.pixel = pixel;
  r.srcxy = 0;
  r.idp = 0;
  r.idm = 0;
  r.color = 0;
  r.flags = kResBad;
  r.score = 0.0f;
  r.ncand = 0;
  emit_result(s, st, b, local, r);
}

// kLean: sessions without guides only (the guide terms compiled out).  Eight
// blocks of four warps per SM at 64 registers: nine at 56 ran the last stage
// of the remix in 0.95 against 0.82 ms (more items wait behind a launch's
// slowest ones).
//
// What bounds it: a step's warps take 3 to 8 items each, one after another,
// so the latency of an item (dependent gathers, then the issue slots its
// warps share) and the launch's tail; DRAM carries a few percent.  50 neighbours propose 3 to 8 different coherence candidates
// on the benchmark workloads, and the first of them costs exactly 0 for 12 to
// 49% of the items, which ends the item.  Distances stay in integers and f32
// pairs: an f64 instruction takes 18 cycles of an SM.  Repeats are found with
// a 32-bit __match_any_sync: 2 cycles of the SM per distinct value, 4 with 64
// bits (an atomicMin per lane into a shared hash table: 1 per lane of a slot,
// and most lanes share one).  Resolves of 2048^2 tiling: 25.8 -> 21.5 ms.
template <bool kLean, int kMode>
__device__ __forceinline__ void resolve_body(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t vb,
                                             uint32_t vg) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float tab_ff[128];
  float *lc = (float *)smem;
  float *lg = lc + 256;
  for (int i = threadIdx.x; i < 512; i += blockDim.x) lc[i] = st.lut[i];
  tab_ff[threadIdx.x] = g_exp2_ff[threadIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const WarpSmem w = carve(smem + 2048 + (size_t)warp * warp_smem_bytes(s.k, s.m), s.k, s.m);
  __syncthreads();
  const uint32_t nb = b.i1 - b.i0;
  const uint32_t grid_warps = vg * kResolveWarps;
  uint32_t evals = 0;  // candidates of the items committed here, added once at the end
  // The next item of this warp: the grid stride, or (BatchDev::work_ctr) the
  // next one nobody has taken once every warp has had its first (asked for
  // at an item's end: asked for at its start, the item waits behind a slow
  // one; remix 0.95 against 0.87 ms in the last stage).  One counter serves
  // an item per 0.95 ns at best, so there are kWorkCtrs of them (no more than
  // blocks), each for the items of one residue; a block uses its own.
  const uint32_t ctrs = min(kWorkCtrs, vg), res = vb % ctrs;
  const uint32_t res_warps = ((vg - res + ctrs - 1) / ctrs) * kResolveWarps;
  uint32_t local = vb * kResolveWarps + warp;
  if (b.work_ctr) local = (vb / ctrs * kResolveWarps + warp) * ctrs + res;
  auto take = [&](uint32_t cur) -> uint32_t {
    if (!b.work_ctr) return cur + grid_warps;
    uint32_t v = 0;
    if (lane == 0) v = (atomicAdd(b.work_ctr + res * kWorkCtrStride, 1u) + res_warps) * ctrs + res;
    return __shfl_sync(0xffffffffu, v, 0);
  };
  for (; local < nb; local = take(local)) {
    const uint32_t item = b.i0 + local;
    const uint32_t pixel = st.items[item];
    const uint32_t nk = s.k ? b.ncnt[local] : 0u;
    if (nk == 0) {
      // no resolved neighbours: resolve_at_random with the stage seed, kept
      // in the resolved list without tiling mirrors (ms.rs:1002-1010, 473)
      if (lane == 0) write_random_result(s, st, b, local, pixel);
      continue;
    }
    int px, py;
    pixel_xy(s, pixel, px, py);
    const int32_t *nbo = b.nbuf + (size_t)local * s.k;
    const double avg = b.mean[local];
    const FfMean fm = ts_ff_mean(avg);
    // neighbours: offsets, weights, own pattern, coherence candidates.
    // With `dedupe`, a coherence candidate equal to an earlier one (same
    // source and map) is left out: its cost equals the earlier one's, so it
    // can neither beat it nor tie it with a lower index, and the reference's
    // winner is the same without it.  The exact sequential form for
    // non-finite costs keeps every candidate.
    bool nan_w = false;
    int maxoff = 0;
    uint32_t ncoh = 0, ncoh_all = 0;
    bool bad_map = false;
    auto coherence = [&](bool dedupe) {
      ncoh = ncoh_all = 0;
      for (uint32_t j0 = 0; j0 < nk; j0 += kWarp) {
        const uint32_t j = j0 + lane;
        bool valid = false;
        uint32_t cxy = 0, aux = 0;
        if (j < nk) {
          const int32_t off = nbo[j];
          const float wv = item_weight(s, b, local, nb, px, py, j, off, avg, fm, tab_ff);
          nan_w |= (wv != wv);
          valid = neighbour_records<!kLean>(s, st, b, px, py, j, off, wv, w, cxy, aux, maxoff, bad_map);
        }
        bool keep = valid;
        if (dedupe) {
          const uint32_t map = aux & 0x7fffu, vm = __ballot_sync(0xffffffffu, valid);
          uint32_t same;  // lanes with the same source and map
          if (s.n_maps <= 16)
            same = __match_any_sync(0xffffffffu, (cxy & 0x3fffu) | ((cxy >> 16) << 14) | (map << 28));
          else
            same = __match_any_sync(0xffffffffu, ((unsigned long long)map << 32) | cxy);
          if (same & vm & lt) keep = false;  // a lower lane holds it
          for (uint32_t i = 0; i < ncoh; ++i) {
            const uint2 c1 = w.cand[i];
            if (c1.x == cxy && ((c1.y ^ aux) & 0x7fffu) == 0u) keep = false;
          }
        }
        ncoh_all += __popc(__ballot_sync(0xffffffffu, valid));
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        if (keep) w.cand[ncoh + __popc(bal & lt)] = make_uint2(cxy, aux);
        ncoh += __popc(bal);
        __syncwarp();
      }
    };
    coherence(!costs_exact<kMode>(st));
    const bool nan_any = __any_sync(0xffffffffu, nan_w);
    if (!costs_exact<kMode>(st) && nan_any) coherence(false);
    if (__any_sync(0xffffffffu, bad_map)) {
      // the reference panics on this index; record the error and leave the
      // pixel untouched (commit skips results with an invalid map)
      if (lane == 0) write_bad_result(s, st, b, local, pixel);
      continue;
    }
    // random candidates after the coherence ones
    const uint2 *rc = st.rcand + (size_t)item * s.m;
    for (uint32_t t = lane; t < s.m; t += kWarp) w.cand[ncoh + t] = random_candidate(s, rc, t);
    const bool slow = costs_exact<kMode>(st) || nan_any;
    maxoff = __reduce_max_sync(0xffffffffu, maxoff);
    const bool padded = maxoff <= kPad && !s.guide_dims_differ;
    __syncwarp();
    const uint32_t nc = ncoh + s.m;
    float best_s = FLT_MAX;
    uint32_t best_i = 0;
    if (!slow && costs_in_order<kMode>(st)) {
      best_in_order<!kLean>(s, st, w, lc, lg, nk, nc, best_s, best_i);
    } else if (!slow) {
      // candidate 0 first: its terms on all lanes, their in-order sum on
      // every lane; it wins ties with every later candidate, so the rest run
      // against min(S_0, f32::MAX) from the start, and a cost of 0 ends the
      // item (no term is negative)
      const float s0 = candidate0_score<kWarp, !kLean>(s, st, w, lc, lg, nk, lane, 0xffffffffu);
      if (s0 < best_s) best_s = s0;
      for (uint32_t base = 1; base < nc && best_s > 0.0f; base += kWarp) {
        const uint32_t c = base + lane;
        float sc = __builtin_huge_valf(), v = 0.0f;
        if (c < nc) {
          const uint2 cd = w.cand[c];
          bool alive;
          if (!padded) {
            alive = candidate_cost<!kLean>(s, st, w, lc, lg, nk, cd.x, cd.y, best_s, v);
          } else {
            const uint64_t centre = padded_centre(s.maps[cd.y & 0x7fffu], st.level, cd.x);
            const bool neg = (cd.y & kAuxNeg) != 0;
            if (!kLean && s.guided)
              alive = candidate_cost_padded<true>(s, st, w, lc, lg, nk, centre, neg, best_s, v);
            else
              alive = candidate_cost_padded<false>(s, st, w, lc, lg, nk, centre, neg, best_s, v);
          }
          if (alive) sc = v;
        }
        // the round's lowest cost, its first lane
        const float lo = warp_min(sc);
        if (lo < best_s) {
          best_s = lo;
          best_i = base + __ffs(__ballot_sync(0xffffffffu, sc == lo)) - 1;
        }
      }
    } else if (lane == 0) {
      sequential_best<!kLean>(s, st, w, lc, lg, nk, nc, best_s, best_i);
    }
    if (lane == 0)
      write_result(s, st, w, b, local, pixel, px, py, item >= st.redo, ncoh_all + s.m, best_s, best_i, false);
    evals += ncoh_all + s.m;
    __syncwarp();  // the records and candidates are rebuilt for the next item
  }
  // (a batch left to a later commit is counted there)
  if (b.fused_commit && lane == 0 && evals) atomicAdd(s.evals, (unsigned long long)evals);
}


// ---------------------------------------------------------------------------
// resolve, team form: one CTA of T threads per item, one candidate per
// thread.  Candidate 0's exact score is computed first (its neighbour terms
// in parallel, their in-order sum on one thread); every other candidate then
// runs against min(S_0, its thread's earlier results) and stops as soon as
// its partial sum reaches that bound; a block-wide first-index argmin picks
// the winner.  The first strict minimum of the reference never stops early
// (every bound it meets is larger, or equal with a later index), so the
// result is the reference's.  Latency per item is about one candidate's
// evaluation, which suits batches too small to fill the GPU with warps.
// ---------------------------------------------------------------------------
template <int T, bool kFull, int kMode>
__device__ __forceinline__ void resolve_team_body(const SessionDev &s, const StageDev &st, const BatchDev &b,
                                                  uint32_t vb, uint32_t vg) {
  constexpr int NW = T / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float tab_ff[128];
  __shared__ uint32_t wcnt[NW];
  __shared__ float red_s[NW];
  __shared__ uint32_t red_i[NW];
  __shared__ int sh_flags, sh_maxoff;
  __shared__ float sh_s0;
  float *lc = (float *)smem;
  float *lg = lc + 256;
  for (int i = threadIdx.x; i < 512; i += T) lc[i] = st.lut[i];
  for (int i = threadIdx.x; i < 128; i += T) tab_ff[i] = g_exp2_ff[i];
  const WarpSmem w = carve(smem + 2048, s.k, s.m);
  float *term = (float *)(smem + 2048 + warp_smem_bytes(s.k, s.m));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t nb = b.i1 - b.i0;
  __syncthreads();
  for (uint32_t local = vb; local < nb; local += vg) {
    const uint32_t item = b.i0 + local;
    const uint32_t pixel = st.items[item];
    int px, py;
    pixel_xy(s, pixel, px, py);
    const bool is_new = item >= st.redo;
    const uint32_t nk = s.k ? b.ncnt[local] : 0u;
    if (nk == 0) {
      if (tid == 0) write_random_result(s, st, b, local, pixel);
      continue;
    }
    if (tid == 0) {
      sh_flags = 0;
      sh_maxoff = 0;
    }
    __syncthreads();
    const int32_t *nbo = b.nbuf + (size_t)local * s.k;
    const double avg = b.mean[local];
    const FfMean fm = ts_ff_mean(avg);
    bool nan_w = false, bad_map = false;
    int maxoff = 0;
    uint32_t ncoh = 0;
    for (uint32_t j0 = 0; j0 < nk; j0 += T) {
      const uint32_t j = j0 + tid;
      bool valid = false;
      uint32_t cxy = 0, aux = 0;
      if (j < nk)
        valid = neighbour_setup(s, st, b, local, nb, px, py, j, nbo[j], avg, fm, tab_ff, w, cxy, aux, nan_w,
                                maxoff, bad_map);
      // order-preserving compaction of the valid coherence candidates
      const uint32_t bal = __ballot_sync(0xffffffffu, valid);
      if (lane == 0) wcnt[warp] = __popc(bal);
      __syncthreads();
      uint32_t base = ncoh, total = 0;
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        if (i < warp) base += wcnt[i];
        total += wcnt[i];
      }
      if (valid) {
        const uint32_t slot = base + __popc(bal & lt);
        w.cand[slot] = make_uint2(cxy, aux);
      }
      ncoh += total;
      __syncthreads();
    }
    if (nan_w) atomicOr(&sh_flags, 1);
    if (bad_map) atomicOr(&sh_flags, 2);
    if (maxoff) atomicMax(&sh_maxoff, maxoff);
    const uint2 *rc = st.rcand + (size_t)item * s.m;
    for (uint32_t t = tid; t < s.m; t += T) {
      const uint2 v = use_rcand(s, rc[t]);
      w.cand[ncoh + t] = make_uint2(v.x, v.y | kAuxNeg | (t << 16));
    }
    __syncthreads();
    if (sh_flags & 2) {
      if (tid == 0) write_bad_result(s, st, b, local, pixel);
      __syncthreads();
      continue;
    }
    const bool slow = st.slow_lut || (sh_flags & 1);
    const bool padded = sh_maxoff <= kPad && !s.guide_dims_differ;
    const uint32_t nc = ncoh + s.m;
    float best_s = FLT_MAX;
    uint32_t best_i = 0;
    if (!slow && kFull && padded) {
      // every term nps(c, j) * w_j in parallel, then each candidate's
      // in-order sum on one thread: the reference's scores, all of them.
      // Padded planes: each candidate's plane offset once, then eight texel
      // loads in flight per thread before their terms are formed.
      unsigned long long *cb = (unsigned long long *)(term + (((size_t)nk * nc + 1) & ~(size_t)1));
      for (uint32_t c = tid; c < nc; c += T) {
        const uint32_t cxy = w.cand[c].x, aux = w.cand[c].y;
        cb[c] = padded_centre(s.maps[aux & 0x7fffu], st.level, cxy) | ((aux & kAuxNeg) ? (1ull << 63) : 0ull);
      }
      __syncthreads();
      const uint32_t total = nc * nk;
      for (uint32_t i0 = tid; i0 < total; i0 += 8 * T) {
        uint32_t tx[8], gx[8], ii[8], jj[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint32_t i = i0 + (uint32_t)u * T;
          ii[u] = i;
          if (i < total) {
            const uint32_t c = i / nk;
            jj[u] = i - c * nk;
            const unsigned long long v = cb[c];
            const int lj = (int32_t)w.nbr[jj[u]].x, lin = (v >> 63) ? -lj : lj;
            const size_t off = (size_t)(v & 0x7fffffffffffffffull) + lin;
            tx[u] = __ldg(s.plevels + off);
            if (s.guided) gx[u] = __ldg(s.pguides + off);
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (ii[u] < total) {
            const uint4 nr = w.nbr[jj[u]];
            float nps = lut4r(lc, __vabsdiffu4(nr.y, tx[u]), 0.0f, st.opaque);
            if (s.guided) nps = lut4r(lg, __vabsdiffu4(nr.z, gx[u]), nps, st.opaque);
            term[ii[u]] = __fmul_rn(nps, __uint_as_float(nr.w));
          }
        }
      }
    }
    if (!slow && kFull && !padded) {
      // the same with bounds-checked gathers (far neighbours or guides of
      // other sizes); consecutive threads take consecutive neighbours of one
      // candidate
      uint32_t c = tid / nk, j = tid - c * nk;
      const uint32_t dc = T / nk, dj = T - dc * nk;
      for (uint32_t i = tid; i < nc * nk; i += T) {
        const uint32_t cxy = w.cand[c].x, aux = w.cand[c].y;
        const uint32_t map = aux & 0x7fffu;
        const int sg = (aux & kAuxNeg) ? -1 : 1;
        const MapDesc md = s.maps[map];
        const uint4 nr = w.nbr[j];
        const int qx = (int)(cxy & 0xffffu) + sg * off_dx(w.off[j]);
        const int qy = (int)(cxy >> 16) + sg * off_dy(w.off[j]);
        uint32_t t = kOutside;
        if ((unsigned)qx < md.w && (unsigned)qy < md.h)
          t = __ldg(&s.levels[md.off + (size_t)st.level * md.w * md.h + (size_t)qy * md.w + qx]);
        float nps = lut4(lc, __vabsdiffu4(nr.y, t), 0.0f);
        if (s.guided) {
          const GuideDesc gd = s.gdesc[map];
          uint32_t gt = kOutside;
          if ((unsigned)qx < gd.w && (unsigned)qy < gd.h)
            gt = __ldg(&s.guides[gd.off + (size_t)st.level * gd.w * gd.h + (size_t)qy * gd.w + qx]);
          nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
        }
        term[i] = __fmul_rn(nps, __uint_as_float(nr.w));
        c += dc;
        j += dj;
        if (j >= nk) {
          j -= nk;
          ++c;
        }
      }
    }
    if (!slow && kFull) {
      __syncthreads();
      float my_s = FLT_MAX;
      uint32_t my_i = 0xffffffffu;
      for (uint32_t cc = tid; cc < nc; cc += T) {
        float sc = 0.0f;
        const float *tc = term + (size_t)cc * nk;
        for (uint32_t jj = 0; jj < nk; ++jj) sc = __fadd_rn(sc, tc[jj]);
        if (sc < my_s) {  // first strict minimum among this thread's candidates
          my_s = sc;
          my_i = cc;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, my_s, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, my_i, o);
        if (ov < my_s || (ov == my_s && oi < my_i)) {
          my_s = ov;
          my_i = oi;
        }
      }
      if (lane == 0) {
        red_s[warp] = my_s;
        red_i[warp] = my_i;
      }
      __syncthreads();
      best_s = red_s[0];
      best_i = red_i[0];
      for (int i = 1; i < NW; ++i) {
        if (red_s[i] < best_s || (red_s[i] == best_s && red_i[i] < best_i)) {
          best_s = red_s[i];
          best_i = red_i[i];
        }
      }
      if (best_i == 0xffffffffu) {  // no score below f32::MAX: the reference keeps candidate 0
        best_s = FLT_MAX;
        best_i = 0;
      }
    } else if (!slow) {
      // S_0: candidate 0's terms nps_j * w_j in parallel, summed in order
      {
        const uint32_t cxy0 = w.cand[0].x, aux0 = w.cand[0].y;
        const uint32_t map = aux0 & 0x7fffu;
        const bool neg = (aux0 & kAuxNeg) != 0;
        const MapDesc md = s.maps[map];
        const uint32_t *lv = s.levels + md.off + (size_t)st.level * md.w * md.h;
        const int cx = (int)(cxy0 & 0xffffu), cy = (int)(cxy0 >> 16);
        for (uint32_t j = tid; j < nk; j += T) {
          const uint4 nr = w.nbr[j];
          int dx = off_dx(w.off[j]), dy = off_dy(w.off[j]);
          if (neg) {
            dx = -dx;
            dy = -dy;
          }
          const int qx = cx + dx, qy = cy + dy;
          float nps = lut4(lc, __vabsdiffu4(nr.y, texel(lv, md, qx, qy)), 0.0f);
          if (s.guided) {
            const GuideDesc gd = s.gdesc[map];
            const uint32_t *gv = s.guides + gd.off + (size_t)st.level * gd.w * gd.h;
            uint32_t gt = kOutside;
            if ((unsigned)qx < gd.w && (unsigned)qy < gd.h) gt = __ldg(&gv[(size_t)qy * gd.w + qx]);
            nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
          }
          term[j] = __fmul_rn(nps, __uint_as_float(nr.w));
        }
        __syncthreads();
        if (tid == 0) {
          float sc = 0.0f;
          for (uint32_t j = 0; j < nk; ++j) sc = __fadd_rn(sc, term[j]);
          sh_s0 = sc;
        }
        __syncthreads();
      }
      float my_s = sh_s0;
      uint32_t my_i = 0;
      for (uint32_t c = 1 + tid; c < nc; c += T) {
        float sc;
        bool alive;
        const uint2 cd = w.cand[c];
        const bool neg = (cd.y & kAuxNeg) != 0;
        if (!padded)
          alive = candidate_cost(s, st, w, lc, lg, nk, cd.x, cd.y, my_s, sc);
        else if (s.guided)
          alive = candidate_cost_padded<true>(s, st, w, lc, lg, nk, padded_centre(s.maps[cd.y & 0x7fffu], st.level, cd.x),
                                              neg, my_s, sc);
        else
          alive = candidate_cost_padded<false>(s, st, w, lc, lg, nk, padded_centre(s.maps[cd.y & 0x7fffu], st.level, cd.x),
                                               neg, my_s, sc);
        if (alive) {
          my_s = sc;
          my_i = c;
        }
      }
      // first index of the minimum over the block
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, my_s, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, my_i, o);
        if (ov < my_s || (ov == my_s && oi < my_i)) {
          my_s = ov;
          my_i = oi;
        }
      }
      if (lane == 0) {
        red_s[warp] = my_s;
        red_i[warp] = my_i;
      }
      __syncthreads();
      best_s = red_s[0];
      best_i = red_i[0];
      for (int i = 1; i < NW; ++i) {
        if (red_s[i] < best_s || (red_s[i] == best_s && red_i[i] < best_i)) {
          best_s = red_s[i];
          best_i = red_i[i];
        }
      }
    } else if (costs_in_order<kMode>(st) && !(sh_flags & 1)) {
      if (warp == 0) best_in_order(s, st, w, lc, lg, nk, nc, best_s, best_i);
    } else if (tid == 0) {
      sequential_best(s, st, w, lc, lg, nk, nc, best_s, best_i);
    }
    if (tid == 0) write_result(s, st, w, b, local, pixel, px, py, is_new, nc, best_s, best_i);
    __syncthreads();
  }
}

// update + flush_resolved for a batch (ms.rs:296-377): one thread per item.

__device__ __forceinline__ void commit_body(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t vb) {
  const uint32_t local = vb * blockDim.x + threadIdx.x;
  const uint32_t nb = b.i1 - b.i0;
  if (local >= nb) return;
  commit_item(s, st, b, local, b.res[local]);
}

// next_pyramid_level (ms.rs:687-700)
__device__ __forceinline__ void level_switch_body(const SessionDev &s, uint32_t level, uint32_t n_res, uint32_t vb) {
  const uint32_t e = vb * blockDim.x + threadIdx.x;
  if (e >= n_res) return;
  const uint32_t p = s.resolved[e];
  const uint4 sv = s.state[p];
  if (sv.w >= s.n_maps) {
    set_err(s.err, kDevErrIndex);
    return;
  }
  const MapDesc md = s.maps[sv.w];
  const uint32_t x = sv.x & 0xffffu, y = sv.x >> 16;
  if (x >= md.w || y >= md.h) {  // a coordinate drawn for another example (the reference panics)
    set_err(s.err, kDevErrIndex);
    return;
  }
  s.color[p] = s.levels[md.off + (size_t)level * md.w * md.h + (size_t)y * md.w + x];
}

// Initial state of the random-init pixels (Generator::new, ms.rs:427-475):
// list[6i..6i+6] = {pixel, colour, state.x, state.y, state.z, state.w}.
__global__ void k_scatter_init(const uint32_t *list, uint32_t n, uint32_t *color, uint4 *state, uint32_t *res) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t *e = list + (size_t)i * 6;
  color[e[0]] = e[1];
  state[e[0]] = make_uint4(e[2], e[3], e[4], e[5]);
  res[i] = e[0];
}

// Initial state of an inpainting run (Generator::new_from_inpaint,
// ms.rs:236-293), a warp per 32 pixels of a row: a locked pixel's state, its
// place in the resolved list and the tree, and the others' place in the
// unresolved list (both in pixel order; a random init's picks have shortened
// the latter, and k_pick_over puts in what they moved).  in.before counts the pixels to synthesise before each
// word.  The host's loops took 1.9 ms of a 512^2 run, beside the upload of
// colours and states.
__global__ void k_inpaint_init(const __grid_constant__ SessionDev s, const __grid_constant__ InpaintDev in) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (w >= s.wpr * s.H) return;
  const uint32_t y = w / s.wpr, x = (w - y * s.wpr) * 32u + lane;
  const uint32_t open = in.open[w], locked = __ballot_sync(0xffffffffu, x < s.W) & ~open;
  if (lane == 0 && locked) {
    s.occ[w] |= locked;  // beside the random init's bits
    if (s.tiling) s.mir[w] |= locked;
  }
  if (x >= s.W) return;
  const uint32_t p = y * s.W + x, rank = in.before[w] + (uint32_t)__popc(open & ((1u << lane) - 1u));
  if ((open >> lane) & 1u) {
    s.state[p] = make_uint4(0, 0, 0, 0);
    if (rank < in.n_un) in.un[rank] = p;
  } else {
    s.state[p] = make_uint4(x | (y << 16), 0, 0, in.map);
    s.resolved[p - rank] = p;
    add_cells(s, (int)x, (int)y, s.tiling);
  }
}

// ---------------------------------------------------------------------------
// The pick chain of a stage (pick_random_unresolved, ms.rs:380-389): new item
// q takes entry d(q) = Pcg32(seed + redo + q).gen_range(0..len0 - q) of the
// unresolved list, whose last entry then moves there.  The draws do not
// depend on the list, and neither does the list's history: what entry p holds
// at time t is what the latest earlier pick t' < t with d(t') = p put there,
// that is what the then last entry, len0 - 1 - t', held at time t'; with no
// such pick it is the entry at the stage's start.  So every pick follows its
// own chain backwards (a few hops: an entry is drawn about once), with the
// picks of each entry linked in any order.  The host's chain of swap-removes
// takes some 10 ns a pick, 27 ms for the last stage of a 2048^2 output.
// ---------------------------------------------------------------------------
constexpr uint32_t kPickChainThreads = 1024;
__global__ void k_pick_init(uint32_t *un, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) un[i] = i;
}
__global__ void k_pick_over(uint32_t *un, const uint32_t *over, uint32_t n_over) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_over; i += gridDim.x * blockDim.x)
    un[over[2 * (size_t)i]] = over[2 * (size_t)i + 1];
}
__device__ __forceinline__ void pick_draw(const PickStage &ps, uint32_t first, uint32_t step) {
  for (uint32_t i = first; i < ps.redo + ps.n_new; i += step) {
    if (i < ps.redo) {
      const uint32_t v = ps.redo_from[i];
      ps.items[i] = v;
      if (ps.append_redo) ps.resolved[i] = v;
      continue;
    }
    const uint32_t q = i - ps.redo;
    Pcg32 g = pcg_from_u64(ps.seed + (uint64_t)i);
    uint64_t v = 0;
    gen_range_u64_bounded(g, ps.len0 - q, 1u << 20, v);  // (a draw is rejected with probability below 1/2)
    ps.draw[q] = (uint32_t)v;
    ps.next[q] = atomicExch(&ps.head[v], q + 1u);
  }
}
// What entry p of the unresolved list holds at time t.
__device__ __forceinline__ uint32_t pick_follow(const PickStage &ps, uint32_t p, uint32_t t) {
  for (;;) {  // t falls with every hop
    uint32_t last = 0;  // the latest earlier pick of p, plus one
    for (uint32_t e = ps.head[p]; e; e = ps.next[e - 1u])
      if (e <= t && e > last) last = e;
    if (last == 0) return ps.un[p];
    t = last - 1u;
    p = ps.len0 - 1u - t;
  }
}
__device__ __forceinline__ void pick_follow_all(const PickStage &ps, uint32_t first, uint32_t step) {
  // threads [n_new, len0): the entries of the list after the stage
  for (uint32_t i = first; i < ps.len0; i += step) {
    if (i < ps.n_new) {
      const uint32_t v = pick_follow(ps, ps.draw[i], i);
      ps.items[ps.redo + i] = v;
      ps.resolved[(ps.append_redo ? ps.redo : 0u) + i] = v;
    } else {
      ps.un_next[i - ps.n_new] = pick_follow(ps, i - ps.n_new, ps.n_new);
    }
  }
}

__global__ void k_pick_draw(const __grid_constant__ PickStage ps) {
  pick_draw(ps, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void k_pick_follow(const __grid_constant__ PickStage ps) {
  pick_follow_all(ps, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
// The whole chain of a run of few items, a block per run: one launch instead
// of three calls a stage.
__global__ void __launch_bounds__(kPickChainThreads) k_pick_chain(const PickChain *chains) {
  const PickChain &ch = chains[blockIdx.x];
  for (uint32_t i = threadIdx.x; i < ch.n_un; i += blockDim.x) ch.un[i] = i;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ch.n_over; i += blockDim.x) ch.un[ch.over[2 * i]] = ch.over[2 * i + 1];
  __syncthreads();
  for (uint32_t q = 0; q < ch.n; ++q) {
    const PickStage &ps = ch.st[q];
    for (uint32_t i = threadIdx.x; i < ps.len0; i += blockDim.x) ps.head[i] = 0;
    __syncthreads();
    pick_draw(ps, threadIdx.x, blockDim.x);
    __syncthreads();
    if (ps.n_new) pick_follow_all(ps, threadIdx.x, blockDim.x);
    __syncthreads();
  }
}

// CoordinateTransform::apply (lib.rs:176-212): output pixel i takes texel
// (x, y) of source map `map`, (x, y, map) = buf[3i..3i+3].  maps[m] =
// {texel offset low, high, width, height}.  An entry outside the maps (the
// reference panics in get_pixel) writes 0 and sets *err.
__global__ void k_transform_apply(const uint32_t *buf, size_t n, const uint32_t *texels, const uint4 *maps,
                                  uint32_t n_maps, uint32_t *out, int *err) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = buf[3 * i], y = buf[3 * i + 1], m = buf[3 * i + 2];
    uint32_t v = 0;
    if (m < n_maps) {
      const uint4 md = maps[m];
      if (x < md.z && y < md.w)
        v = texels[(((size_t)md.y << 32) | md.x) + (size_t)y * md.z + x];
      else
        set_err(err, 1);
    } else {
      set_err(err, 1);
    }
    out[i] = v;
  }
}

// Debug maps (ms.rs:604-653): the patch-id and map-id colours of every
// pixel, and the uncertainty colour of every resolved pixel (the others
// stay 0).  Ids combine in u32 arithmetic, which wraps as the reference's
// release build does.
__global__ void k_id_maps(const uint32_t *ids, size_t n, uint32_t *patch_rgba, uint32_t *map_rgba) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t p = ids[2 * i], m = ids[2 * i + 1];
    patch_rgba[i] = (uint32_t)id_colour(p) | ((uint32_t)id_colour(p * 5u + 21u) << 8) |
                    ((uint32_t)id_colour(p / 4u + 12u) << 16) | 0xff000000u;
    map_rgba[i] = (uint32_t)id_colour((uint64_t)m * 200u) | ((uint32_t)id_colour(m * 5u + 341u) << 8) |
                  ((uint32_t)id_colour(m * 1200u - 35412u) << 16) | 0xff000000u;
  }
}

__global__ void k_uncertainty(const uint32_t *flat, const float *score, size_t n_res, size_t n_px, uint32_t *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_res; i += (size_t)gridDim.x * blockDim.x) {
    // (score.min(1.0) * 255.0) as u8: f32::min returns the other operand
    // for NaN, and `as` truncates and saturates
    const float v = __fmul_rn(fminf(score[i], 1.0f), 255.0f);
    const uint32_t ns = v >= 255.0f ? 255u : (v > 0.0f ? (uint32_t)v : 0u);
    if (flat[i] < n_px) out[flat[i]] = ns | ((255u - ns) << 8) | 0xff000000u;
  }
}

// Automatic guide maps (utils.rs:101-183).  DynamicImage::grayscale of RGBA8
// (image 0.23 rgb_to_luma): l = 0.2126 R + 0.7152 G + 0.0722 B in f32, left
// to right, truncated to u8 (NumCast), with the histogram of l; the
// histogram of channel 0 of an RGBA8 image; and the histogram-matching map
// applied as (n, n, n, 255).
__global__ void k_luma_hist(const uint32_t *src, size_t n, uint8_t *luma, uint32_t *hist) {
  __shared__ uint32_t h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t p = src[i];
    float l = __fmul_rn(0.2126f, (float)(p & 0xffu));
    l = __fadd_rn(l, __fmul_rn(0.7152f, (float)((p >> 8) & 0xffu)));
    l = __fadd_rn(l, __fmul_rn(0.0722f, (float)((p >> 16) & 0xffu)));
    const uint32_t v = l >= 255.0f ? 255u : (uint32_t)l;
    luma[i] = (uint8_t)v;
    atomicAdd(&h[v], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

__global__ void k_hist_r(const uint32_t *src, size_t n, uint32_t *hist) {
  __shared__ uint32_t h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    atomicAdd(&h[src[i] & 0xffu], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

__global__ void k_apply_map(const uint8_t *luma, size_t n, const uint8_t *map, uint32_t *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = map[luma[i]];
    out[i] = v | (v << 8) | (v << 16) | 0xff000000u;
  }
}

// vertical_sample: u8 RGBA -> f32 RGBA, new height nh.
__global__ void k_resize_v(const uint8_t *src, uint32_t w, uint32_t h, float *tmp, uint32_t nh, const uint4 *taps,
                           const float *wts) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t oy = blockIdx.y;
  if (x >= w || oy >= nh) return;
  const uint4 t = taps[oy];
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
  for (uint32_t i = 0; i < t.y; ++i) {
    const uchar4 p = *(const uchar4 *)(src + ((size_t)(t.x + i) * w + x) * 4);
    const float wt = wts[t.z + i];
    a0 = __fadd_rn(a0, __fmul_rn((float)p.x, wt));
    a1 = __fadd_rn(a1, __fmul_rn((float)p.y, wt));
    a2 = __fadd_rn(a2, __fmul_rn((float)p.z, wt));
    a3 = __fadd_rn(a3, __fmul_rn((float)p.w, wt));
  }
  *(float4 *)(tmp + ((size_t)oy * w + x) * 4) = make_float4(a0, a1, a2, a3);
}

__device__ __forceinline__ uint8_t to_u8(float v) {
  v = v < 0.0f ? 0.0f : v;
  v = v > 255.0f ? 255.0f : v;
  return (uint8_t)roundf(v);
}

// horizontal_sample: f32 RGBA -> u8 RGBA (clamped, rounded half away from 0).
__global__ void k_resize_h(const float *tmp, uint32_t w, uint32_t nh, uint8_t *dst, uint32_t nw, const uint4 *taps,
                           const float *wts) {
  const uint32_t ox = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t y = blockIdx.y;
  if (ox >= nw || y >= nh) return;
  const uint4 t = taps[ox];
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
  for (uint32_t i = 0; i < t.y; ++i) {
    const float4 p = *(const float4 *)(tmp + ((size_t)y * w + t.x + i) * 4);
    const float wt = wts[t.z + i];
    a0 = __fadd_rn(a0, __fmul_rn(p.x, wt));
    a1 = __fadd_rn(a1, __fmul_rn(p.y, wt));
    a2 = __fadd_rn(a2, __fmul_rn(p.z, wt));
    a3 = __fadd_rn(a3, __fmul_rn(p.w, wt));
  }
  uchar4 o;
  o.x = to_u8(a0);
  o.y = to_u8(a1);
  o.z = to_u8(a2);
  o.w = to_u8(a3);
  *(uchar4 *)(dst + ((size_t)y * nw + ox) * 4) = o;
}

// The job owning block b of a pass: jobs sorted by first block, one ballot
// per 32 (block0 selects the pass's column).
template <bool kV>
__device__ __forceinline__ uint32_t find_job(const ResizeJob *jobs, uint32_t n, uint32_t b) {
  const int lane = threadIdx.x & 31;
  uint32_t j = 0;
  for (uint32_t c = 0; c < n; c += 32) {
    const uint32_t i = c + lane;
    const bool le = i < n && (kV ? jobs[i].block0_v : jobs[i].block0_h) <= b;
    const uint32_t bal = __ballot_sync(0xffffffffu, le);
    j = c + __popc(bal) - 1;
    if (bal != 0xffffffffu) break;
  }
  return j;
}

// k_resize_v over many jobs: job blocks laid out as cdiv(w, 128) x nh.
__global__ void k_resize_v_jobs(const ResizeJob *jobs, uint32_t n) {
  const uint32_t j = find_job<true>(jobs, n, blockIdx.x);
  const ResizeJob jb = jobs[j];
  const uint32_t lb = blockIdx.x - jb.block0_v, bx = (jb.w + 127) / 128;
  const uint32_t x = (lb % bx) * 128 + threadIdx.x, oy = lb / bx;
  if (x >= jb.w || oy >= jb.nh) return;
  const uint4 t = jb.tv[oy];
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
  for (uint32_t i = 0; i < t.y; ++i) {
    const uchar4 p = *(const uchar4 *)(jb.src + ((size_t)(t.x + i) * jb.w + x) * 4);
    const float wt = jb.wv[t.z + i];
    a0 = __fadd_rn(a0, __fmul_rn((float)p.x, wt));
    a1 = __fadd_rn(a1, __fmul_rn((float)p.y, wt));
    a2 = __fadd_rn(a2, __fmul_rn((float)p.z, wt));
    a3 = __fadd_rn(a3, __fmul_rn((float)p.w, wt));
  }
  *(float4 *)(jb.tmp + ((size_t)oy * jb.w + x) * 4) = make_float4(a0, a1, a2, a3);
}

// k_resize_h over many jobs: job blocks laid out as cdiv(nw, 128) x nh.
__global__ void k_resize_h_jobs(const ResizeJob *jobs, uint32_t n) {
  const uint32_t j = find_job<false>(jobs, n, blockIdx.x);
  const ResizeJob jb = jobs[j];
  const uint32_t lb = blockIdx.x - jb.block0_h, bx = (jb.nw + 127) / 128;
  const uint32_t ox = (lb % bx) * 128 + threadIdx.x, y = lb / bx;
  if (ox >= jb.nw || y >= jb.nh) return;
  const uint4 t = jb.th[ox];
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
  for (uint32_t i = 0; i < t.y; ++i) {
    const float4 p = *(const float4 *)(jb.tmp + ((size_t)y * jb.w + t.x + i) * 4);
    const float wt = jb.wh[t.z + i];
    a0 = __fadd_rn(a0, __fmul_rn(p.x, wt));
    a1 = __fadd_rn(a1, __fmul_rn(p.y, wt));
    a2 = __fadd_rn(a2, __fmul_rn(p.z, wt));
    a3 = __fadd_rn(a3, __fmul_rn(p.w, wt));
  }
  uchar4 o;
  o.x = to_u8(a0);
  o.y = to_u8(a1);
  o.z = to_u8(a2);
  o.w = to_u8(a3);
  *(uchar4 *)(jb.dst + ((size_t)y * jb.nw + ox) * 4) = o;
}

// Padded copy: dst[l][y + kPad][x + kPad] = src[l][y][x], border = kOutside.
__global__ void k_pad(const uint32_t *src, uint32_t w, uint32_t h, uint32_t levels, uint32_t pw, uint32_t *dst) {
  const uint32_t ph = h + 2 * kPad;
  const size_t n = (size_t)pw * ph * levels;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t l = i / ((size_t)pw * ph);
    const uint32_t r = (uint32_t)(i - l * pw * ph);
    const int y = (int)(r / pw) - kPad, x = (int)(r % pw) - kPad;
    dst[i] = ((unsigned)x < w && (unsigned)y < h) ? src[l * w * h + (size_t)y * w + x] : kOutside;
  }
}

// Programmatic dependent launch: every hot-loop kernel first waits for the
// kernel before it in the stream to complete (its memory is then visible),
// then lets the next one launch, whose blocks start and wait in turn while
// this one's last wave runs.  Kernels launched without the attribute pass
// both instructions at once.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
  pdl_wait();
  pdl_launch();
}

// ---------------------------------------------------------------------------
// Kernels.  The plain form takes one session's descriptors as parameters;
// the multi form runs one phase of one batch step for many sessions, each
// segment of its grid belonging to one (session, step).
// ---------------------------------------------------------------------------
struct SegView {
  const SessionDev *s;
  const StepDev *d;
  uint32_t vb, vg;
};

// The segment owning this block: segments are sorted by first block, so the
// ones starting at or before blockIdx.x form a prefix; one ballot per 32.
__device__ __forceinline__ SegView find_segment(const MultiLaunch &ml) {
  const uint32_t bx = blockIdx.x + ml.block_base;
  const int lane = threadIdx.x & 31;
  uint32_t j = 0;
  for (uint32_t c = 0; c < ml.n_segs; c += kWarp) {
    const uint32_t i = c + lane;
    const bool le = i < ml.n_segs && __ldg(&ml.segs[i].block0) <= bx;
    const uint32_t bal = __ballot_sync(0xffffffffu, le);
    j = c + __popc(bal) - 1;
    if (bal != 0xffffffffu) break;
  }
  const Segment g = ml.segs[j];
  SegView v;
  v.s = ml.sessions + g.session;
  v.d = ml.step_tabs[g.session] + g.step;
  v.vb = bx - g.block0;
  v.vg = g.nblocks;
  return v;
}

// The tree entries of a chunk of appended stage items, for k-NN made ahead
// of the resolves (SessionDev::rank): what the commits of those items
// enter in flush_resolved (ms.rs:296-331), the resolved-list slot, bitmap
// and mirror bits and cell counts, plus the tree position.  The appended
// pixels and their order come from the pick chain alone, so this runs
// before their resolves; the k-NN kernels check every set bit against the
// item's own tree length.
__global__ void k_tree_append(SessionDev s, StageDev st, uint32_t a0, uint32_t a1, uint32_t pos0, uint32_t nomir_end) {
  pdl_enter();
  const uint32_t i = a0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a1) return;
  const uint32_t p = st.items[i];
  if (p >= s.W * s.H) {
    set_err(s.err, kDevErrIndex);
    return;
  }
  const uint32_t pos = pos0 + (i - a0);
  s.resolved[pos] = p;
  s.rank[p] = pos + 1u;
  const uint32_t x = p % s.W, y = p / s.W;
  atomicOr(&s.occ[(size_t)y * s.wpr + (x >> 5)], 1u << (x & 31));
  add_cell_point(s, (int)x, (int)y);
  if (s.tiling && i >= nomir_end) {
    atomicOr(&s.mir[(size_t)y * s.wpr + (x >> 5)], 1u << (x & 31));
    if ((int)x < s.x_l)
      add_cell_point(s, (int)x + (int)s.W, (int)y);
    else if ((int)x > s.x_r)
      add_cell_point(s, (int)x - (int)s.W, (int)y);
    if ((int)y < s.y_b)
      add_cell_point(s, (int)x, (int)y + (int)s.H);
    else if ((int)y > s.y_t)
      add_cell_point(s, (int)x, (int)y - (int)s.H);
  }
}

// Tree positions of the initial tree (random-init or locked pixels).
__global__ void k_rank_init(SessionDev s, uint32_t n) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const uint32_t p = s.resolved[e];
  if (p < s.W * s.H) s.rank[p] = e + 1u;
}

__global__ void k_random_candidates(SessionDev s, StageDev st) {
  pdl_enter(); random_candidates_body(s, st, blockIdx.x); }
__global__ void k_random_candidates_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  random_candidates_body(*v.s, v.d->rc, v.vb);
}

// The commit of a pending batch of redo items, spread over the launch's
// threads (PendingCommit).
__device__ __forceinline__ void pending_commit(const SessionDev &s, const PendingCommit &pc) {
  uint32_t evals = 0;  // one atomic per warp instead of one per item
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < pc.n; i += gridDim.x * blockDim.x) {
    const Result r = pc.b.res[i];
    evals += r.ncand;
    commit_item(s, pc.st, pc.b, i, r, false);
  }
  evals = __reduce_add_sync(0xffffffffu, evals);
  if ((threadIdx.x & 31) == 0 && evals) atomicAdd(s.evals, (unsigned long long)evals);
}

template <bool kWin>
__global__ void __launch_bounds__(kWalkWarps *kWarp, 4)
    k_knn_walk(SessionDev s, StageDev st, BatchDev b, const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  knn_walk_body<kWin>(s, st, b, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kWalkWarps *kWarp, 4) k_knn_walk_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  knn_walk_body<false>(*v.s, v.d->st, v.d->b, v.vb, v.vg);
}

__global__ void __launch_bounds__(kListWarps *kWarp)
    k_knn_list(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
               const __grid_constant__ BatchDev b) {
  pdl_enter();
  knn_list_body(s, st, b);
}

__global__ void __launch_bounds__(kExhThreads) k_knn_exhaustive(SessionDev s, StageDev st, BatchDev b, uint32_t cap,
                                                                 int all_items,
                                                                 const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  knn_exhaustive_body(s, st, b, all_items, cap, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kExhThreads) k_knn_exhaustive_multi(MultiLaunch ml) {
  pdl_enter();
  __shared__ ExhShared sh;
  extern __shared__ unsigned long long all_keys[];
  if (blockIdx.x < ml.pool_block0) {  // whole batches of sparse steps
    const SegView v = find_segment(ml);
    const StepDev &d = *v.d;
    const uint32_t n = d.b.i1 - d.b.i0;
    for (uint32_t e = v.vb; e < n; e += v.vg) {
      knn_exhaustive_item(*v.s, d.st, d.b, e, sh, all_keys, ml.key_cap, true);
      __syncthreads();
    }
    return;
  }
  // the pool: the fallback lists of all walk steps, concatenated, in turn;
  // their lengths are read in parallel, kExhThreads at a time
  __shared__ uint32_t fb_cnt[kExhThreads];
  const uint32_t vb = blockIdx.x - ml.pool_block0, vg = gridDim.x - ml.pool_block0;
  uint32_t base = 0;
  for (uint32_t c0 = 0; c0 < ml.n_fb; c0 += kExhThreads) {
    const uint32_t nc = min((uint32_t)kExhThreads, ml.n_fb - c0);
    __syncthreads();
    if (threadIdx.x < nc) {
      const Segment g = ml.fb[c0 + threadIdx.x];
      fb_cnt[threadIdx.x] = *ml.step_tabs[g.session][g.step].b.fb_count;
    }
    __syncthreads();
    for (uint32_t j = 0; j < nc; ++j) {
      const uint32_t cnt = fb_cnt[j];
      uint32_t v = base + (vb + vg - base % vg) % vg;
      if (v < base + cnt) {
        const Segment g = ml.fb[c0 + j];
        const StepDev &d = ml.step_tabs[g.session][g.step];
        for (; v < base + cnt; v += vg) {
          knn_exhaustive_item(ml.sessions[g.session], d.st, d.b, d.b.fb_list[v - base], sh, all_keys, ml.key_cap,
                              false);
          __syncthreads();
        }
      }
      base += cnt;
    }
  }
}

// The single-session mean: each thread first copies its item's distances
// into its own column of shared memory with asynchronous copies (all in
// flight at once), so that only the f64 chain itself stays on the
// critical path of these mostly latency-bound launches.
constexpr uint32_t kMeanThreads = 64;
__device__ __forceinline__ void mean_body_staged(const BatchDev &b, uint32_t vb) {
  extern __shared__ double md[];  // [k][kMeanThreads]
  const uint32_t nb = b.i1 - b.i0;
  const uint32_t local = vb * kMeanThreads + threadIdx.x;
  if (local >= nb) return;
  const uint32_t nk = b.ncnt[local];
  if (nk == 0) return;
  double *col = md + threadIdx.x;
  for (uint32_t j = 0; j < nk; ++j) __pipeline_memcpy_async(col + j * kMeanThreads, b.dist + (size_t)j * nb + local, 8);
  __pipeline_commit();
  __pipeline_wait_prior(0);
  double sum = 0.0;
  for (uint32_t j = 0; j < nk; ++j) {
    const double d = col[j * kMeanThreads];
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
  }
  b.mean[local] = __ddiv_rn(sum, (double)(nk * 4u));
}

__global__ void __launch_bounds__(kMeanThreads) k_mean_staged(SessionDev s, StageDev st, BatchDev b) {
  pdl_enter();
  mean_body_staged(b, blockIdx.x);
}

// The means of lists made ahead (sessions without exact sums): a block's
// items' distances from the coordinate tables into shared memory, one column
// per item (an odd pitch of doubles spreads the columns' writes over the
// banks), then each item's chain of 4k f64 adds on one lane.  The chain keeps
// the FP64 pipe busy (an f64 warp instruction takes it 18 cycles whatever its
// active lanes), so every lane of a warp carries an item; the launches run on
// the side stream, off the step chain.
// Four threads per item form the distances, four at a time each (chained
// loads and f64 operations: with one thread and one distance at a time a
// launch over far neighbours took 81 us).
constexpr uint32_t kMeanPitch = kMeanThreads + 1;
constexpr uint32_t kMeanAheadThreads = 4 * kMeanThreads;
__global__ void __launch_bounds__(kMeanAheadThreads)
    k_mean_ahead(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                 const __grid_constant__ BatchDev b) {
  pdl_enter();
  extern __shared__ double md[];  // [k][kMeanPitch]
  __shared__ int xs[kMeanThreads], ys[kMeanThreads];
  __shared__ uint32_t cnt[kMeanThreads];
  const uint32_t first = blockIdx.x * kMeanThreads, n = min(kMeanThreads, b.i1 - b.i0 - first);
  const uint32_t tid = threadIdx.x;
  if (tid < kMeanThreads) {
    cnt[tid] = 0;
    xs[tid] = ys[tid] = 0;  // (the entries past the last item look up pixel 0's tables)
    if (tid < n) {
      pixel_xy(s, st.items[b.i0 + first + tid], xs[tid], ys[tid]);
      cnt[tid] = b.ncnt[first + tid];
    }
  }
  __syncthreads();
  const int32_t *nbo = b.nbuf + (size_t)first * s.k;
  constexpr int kPer = 4;
  for (uint32_t e0 = tid; e0 < n * s.k; e0 += kPer * kMeanAheadThreads) {
    uint32_t it[kPer], jt[kPer];
    int32_t off[kPer];
    double d[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const uint32_t e = e0 + (uint32_t)u * kMeanAheadThreads;
      it[u] = min(e / s.k, kMeanThreads - 1u);
      jt[u] = e - it[u] * s.k;
      off[u] = e < n * s.k && jt[u] < cnt[it[u]] ? __ldg(&nbo[e]) : 0;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) d[u] = neighbour_dist(s, xs[it[u]], ys[it[u]], off_dx(off[u]), off_dy(off[u]));
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (e0 + (uint32_t)u * kMeanAheadThreads < n * s.k && jt[u] < cnt[it[u]]) md[jt[u] * kMeanPitch + it[u]] = d[u];
  }
  __syncthreads();
  if (tid >= n || cnt[tid] == 0) return;
  double sum = 0.0;
#pragma unroll 4
  for (uint32_t q = 0; q < cnt[tid]; ++q) {
    const double d = md[q * kMeanPitch + tid];
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
    sum = __dadd_rn(sum, d);
  }
  b.mean[first + tid] = __ddiv_rn(sum, (double)(cnt[tid] * 4u));
}

// The coordinate tables of a session without exact sums (SessionDev::xdiv,
// ydiv, dxt, dy2t), with the IEEE operations of get_distances_to_k_neighs
// (ms.rs:410-415): n_x, n_y entries of xdiv and ydiv, then 2 R + 1 offsets
// per column and per row.
__global__ void k_dist_tables(const __grid_constant__ SessionDev s, double *xdiv, double *ydiv, double *dxt,
                              double *dy2t, uint32_t n_x, uint32_t n_y) {
  const uint32_t w = 2u * (uint32_t)s.dtab_r + 1u, n_dx = s.W * w, n_dy = s.H * w;
  const double dw = (double)s.W, dh = (double)s.H;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_x + n_y + n_dx + n_dy; i += gridDim.x * blockDim.x) {
    uint32_t e = i;
    if (e < n_x) {
      xdiv[e] = __ddiv_rn((double)((int)e - s.xdiv_off), dw);
      continue;
    }
    e -= n_x;
    if (e < n_y) {
      ydiv[e] = __ddiv_rn((double)((int)e - s.ydiv_off), dh);
      continue;
    }
    e -= n_y;
    const bool col = e < n_dx;
    if (!col) e -= n_dx;
    const int q = (int)(e / w), o = (int)(e - (uint32_t)q * w) - s.dtab_r;
    const double side = col ? dw : dh;
    const double d = __dsub_rn(__ddiv_rn((double)(q + o), side), __ddiv_rn((double)q, side));
    if (col)
      dxt[e] = d;
    else
      dy2t[e] = __dmul_rn(d, d);
  }
}

__global__ void __launch_bounds__(128) k_mean_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  mean_body(*v.s, v.d->b, v.vb);
}

// pc: the previous batch step's deferred commit (BatchDev::prev_tag), made
// here by every thread of the grid before its own item; this launch's
// readers of those pixels take their values from pc.b.res instead.
__global__ void __launch_bounds__(kResolveWarps *kWarp, 8)
    k_resolve(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
              const __grid_constant__ BatchDev b, const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  resolve_body<false, kCostPlain>(s, st, b, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kResolveWarps *kWarp, 8)
    k_resolve_signed(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                     const __grid_constant__ BatchDev b, const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  resolve_body<false, kCostSigned>(s, st, b, blockIdx.x, gridDim.x);
}
// Sessions without guides (the guide terms compiled out).
__global__ void __launch_bounds__(kResolveWarps *kWarp, 8)
    k_resolve_lean(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                   const __grid_constant__ BatchDev b, const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  resolve_body<true, kCostPlain>(s, st, b, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kResolveWarps *kWarp, 8) k_resolve_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  if (v.s->guided)
    resolve_body<false, kCostAny>(*v.s, v.d->st, v.d->b, v.vb, v.vg);
  else
    resolve_body<true, kCostPlain>(*v.s, v.d->st, v.d->b, v.vb, v.vg);
}
// Segments of sessions without guides.
__global__ void __launch_bounds__(kResolveWarps *kWarp, 8) k_resolve_multi_lean(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  resolve_body<true, kCostPlain>(*v.s, v.d->st, v.d->b, v.vb, v.vg);
}

template <int T, bool kFull>
__global__ void __launch_bounds__(T)
    k_resolve_team(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                   const __grid_constant__ BatchDev b, const __grid_constant__ PendingCommit pc) {
  pdl_enter();
  if (pc.n) pending_commit(s, pc);
  resolve_team_body<T, kFull, kCostPlain>(s, st, b, blockIdx.x, gridDim.x);
}
template <int T, bool kFull>
__global__ void __launch_bounds__(T) k_resolve_team_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  resolve_team_body<T, kFull, kCostAny>(*v.s, v.d->st, v.d->b, v.vb, v.vg);
}

// ---------------------------------------------------------------------------
// resolve, small steps: a CTA of T threads per item, for steps too small to
// fill the GPU with warps, where the time of a step is one item's chain of
// dependent loads, barriers and sums (the plain path runs some 60 to 130 such
// steps one after another).
//
// With its lists and random candidates made ahead (BatchDev::early) nearly all
// of an item is known before the step it builds on is done: its weights, its
// target-guide texels, its random candidates and their texels.  All of that
// runs before griddepcontrol.wait, and the launch lets the next step's launch
// start before it waits itself, so it overlaps the steps before.  What
// remains after the wait is one warp's loads of the neighbours' state, the
// repeat match, one gather of the few different coherence candidates (the
// random ones' terms are formed while it is in flight), one in-order sum per
// lane and the argmin.  A step of one item, k = m = 50: 18.8 -> 4.7 us, of
// which 1.2 from the end of the step before to the wait's return, 1 state and
// repeats, 1.2 gather and terms, 0.8 sums and argmin, 0.4 commit.
//
// F: terms of a random candidate formed at once: all of them while the steps
// are small; for larger ones (kSmallFirst) only the candidates that are still
// below the best coherence cost after F terms go on.
// ---------------------------------------------------------------------------
constexpr uint32_t kSmallK = 64;      // neighbours one warp takes in two rounds
constexpr uint32_t kSmallFirst = 8;
constexpr size_t kSmallMaxSmem = 64 * 1024;
// Floats per term row: a multiple of 4 whose quarter is odd, so that the lanes'
// in-order sums read 16 bytes each from different banks.
__host__ __device__ __forceinline__ uint32_t term_pitch(uint32_t k) { return 4u * (((k + 3u) / 4u) | 1u); }
// LUTs, records, offsets, patch ids, then per candidate {record, centre,
// centre colour} and its term row; coherence candidates in slots [0, k),
// random ones in [k, k + m).
__host__ __device__ __forceinline__ size_t small_smem_bytes(uint32_t k, uint32_t m, uint32_t n_maps) {
  return 2048 + kSmallK * 24 + (size_t)n_maps * 16 + (((size_t)(k + m) * 20 + 15) & ~(size_t)15) +
         (size_t)(k + m) * term_pitch(k) * 4;
}

template <int T, bool kG, int kMode>
__device__ __forceinline__ void resolve_small_body(const SessionDev &s, const StageDev &st, const BatchDev &b,
                                                   const PendingCommit &pc, uint32_t F) {
  constexpr int NW = T / kWarp;
  constexpr int NR = T >= 512 ? 6 : (T >= 256 ? 10 : 4);  // random texels held per thread
  constexpr int NC = 2;                                   // coherence texels in flight per thread
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float tab_ff[128];
  __shared__ float red_s[NW];
  __shared__ uint32_t red_i[NW];
  __shared__ uint32_t sh_ncoh, sh_all, sh_bad, sh_live;
  __shared__ uint2 first[kWarp];
  __shared__ uint8_t slots[128];
  float *lc = (float *)smem, *lg = lc + 256;
  uint4 *nbr = (uint4 *)(smem + 2048);
  int32_t *offs = (int32_t *)(nbr + kSmallK);
  uint32_t *pid = (uint32_t *)(offs + kSmallK);
  uint4 *mt = (uint4 *)(pid + kSmallK);  // {w | mask flag | h << 16, -, texel index of (0, 0) on the padded planes}
  uint64_t *cen = (uint64_t *)(mt + s.n_maps);
  uint2 *cand = (uint2 *)(cen + s.k + s.m);
  uint32_t *ccol = (uint32_t *)(cand + s.k + s.m);
  float *rows = (float *)(smem + 2048 + kSmallK * 24 + (size_t)s.n_maps * 16 +
                          align16((size_t)(s.k + s.m) * 20));
  constexpr uint32_t kMasked = 0x8000u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u, pitch = term_pitch(s.k);
  const uint32_t nb = b.i1 - b.i0;
  for (int i = tid; i < (kG ? 512 : 256); i += T) lc[i] = st.lut[i];
  for (int i = tid; i < 128; i += T) tab_ff[i] = g_exp2_ff[i];
  for (uint32_t i = tid; i < s.n_maps; i += T) {
    const MapDesc md = s.maps[i];
    const uint64_t c0 = padded_centre(md, st.level, 0u);
    mt[i] = make_uint4(md.w | (md.h << 16) | (md.mask_off >= 0 ? kMasked : 0u), 0u, (uint32_t)c0, (uint32_t)(c0 >> 32));
  }
  auto centre_of = [&](uint32_t map, uint32_t cxy) -> uint64_t {
    const uint4 e = mt[map];
    return (((uint64_t)e.w << 32) | e.z) + (uint64_t)((cxy >> 16) * s.ppitch + (cxy & 0xffffu));
  };
  // texel (and guide texel) of candidate slot c at neighbour j
  auto fetch = [&](uint32_t c, uint32_t j, bool far, uint32_t &t, uint32_t &g) {
    if (!far) {
      const int lin = (int32_t)nbr[j].x;
      const int64_t at = (int64_t)cen[c] + ((cand[c].y & kAuxNeg) ? -lin : lin);
      t = __ldg(s.plevels + at);
      if (kG) g = __ldg(s.pguides + at);
    } else {
      const uint2 cd = cand[c];
      const uint32_t map = cd.y & 0x7fffu;
      const int sg = (cd.y & kAuxNeg) ? -1 : 1;
      const int qx = (int)(cd.x & 0xffffu) + sg * off_dx(offs[j]), qy = (int)(cd.x >> 16) + sg * off_dy(offs[j]);
      const MapDesc md = s.maps[map];
      t = texel(s.levels + md.off + (size_t)st.level * md.w * md.h, md, qx, qy);
      if (kG) {
        const GuideDesc gd = s.gdesc[map];
        g = kOutside;
        if ((unsigned)qx < gd.w && (unsigned)qy < gd.h)
          g = __ldg(&s.guides[gd.off + (size_t)st.level * gd.w * gd.h + (size_t)qy * gd.w + qx]);
      }
    }
  };
  auto put_term = [&](uint32_t c, uint32_t j, uint32_t t, uint32_t g) {
    const uint4 nr = nbr[j];
    float nps = lut4r(lc, __vabsdiffu4(nr.y, t), 0.0f, st.opaque);
    if (kG) nps = lut4r(lg, __vabsdiffu4(nr.z, g), nps, st.opaque);
    rows[c * pitch + j] = __fmul_rn(nps, __uint_as_float(nr.w));
  };
  // in-order sum of row c over [j, n), from acc (j a multiple of 4)
  auto row_sum = [&](uint32_t c, uint32_t j, uint32_t n, float acc) -> float {
    const float *row = rows + c * pitch;
    for (; j + 8 <= n; j += 8) {  // both loads in flight ahead of their adds
      const float4 v = *(const float4 *)(row + j), x = *(const float4 *)(row + j + 4);
      acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v.x), v.y), v.z), v.w);
      acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, x.x), x.y), x.z), x.w);
    }
    for (; j + 4 <= n; j += 4) {
      const float4 v = *(const float4 *)(row + j);
      acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v.x), v.y), v.z), v.w);
    }
    for (; j < n; ++j) acc = __fadd_rn(acc, row[j]);
    return acc;
  };
  // lowest (score, index) over the block; every thread gets it
  auto block_best = [&](float v, uint32_t i, float &bs, uint32_t &bi) {
    const float wv = warp_min(v);
    const uint32_t wi = __reduce_min_sync(0xffffffffu, v == wv ? i : 0xffffffffu);
    if (lane == 0) {
      red_s[warp] = wv;
      red_i[warp] = wi;
    }
    __syncthreads();
    const float qv = lane < NW ? red_s[lane] : __builtin_huge_valf();
    const uint32_t qi = lane < NW ? red_i[lane] : 0xffffffffu;
    bs = warp_min(qv);
    bi = __reduce_min_sync(0xffffffffu, qv == bs ? qi : 0xffffffffu);
  };

  bool waited = false;
  uint32_t evals = 0;  // thread 0: candidates of the items committed here
  auto wait_once = [&]() {
    if (waited) return;
    waited = true;
    pdl_wait();
    // the previous step's deferred commit, by the last threads first (the
    // first warp has the chain to run)
    uint32_t ev = 0;
    for (uint32_t i = blockIdx.x * T + (T - 1 - tid); i < pc.n; i += gridDim.x * T) {
      const Result r = pc.b.res[i];
      ev += r.ncand;
      commit_item(s, pc.st, pc.b, i, r, false);
    }
    if (pc.n) {
      ev = __reduce_add_sync(0xffffffffu, ev);
      if (lane == 0 && ev) atomicAdd(s.evals, (unsigned long long)ev);
    }
  };
  if (!b.early) wait_once();  // the lists come from the launches before this one

  for (uint32_t local = blockIdx.x; local < nb; local += gridDim.x) {
    __syncthreads();  // the tables (first item), the records of the item before
    const uint32_t item = b.i0 + local;
    const uint32_t pixel = st.items[item];
    const uint32_t nk = b.ncnt[local];
    if (nk == 0) {
      wait_once();
      if (tid == 0) write_random_result(s, st, b, local, pixel);
      continue;
    }
    int px, py;
    pixel_xy(s, pixel, px, py);
    const double avg = b.mean[local];
    const FfMean fm = ts_ff_mean(avg);
    bool nan_w = false;
    int maxoff = 0;
    for (uint32_t j = tid; j < nk; j += T) {
      const int32_t off = b.nbuf[(size_t)local * s.k + j];
      const int dx = off_dx(off), dy = off_dy(off);
      maxoff = max(maxoff, max(abs(dx), abs(dy)));
      uint32_t gpat = 0;
      if (kG) {
        const uint32_t p = (uint32_t)wrap1(py + dy, (int)s.H) * s.W + (uint32_t)wrap1(px + dx, (int)s.W);
        gpat = __ldg(&s.tguide[(size_t)st.level * s.W * s.H + p]);
      }
      const float wv = item_weight(s, b, local, nb, px, py, j, off, avg, fm, tab_ff);
      nan_w |= (wv != wv);
      nbr[j] = make_uint4((uint32_t)(dy * (int)s.ppitch + dx), 0u, gpat, __float_as_uint(wv));
      offs[j] = off;
    }
    const uint2 *rc = st.rcand + (size_t)item * s.m;
    for (uint32_t t = tid; t < s.m; t += T) {
      const uint2 cd = random_candidate(s, rc, t);
      const uint64_t c = centre_of(cd.y & 0x7fffu, cd.x);
      cand[s.k + t] = cd;
      cen[s.k + t] = c;
      ccol[s.k + t] = __ldg(s.plevels + c);
    }
    const bool far = __syncthreads_or(maxoff > kPad) || s.guide_dims_differ;
    const bool in_order = costs_in_order<kMode>(st);
    const bool slow = __syncthreads_or(nan_w) || costs_exact<kMode>(st);
    // the random candidates' first f texels
    const uint32_t f = in_order ? nk : min(F, nk), n_rnd = slow ? 0u : s.m * f;
    const float rf = __fdividef(1.0f, (float)f);
    auto split = [&](uint32_t i, float r, uint32_t n, uint32_t &c, uint32_t &j) {
      c = (uint32_t)(((float)i + 0.5f) * r);  // i / n, exact below 2^20
      j = i - c * n;
    };
    uint32_t tx[NR], gx[NR];
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const uint32_t i = tid + (uint32_t)u * T;
      tx[u] = gx[u] = 0;
      if (i < n_rnd) {
        uint32_t c, j;
        split(i, rf, f, c, j);
        fetch(s.k + c, j, far, tx[u], gx[u]);
      }
    }
    wait_once();
    // the neighbours' state: own pattern (ms.rs:1151-1181), coherence
    // candidates (ms.rs:497-547) without repeats (the same cost as the first
    // of them; kept where the exact sequential form compares them)
    if (warp == 0) {
      uint32_t pat[2], ncoh = 0, all = 0;
      uint4 sv[2];
      bool bad = false;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t j = lane + (uint32_t)r * kWarp;
        pat[r] = 0;
        sv[r] = make_uint4(0u, 0u, 0u, 0u);
        if (j < nk) {
          const int32_t off = offs[j];
          const uint32_t p = (uint32_t)wrap1(py + off_dy(off), (int)s.H) * s.W + (uint32_t)wrap1(px + off_dx(off), (int)s.W);
          start_pixel(s, b, p, true, pat[r], sv[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t j = lane + (uint32_t)r * kWarp;
        if ((uint32_t)r * kWarp >= nk) break;
        bool valid = false;
        uint32_t cxy = 0;
        const uint32_t map = sv[r].z;
        if (j < nk) {
          nbr[j].y = pat[r];
          pid[j] = sv[r].y;
          if (map >= s.n_maps) {
            bad = true;
          } else {
            const int ccx = (int)(sv[r].x & 0xffffu) - off_dx(offs[j]), ccy = (int)(sv[r].x >> 16) - off_dy(offs[j]);
            const uint32_t wh = mt[map].x, mw = wh & 0x7fffu;
            valid = (uint32_t)ccx < mw && (uint32_t)ccy < (wh >> 16);
            if (valid && (wh & kMasked)) valid = __ldg(&s.masks[s.maps[map].mask_off + (size_t)ccy * mw + ccx]) != 0;
            cxy = (uint32_t)ccx | ((uint32_t)ccy << 16);
          }
        }
        const uint32_t vm = __ballot_sync(0xffffffffu, valid);
        bool keep = valid;
        if (!slow) {
          uint32_t same;
          if (s.n_maps <= 16)
            same = __match_any_sync(0xffffffffu, (cxy & 0x3fffu) | ((cxy >> 16) << 14) | (map << 28));
          else
            same = __match_any_sync(0xffffffffu, ((unsigned long long)map << 32) | cxy);
          if (same & vm & lt) keep = false;
          // the second round against the first: a table from hashes to lanes
          // of the first round (the last writer of a slot; what it holds is
          // compared, so a stale or shared slot only lets a repeat stay)
          const uint32_t h = ((cxy + map * 0x632be5abu) * 0x9e3779b1u) >> 25;
          if (r == 0) {
            first[lane] = make_uint2(cxy, valid ? map : 0xffffffffu);
            if (valid) slots[h] = (uint8_t)lane;
          } else {
            const uint2 c1 = first[slots[h] & 31u];
            if (c1.x == cxy && c1.y == map) keep = false;
          }
        }
        all += __popc(vm);
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const uint32_t slot = ncoh + __popc(bal & lt);
          cand[slot] = make_uint2(cxy, map | (j << 16));
          cen[slot] = centre_of(map, cxy);
        }
        ncoh += __popc(bal);
        __syncwarp();
      }
      const bool any_bad = __any_sync(0xffffffffu, bad);
      if (lane == 0) {
        sh_ncoh = ncoh;
        sh_all = all;
        sh_bad = any_bad ? 1u : 0u;
        sh_live = 0;
      }
    }
    __syncthreads();
    const uint32_t ncoh = sh_ncoh;
    if (sh_bad) {
      // the reference panics on this index; record the error and leave the
      // pixel untouched (commit skips results with an invalid map)
      if (tid == 0) write_bad_result(s, st, b, local, pixel);
      continue;
    }
    float best_s = FLT_MAX;
    uint32_t best_i = 0;
    if (slow) {
      WarpSmem w;
      w.nbr = nbr;
      w.cand = cand;
      w.term = nullptr;
      w.off = offs;
      if (tid == 0) {
        sequential_best<kG>(s, st, w, lc, lg, nk, ncoh + s.m, best_s, best_i, ncoh, s.k - ncoh);
        const uint32_t slot = best_i < ncoh ? best_i : s.k + best_i - ncoh;
        ccol[slot] = __ldg(s.plevels + cen[slot]);
      }
    } else {
      // the coherence candidates' texels in flight, the random ones' terms
      // meanwhile
      const uint32_t n_coh_terms = ncoh * nk;
      const float rk = __fdividef(1.0f, (float)nk);
      uint32_t t2[NC], g2[NC], c2[NC], j2[NC], col = 0;
#pragma unroll
      for (int u = 0; u < NC; ++u) {
        const uint32_t i = tid + (uint32_t)u * T;
        t2[u] = g2[u] = c2[u] = j2[u] = 0;
        if (i < n_coh_terms) {
          split(i, rk, nk, c2[u], j2[u]);
          fetch(c2[u], j2[u], far, t2[u], g2[u]);
        }
      }
      if ((uint32_t)tid < ncoh) col = __ldg(s.plevels + cen[tid]);
#pragma unroll
      for (int u = 0; u < NR; ++u) {
        const uint32_t i = tid + (uint32_t)u * T;
        if (i < n_rnd) {
          uint32_t c, j;
          split(i, rf, f, c, j);
          put_term(s.k + c, j, tx[u], gx[u]);
        }
      }
      for (uint32_t i = tid + (uint32_t)NR * T; i < n_rnd; i += T) {
        uint32_t c, j, t, g = 0;
        split(i, rf, f, c, j);
        fetch(s.k + c, j, far, t, g);
        put_term(s.k + c, j, t, g);
      }
#pragma unroll
      for (int u = 0; u < NC; ++u)
        if (tid + (uint32_t)u * T < n_coh_terms) put_term(c2[u], j2[u], t2[u], g2[u]);
      if ((uint32_t)tid < ncoh) ccol[tid] = col;
      for (uint32_t i = tid + (uint32_t)NC * T; i < n_coh_terms; i += T) {
        uint32_t c, j, t, g = 0;
        split(i, rk, nk, c, j);
        fetch(c, j, far, t, g);
        put_term(c, j, t, g);
      }
      for (uint32_t c = tid + T; c < ncoh; c += T) ccol[c] = __ldg(s.plevels + cen[c]);
      __syncthreads();
      // sums, one candidate per thread; the first strict minimum
      float my_s = FLT_MAX;
      uint32_t my_i = 0xffffffffu;
      auto offer = [&](float v, uint32_t i) {
        if (v < my_s || (v == my_s && i < my_i)) {
          my_s = v;
          my_i = i;
        }
      };
      if (in_order) {
        // each candidate's {cost, largest partial sum} into its row, then in order
        const uint32_t nc = ncoh + s.m;
        for (uint32_t q = tid; q < nc; q += T) {
          float *row = rows + (q < ncoh ? q : s.k + q - ncoh) * pitch;
          float sum = 0.0f, peak = -FLT_MAX;
          for (uint32_t j = 0; j < nk; ++j) {
            sum = __fadd_rn(sum, row[j]);
            peak = fmaxf(peak, sum);
          }
          *(float2 *)row = make_float2(sum, peak);
        }
        __syncthreads();
        if (warp == 0) {
          for (uint32_t base = 0; base < nc; base += kWarp) {
            const uint32_t q = base + lane;
            float2 v = make_float2(0.0f, __builtin_huge_valf());
            if (q < nc) v = *(const float2 *)(rows + (q < ncoh ? q : s.k + q - ncoh) * pitch);
            take_signed(v.x, v.y, base, best_s, best_i);
          }
        }
      } else if (f == nk) {
        for (uint32_t q = tid; q < ncoh + s.m; q += T) offer(row_sum(q < ncoh ? q : s.k + q - ncoh, 0, nk, 0.0f), q);
        block_best(my_s, my_i, best_s, best_i);
      } else {
        for (uint32_t q = tid; q < ncoh; q += T) offer(row_sum(q, 0, nk, 0.0f), q);
        block_best(my_s, my_i, best_s, best_i);
        // random candidates below that cost after f terms: their other terms
        uint32_t *live = (uint32_t *)(rows + (size_t)ncoh * pitch);  // the coherence rows from ncoh on are unused
        const uint32_t live_cap = (s.k - ncoh) * pitch;
        my_s = best_s;
        my_i = best_i;
        for (uint32_t t = tid; t < s.m; t += T) {
          const float part = row_sum(s.k + t, 0, f, 0.0f);
          if (part < best_s) {
            const uint32_t at = atomicAdd(&sh_live, 1u);
            if (at < live_cap) {
              live[at] = t;
              rows[(s.k + t) * pitch] = part;  // the sum so far, in the place of the first terms
            } else {
              // no room for the list: this thread scores the rest itself
              float acc = part;
              for (uint32_t j = f; j < nk; ++j) {
                uint32_t tt, gg = 0;
                fetch(s.k + t, j, far, tt, gg);
                put_term(s.k + t, j, tt, gg);
                acc = __fadd_rn(acc, rows[(s.k + t) * pitch + j]);
              }
              offer(acc, ncoh + t);
            }
          }
        }
        __syncthreads();
        const uint32_t n_live = min(sh_live, live_cap), rest = nk - f;
        const float rr = __fdividef(1.0f, (float)rest);
        for (uint32_t i = tid; i < n_live * rest; i += T) {
          uint32_t c, j, t, g = 0;
          split(i, rr, rest, c, j);
          const uint32_t slot = s.k + live[c];
          fetch(slot, f + j, far, t, g);
          put_term(slot, f + j, t, g);
        }
        __syncthreads();
        for (uint32_t c = tid; c < n_live; c += T) {
          const uint32_t t = live[c];
          offer(row_sum(s.k + t, f, nk, rows[(s.k + t) * pitch]), ncoh + t);
        }
        if (sh_live) block_best(my_s, my_i, best_s, best_i);
      }
      if (best_i == 0xffffffffu) {  // no score below f32::MAX: the reference keeps candidate 0
        best_s = FLT_MAX;
        best_i = 0;
      }
    }
    if (tid == 0) {
      const uint32_t slot = best_i < ncoh ? best_i : s.k + best_i - ncoh;
      const uint2 cd = cand[slot];
      const uint32_t map = cd.y & 0x7fffu;
      Result r;
      r.pixel = pixel;
      r.srcxy = cd.x;
      r.idp = (cd.y & kAuxNeg) ? (cd.x >> 16) * (mt[map].x & 0x7fffu) + (cd.x & 0xffffu) : pid[cd.y >> 16];
      r.idm = map;
      r.color = ccol[slot];
      r.flags = (item >= st.redo ? kResAppend : 0u) | kResMirrors;
      r.score = best_s;
      r.ncand = sh_all + s.m;
      emit_result(s, st, b, local, r, false);
      evals += r.ncand;
    }
  }
  wait_once();
  // (a batch left to a later commit is counted there)
  if (b.fused_commit && tid == 0 && evals) atomicAdd(s.evals, (unsigned long long)evals);
}

template <int T, bool kG, int kMode>
__global__ void __launch_bounds__(T, 1024 / T)
    k_resolve_small(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                    const __grid_constant__ BatchDev b, const __grid_constant__ PendingCommit pc, uint32_t F) {
  pdl_launch();
  resolve_small_body<T, kG, kMode>(s, st, b, pc, F);
}

// One step of a batch of new items whose neighbours the exhaustive k-NN
// finds, one item per CTA at a time (256 threads): the item's k-NN, then its
// full-evaluation resolve (every candidate scored completely, as the team
// form does), in one launch.  The mean's chain of 4k dependent f64 adds
// (ms.rs:417-423) runs on warp 0's first lane while warps 1-7 set up the
// neighbour records and candidates and gather every (candidate, neighbour)
// LUT sum, none of which needs the mean; the weights and each candidate's
// in-order sum of nps_j * w_j follow on all warps.  The other CTAs' commits
// change only their own pixels, the resolved list beyond n_res and the
// occupancy, mirror and cell records of those pixels; this k-NN reads the
// first n_res points and their mirror bits only (the cell grid is not
// searched here; a key buffer overflow rescans the points).
// Barrier of the set-up warps (all but warp 0): TS threads.
template <int TS>
__device__ __forceinline__ void setup_bar() {
  asm volatile("bar.sync 1, %0;" ::"n"(TS) : "memory");
}

// T = 256, or 512 for steps of at most one item per SM, where the extra
// warps shorten each item's latency-bound k-NN and gathers.
template <int T>
__global__ void __launch_bounds__(T) k_step_team_full(const __grid_constant__ SessionDev s, const __grid_constant__ StageDev st,
                     const __grid_constant__ BatchDev b, uint32_t cap) {
  constexpr int NW = T / kWarp, TS = T - kWarp;
  __shared__ ExhShared sh;
  __shared__ float tab_ff[128];
  __shared__ uint32_t wcnt[NW];
  __shared__ float red_s[NW];
  __shared__ uint32_t red_i[NW];
  __shared__ int sh_flags, sh_maxoff;
  __shared__ uint32_t sh_ncoh;
  __shared__ double sh_mean;
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t nb = b.i1 - b.i0;
  float *lc = (float *)smem;
  float *lg = lc + 256;
  const WarpSmem w = carve(smem + 2048, s.k, s.m);
  float *term = (float *)(smem + 2048 + warp_smem_bytes(s.k, s.m));
  for (uint32_t local = blockIdx.x; local < nb; local += gridDim.x) {
    const uint32_t nk = knn_exhaustive_item(s, st, b, local, sh, (unsigned long long *)smem, cap, true, false, false);
    __syncthreads();  // sh.dist, sh.nbo; the key buffer is free again
    const uint32_t item = b.i0 + local;
    const uint32_t pixel = st.items[item];
    int px, py;
    pixel_xy(s, pixel, px, py);
    const bool is_new = item >= st.redo;
    if (nk == 0) {
      if (tid == 0) write_random_result(s, st, b, local, pixel);
      __syncthreads();
      continue;
    }
    if (warp == 0) {
      if (s.exact_sum) {
        unsigned long long part = 0;
        for (uint32_t j = lane; j < nk; j += kWarp) part += exact_units(s, off_dx(sh.nbo[j]), off_dy(sh.nbo[j]));
        part = warp_sum_units(part);
        if (lane == 0) {
          const double mean = exact_mean(s, part, nk);
          sh_mean = mean;
          b.mean[local] = mean;
        }
      } else if (lane == 0) {
        const double mean = mean_chain(sh.dist, nk);
        sh_mean = mean;
        b.mean[local] = mean;
      }
    } else {
      const int t = tid - kWarp;
      // the LUTs, the exp tables and the first random candidates go into
      // registers first, so that their loads are in flight together with
      // the neighbour records' loads; they reach shared memory after the
      // records (the records loop's barriers order the flags' reset before
      // their first update)
      constexpr int kLutPer = (512 + TS - 1) / TS;
      float lreg[kLutPer];
#pragma unroll
      for (int u = 0; u < kLutPer; ++u) {
        const int i = t + u * TS;
        lreg[u] = i < 512 ? st.lut[i] : 0.0f;
      }
      const float freg = t < 128 ? g_exp2_ff[t] : 0.0f;
      const uint2 *rc = st.rcand + (size_t)item * s.m;
      const uint2 rv0 = (uint32_t)t < s.m ? rc[t] : make_uint2(0u, 0u);
      if (t == 0) {
        sh_flags = 0;
        sh_maxoff = 0;
      }
      // neighbour records and coherence candidates, compacted in order
      bool bad_map = false;
      int maxoff = 0;
      uint32_t ncoh = 0;
      for (uint32_t j0 = 0; j0 < nk; j0 += TS) {
        const uint32_t j = j0 + t;
        bool valid = false;
        uint32_t cxy = 0, aux = 0;
        if (j < nk) valid = neighbour_records(s, st, b, px, py, j, sh.nbo[j], 0.0f, w, cxy, aux, maxoff, bad_map);
        const uint32_t bal = __ballot_sync(0xffffffffu, valid);
        if (lane == 0) wcnt[warp] = __popc(bal);
        setup_bar<TS>();
        uint32_t base = ncoh, total = 0;
#pragma unroll
        for (int i = 1; i < NW; ++i) {
          if (i < warp) base += wcnt[i];
          total += wcnt[i];
        }
        if (valid) {
          const uint32_t slot = base + __popc(bal & lt);
          w.cand[slot] = make_uint2(cxy, aux);
        }
        ncoh += total;
        setup_bar<TS>();
      }
#pragma unroll
      for (int u = 0; u < kLutPer; ++u) {
        const int i = t + u * TS;
        if (i < 512) lc[i] = lreg[u];
      }
      if (t < 128) tab_ff[t] = freg;
      if (bad_map) atomicOr(&sh_flags, 2);
      if (maxoff) atomicMax(&sh_maxoff, maxoff);
      for (uint32_t q = t; q < s.m; q += TS) {
        const uint2 v = use_rcand(s, q == (uint32_t)t ? rv0 : rc[q]);
        w.cand[ncoh + q] = make_uint2(v.x, v.y | kAuxNeg | (q << 16));
      }
      if (t == 0) sh_ncoh = ncoh;
      setup_bar<TS>();
      if (!(sh_flags & 2) && !st.slow_lut) {
        // every candidate's LUT sums nps(c, j), before the weights exist
        const uint32_t nc = ncoh + s.m, total = nc * nk;
        if (sh_maxoff <= kPad && !s.guide_dims_differ) {
          unsigned long long *cb = (unsigned long long *)(term + (((size_t)nk * nc + 1) & ~(size_t)1));
          for (uint32_t c = t; c < nc; c += TS) {
            const uint32_t cxy = w.cand[c].x, aux = w.cand[c].y;
            cb[c] = padded_centre(s.maps[aux & 0x7fffu], st.level, cxy) | ((aux & kAuxNeg) ? (1ull << 63) : 0ull);
          }
          setup_bar<TS>();
          constexpr int kRound = 16;  // gathers in flight per thread
          for (uint32_t i0 = t; i0 < total; i0 += kRound * TS) {
            uint32_t tx[kRound], gx[kRound], ii[kRound], jj[kRound];
#pragma unroll
            for (int u = 0; u < kRound; ++u) {
              const uint32_t i = i0 + (uint32_t)u * TS;
              ii[u] = i;
              if (i < total) {
                const uint32_t c = i / nk;
                jj[u] = i - c * nk;
                const unsigned long long v = cb[c];
                const int lj = (int32_t)w.nbr[jj[u]].x, lin = (v >> 63) ? -lj : lj;
                const size_t off = (size_t)(v & 0x7fffffffffffffffull) + lin;
                tx[u] = __ldg(s.plevels + off);
                if (s.guided) gx[u] = __ldg(s.pguides + off);
              }
            }
#pragma unroll
            for (int u = 0; u < kRound; ++u) {
              if (ii[u] < total) {
                const uint4 nr = w.nbr[jj[u]];
                float nps = lut4r(lc, __vabsdiffu4(nr.y, tx[u]), 0.0f, st.opaque);
                if (s.guided) nps = lut4r(lg, __vabsdiffu4(nr.z, gx[u]), nps, st.opaque);
                term[ii[u]] = nps;
              }
            }
          }
        } else {
          // bounds-checked gathers (far neighbours or guides of other sizes)
          uint32_t c = (uint32_t)t / nk, j = (uint32_t)t - c * nk;
          const uint32_t dc = (uint32_t)TS / nk, dj = (uint32_t)TS - dc * nk;
          for (uint32_t i = t; i < total; i += TS) {
            const uint32_t cxy = w.cand[c].x, aux = w.cand[c].y;
            const uint32_t map = aux & 0x7fffu;
            const int sg = (aux & kAuxNeg) ? -1 : 1;
            const MapDesc md = s.maps[map];
            const uint4 nr = w.nbr[j];
            const int qx = (int)(cxy & 0xffffu) + sg * off_dx(w.off[j]);
            const int qy = (int)(cxy >> 16) + sg * off_dy(w.off[j]);
            uint32_t tt = kOutside;
            if ((unsigned)qx < md.w && (unsigned)qy < md.h)
              tt = __ldg(&s.levels[md.off + (size_t)st.level * md.w * md.h + (size_t)qy * md.w + qx]);
            float nps = lut4(lc, __vabsdiffu4(nr.y, tt), 0.0f);
            if (s.guided) {
              const GuideDesc gd = s.gdesc[map];
              uint32_t gt = kOutside;
              if ((unsigned)qx < gd.w && (unsigned)qy < gd.h)
                gt = __ldg(&s.guides[gd.off + (size_t)st.level * gd.w * gd.h + (size_t)qy * gd.w + qx]);
              nps = lut4(lg, __vabsdiffu4(nr.z, gt), nps);
            }
            term[i] = nps;
            c += dc;
            j += dj;
            if (j >= nk) {
              j -= nk;
              ++c;
            }
          }
        }
      }
    }
    __syncthreads();  // the mean, the records, the candidates and the LUT sums
    const uint32_t ncoh = sh_ncoh, nc = ncoh + s.m;
    if (sh_flags & 2) {
      if (tid == 0) write_bad_result(s, st, b, local, pixel);
      __syncthreads();
      continue;
    }
    // the weights: into the records (for the sequential form) and, as
    // floats, into w.term
    {
      const double avg = sh_mean;
      bool nan_w = false;
      for (uint32_t j = tid; j < nk; j += T) {
        const float wv = neighbour_weight(sh.dist[j], avg, tab_ff);
        nan_w |= (wv != wv);
        w.nbr[j].w = __float_as_uint(wv);
        w.term[j] = wv;
      }
      if (nan_w) atomicOr(&sh_flags, 1);
    }
    __syncthreads();
    float best_s = FLT_MAX;
    uint32_t best_i = 0;
    if (!st.slow_lut && !(sh_flags & 1)) {
      float my_s = FLT_MAX;
      uint32_t my_i = 0xffffffffu;
      for (uint32_t cc = tid; cc < nc; cc += T) {
        float sc = 0.0f;
        const float *tc = term + (size_t)cc * nk;
        for (uint32_t jj = 0; jj < nk; ++jj) sc = __fadd_rn(sc, __fmul_rn(tc[jj], w.term[jj]));
        if (sc < my_s) {  // first strict minimum among this thread's candidates
          my_s = sc;
          my_i = cc;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, my_s, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, my_i, o);
        if (ov < my_s || (ov == my_s && oi < my_i)) {
          my_s = ov;
          my_i = oi;
        }
      }
      if (lane == 0) {
        red_s[warp] = my_s;
        red_i[warp] = my_i;
      }
      __syncthreads();
      best_s = red_s[0];
      best_i = red_i[0];
      for (int i = 1; i < NW; ++i) {
        if (red_s[i] < best_s || (red_s[i] == best_s && red_i[i] < best_i)) {
          best_s = red_s[i];
          best_i = red_i[i];
        }
      }
      if (best_i == 0xffffffffu) {  // no score below f32::MAX: the reference keeps candidate 0
        best_s = FLT_MAX;
        best_i = 0;
      }
    } else if (costs_in_order<kCostAny>(st) && !(sh_flags & 1)) {
      if (warp == 0) best_in_order(s, st, w, lc, lg, nk, nc, best_s, best_i);
    } else if (tid == 0) {
      sequential_best(s, st, w, lc, lg, nk, nc, best_s, best_i);
    }
    if (tid == 0) write_result(s, st, w, b, local, pixel, px, py, is_new, nc, best_s, best_i);
    __syncthreads();
  }
}

__global__ void k_commit(SessionDev s, StageDev st, BatchDev b) {
  pdl_enter(); commit_body(s, st, b, blockIdx.x); }
__global__ void k_commit_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  commit_body(*v.s, v.d->st, v.d->b, v.vb);
}

__global__ void k_level_switch(SessionDev s, uint32_t level, uint32_t n_res) {
  pdl_enter();
  level_switch_body(s, level, n_res, blockIdx.x);
}
__global__ void k_level_switch_multi(MultiLaunch ml) {
  pdl_enter();
  const SegView v = find_segment(ml);
  level_switch_body(*v.s, v.d->level, v.d->ls_n_res, v.vb);
}

inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

template <typename... KArgs, typename... Args>
void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace

size_t resolve_smem_bytes(uint32_t k, uint32_t m) { return 2048 + (size_t)kResolveWarps * warp_smem_bytes(k, m); }
static size_t team_smem_bytes(uint32_t k, uint32_t m) { return 2048 + warp_smem_bytes(k, m) + (size_t)(k ? k : 1) * 4; }
// the full-evaluation team form keeps every (candidate, neighbour) term
static size_t team_full_smem_bytes(uint32_t k, uint32_t m) {
  const size_t kk = k ? k : 1;
  return 2048 + warp_smem_bytes(k, m) + ((kk * (k + m) * 4 + 7) & ~(size_t)7) + (size_t)(k + m) * 8;
}
constexpr size_t kTeamFullMaxSmem = 96 * 1024;

// Raises (never lowers) a kernel's dynamic shared-memory limit on the
// current device, so that sessions with different (k, m) can be built in
// any order and run later.
template <typename K>
static cudaError_t raise_smem(K *kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, size_t> cur;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cur.find({dev, (const void *)kernel});
  if (it == cur.end()) {
    // without the opt-in, static plus dynamic shared memory stays within 48 KB
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    it = cur.emplace(std::make_pair(dev, (const void *)kernel),
                     fa.sharedSizeBytes < 48 * 1024 ? 48 * 1024 - fa.sharedSizeBytes : 0)
             .first;
  }
  size_t &c = it->second;
  if (bytes <= c) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) c = bytes;
  return e;
}

cudaError_t configure_kernels(uint32_t k, uint32_t m, uint32_t n_maps) {
  cudaError_t e = raise_smem(k_resolve, resolve_smem_bytes(k, m));
  if (e != cudaSuccess) return e;
  e = raise_smem(k_resolve_lean, resolve_smem_bytes(k, m));
  if (e != cudaSuccess) return e;
  e = raise_smem(k_resolve_signed, resolve_smem_bytes(k, m));
  if (e != cudaSuccess) return e;
  e = raise_smem(k_knn_exhaustive, kExhAllKeys * 8);
  if (e != cudaSuccess) return e;
  e = raise_smem(k_mean_staged, (size_t)k * kMeanThreads * 8);
  if (e != cudaSuccess) return e;
  e = raise_smem(k_mean_ahead, (size_t)k * kMeanPitch * 8);
  if (e != cudaSuccess) return e;
  e = raise_smem(k_resolve_team<kTeamThreads, false>, team_smem_bytes(k, m));
  if (e != cudaSuccess) return e;
  if (k > 0 && k <= kSmallK && small_smem_bytes(k, m, n_maps) <= kSmallMaxSmem) {
    const size_t b = small_smem_bytes(k, m, n_maps);
    for (auto kernel :
         {k_resolve_small<512, false, kCostPlain>, k_resolve_small<512, true, kCostPlain>,
          k_resolve_small<256, false, kCostPlain>, k_resolve_small<256, true, kCostPlain>,
          k_resolve_small<128, false, kCostPlain>, k_resolve_small<128, true, kCostPlain>,
          k_resolve_small<512, true, kCostSigned>, k_resolve_small<256, true, kCostSigned>}) {
      e = raise_smem(kernel, b);
      if (e != cudaSuccess) return e;
    }
  }
  const size_t fsm = team_full_smem_bytes(k, m);
  if (fsm <= kTeamFullMaxSmem) {
    e = raise_smem(k_resolve_team<kTeamFullThreads, true>, fsm);
    if (e != cudaSuccess) return e;
    e = raise_smem(k_resolve_team<kStepWideThreads, true>, fsm);
    if (e != cudaSuccess) return e;
    e = raise_smem(k_step_team_full<kTeamFullThreads>, std::max<size_t>(fsm, (size_t)kExhAllKeys * 8));
    if (e != cudaSuccess) return e;
    return raise_smem(k_step_team_full<kStepWideThreads>, std::max<size_t>(fsm, (size_t)kExhAllKeys * 8));
  }
  return cudaSuccess;
}

cudaError_t set_multi_smem(int phase, size_t bytes) {
  switch (phase) {
    case kPhaseExhaustive: return raise_smem(k_knn_exhaustive_multi, bytes);
    case kPhaseResolve: {
      const cudaError_t e = raise_smem(k_resolve_multi, bytes);
      return e != cudaSuccess ? e : raise_smem(k_resolve_multi_lean, bytes);
    }
    case kPhaseTeamPart: return raise_smem(k_resolve_team_multi<kTeamThreads, false>, bytes);
    case kPhaseTeamFull: return raise_smem(k_resolve_team_multi<kTeamFullThreads, true>, bytes);
    default: return cudaSuccess;
  }
}

bool team_full_fits(uint32_t k, uint32_t m) { return team_full_smem_bytes(k, m) <= kTeamFullMaxSmem; }


uint32_t multi_threads(int phase) {
  switch (phase) {
    case kPhaseLevelSwitch: return 256;
    case kPhaseRandom: return 128;
    case kPhaseWalk: return kWalkWarps * kWarp;
    case kPhaseExhaustive: return kExhThreads;
    case kPhaseMean: return 128;
    case kPhaseResolve: return kResolveWarps * kWarp;
    case kPhaseTeamPart: return kTeamThreads;
    case kPhaseTeamFull: return kTeamFullThreads;
    default: return 256;
  }
}

uint32_t multi_blocks(int phase, uint32_t n, uint32_t cap) {
  if (n == 0) return 0;
  uint32_t b = 0;
  switch (phase) {
    case kPhaseLevelSwitch: b = cdiv(n, 256); break;
    case kPhaseRandom: b = cdiv(n, 128); break;
    case kPhaseWalk: b = cdiv(n, kWalkWarps * std::min(8u, std::max(1u, n / 4096u))); break;
    case kPhaseExhaustive: b = n; break;
    case kPhaseMean: b = cdiv(n, 128); break;
    case kPhaseResolve: b = cdiv(n, kResolveWarps); break;
    case kPhaseTeamPart:
    case kPhaseTeamFull: b = n; break;
    default: b = cdiv(n, 256); break;
  }
  // only the grid-stride phases may take fewer blocks than items need
  const bool strided = phase == kPhaseWalk || phase == kPhaseExhaustive || phase == kPhaseResolve ||
                       phase == kPhaseTeamPart || phase == kPhaseTeamFull;
  if (strided && cap && b > cap) b = cap;
  return b;
}

size_t multi_smem_bytes(int phase, uint32_t k, uint32_t m) {
  switch (phase) {
    case kPhaseExhaustive: return (size_t)kExhAllKeys * 8;
    case kPhaseResolve: return resolve_smem_bytes(k, m);
    case kPhaseTeamPart: return team_smem_bytes(k, m);
    case kPhaseTeamFull: return team_full_smem_bytes(k, m);
    default: return 0;
  }
}

static constexpr uint32_t kResolveOneLaunch = 152u * 8u * 8u;
uint32_t resolve_launches(uint32_t n_lean, uint32_t n_segs, uint32_t blocks) {
  return n_lean && n_lean < n_segs && blocks > kResolveOneLaunch ? 2 : 1;
}

void launch_multi(int phase, const MultiLaunch &ml, uint32_t blocks, size_t smem, cudaStream_t stream) {
  if (blocks == 0) return;  // a launch may carry only the exhaustive k-NN's fallback pool (no segments)
  const uint32_t t = multi_threads(phase);
  switch (phase) {
    case kPhaseLevelSwitch: launch_pdl(k_level_switch_multi, blocks, t, 0, stream, ml); break;
    case kPhaseRandom: launch_pdl(k_random_candidates_multi, blocks, t, 0, stream, ml); break;
    case kPhaseWalk: launch_pdl(k_knn_walk_multi, blocks, t, 0, stream, ml); break;
    case kPhaseExhaustive: launch_pdl(k_knn_exhaustive_multi, blocks, t, smem, stream, ml); break;
    case kPhaseMean: launch_pdl(k_mean_multi, blocks, t, 0, stream, ml); break;
    case kPhaseResolve: {
      // Segments [0, n_lean) belong to sessions without guides (blocks
      // [0, lean_blocks)).  Two launches, one after the other, each wait for
      // their slowest item, so both kinds share one up to eight rounds of the
      // GPU's blocks (16 requests: two launches 21.2 ms, one up to 2, 4, 8, 16
      // rounds 20.0, 19.5, 19.4, 19.3); beyond, where the work counts, the
      // lean kernel spills less (24 sessions of up to 1024^2: 64.0 ms against
      // 64.5 always in one)
      if (ml.n_lean < ml.n_segs && resolve_launches(ml.n_lean, ml.n_segs, blocks) == 1) {
        launch_pdl(k_resolve_multi, blocks, t, smem, stream, ml);
        break;
      }
      MultiLaunch a = ml, g = ml;
      a.n_segs = ml.n_lean;
      g.segs = ml.segs + ml.n_lean;
      g.n_segs = ml.n_segs - ml.n_lean;
      g.block_base = ml.block_base + ml.lean_blocks;
      if (a.n_segs) launch_pdl(k_resolve_multi_lean, ml.lean_blocks, t, smem, stream, a);
      if (g.n_segs) launch_pdl(k_resolve_multi, blocks - ml.lean_blocks, t, smem, stream, g);
      break;
    }
    case kPhaseTeamPart: launch_pdl(k_resolve_team_multi<kTeamThreads, false>, blocks, t, smem, stream, ml); break;
    case kPhaseTeamFull: launch_pdl(k_resolve_team_multi<kTeamFullThreads, true>, blocks, t, smem, stream, ml); break;
    case kPhaseCommit: launch_pdl(k_commit_multi, blocks, t, 0, stream, ml); break;
    default: break;
  }
}

void launch_random_candidates(const SessionDev &s, const StageDev &st, cudaStream_t stream) {
  if (st.n_items == 0 || s.m == 0) return;
  launch_pdl(k_random_candidates, cdiv(st.n_items, 128), 128, 0, stream, s, st);
}

// Items per warp of a walk over n items: one while a warp per item fits the
// GPU, then as many as keep its warps (152 SMs x 32) busy some four times
// over.
static uint32_t walk_items(uint32_t n) { return std::min(32u, std::max(1u, n / (152u * 32u * 4u))); }

void launch_knn_walk(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream,
                     const PendingCommit &pc) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 && pc.n == 0) return;
  const uint32_t grid = std::max(cdiv(n, kWalkWarps * walk_items(n)), cdiv(pc.n, kWalkWarps * kWarp));
  if (b.walk_window)
    launch_pdl(k_knn_walk<true>, grid, kWalkWarps * kWarp, kWalkWinBytes, stream, s, st, b, pc);
  else
    launch_pdl(k_knn_walk<false>, grid, kWalkWarps * kWarp, 0, stream, s, st, b, pc);
}

uint32_t exh_key_cap(const SessionDev &s, const BatchDev &b) {
  // every point and its (at most two) tiling mirrors while they fit, else
  // the cell grid's rings (a few times k keys; an overflow falls back to
  // rescanning the points, exactly)
  const uint64_t want = b.n_res <= kExhGridFrom ? (uint64_t)b.n_res * (s.tiling ? 3 : 1) + 64 : 2048;
  return (uint32_t)std::min<uint64_t>(kExhAllKeys, std::max<uint64_t>(want, 4u * std::max<uint32_t>(s.k, 64u)));
}

void launch_knn_exhaustive(const SessionDev &s, const StageDev &st, const BatchDev &b, bool all_items,
                           cudaStream_t stream, const PendingCommit &pc) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 && pc.n == 0) return;
  uint32_t grid = n < 608u ? n : 608u;  // 152 SMs x 4 CTAs, grid-stride beyond
  grid = std::max(grid, std::min(608u, cdiv(pc.n, kExhThreads)));
  const uint32_t cap = exh_key_cap(s, b);
  launch_pdl(k_knn_exhaustive, grid, kExhThreads, (size_t)cap * 8, stream, s, st, b, cap, all_items ? 1 : 0, pc);
}

bool knn_list_fits(const SessionDev &s, const BatchDev &b) { return s.rank != nullptr && b.n_res <= kListMax; }

void launch_knn_list(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0) return;
  launch_pdl(k_knn_list, cdiv(n, kListWarps), kListWarps * kWarp, (size_t)kListWarps * list_cap(s.k) * 8, stream, s, st,
             b);
}

void launch_mean(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 || s.k == 0) return;
  launch_pdl(k_mean_staged, cdiv(n, kMeanThreads), kMeanThreads, (size_t)s.k * kMeanThreads * 8, stream, s, st, b);
}

void launch_mean_ahead(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 || s.k == 0) return;
  launch_pdl(k_mean_ahead, cdiv(n, kMeanThreads), kMeanAheadThreads, (size_t)s.k * kMeanPitch * 8, stream, s, st, b);
}

void launch_dist_tables(const SessionDev &s, double *xdiv, double *ydiv, double *dxt, double *dy2t, uint32_t n_x,
                        uint32_t n_y, cudaStream_t stream) {
  const uint64_t n = (uint64_t)n_x + n_y + (uint64_t)(s.W + s.H) * (2 * s.dtab_r + 1);
  k_dist_tables<<<(uint32_t)std::min<uint64_t>((n + 255) / 256, 152 * 8), 256, 0, stream>>>(s, xdiv, ydiv, dxt, dy2t,
                                                                                             n_x, n_y);
}

// Resident blocks of a kernel on the current device (cached per kernel and
// dynamic shared-memory size).
template <typename K>
static uint32_t resident_blocks(K *kernel, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<const void *, size_t>, uint32_t> cache;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find({(const void *)kernel, smem});
  if (it != cache.end()) return it->second;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm <= 0)
    return 0;  // unknown: the caller keeps a full grid
  const uint32_t n = (uint32_t)sms * (uint32_t)per_sm;
  cache[{(const void *)kernel, smem}] = n;
  return n;
}

void launch_resolve(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream,
                    const PendingCommit &pc) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 && pc.n == 0) return;
  const size_t smem = resolve_smem_bytes(s.k, s.m);
  const auto kernel = !s.guided ? k_resolve_lean : st.slow_lut == kLutSigned ? k_resolve_signed : k_resolve;
  uint32_t grid = cdiv(n, kResolveWarps);
  if (b.work_ctr) {
    // a resident grid whose warps take further items from the counter
    const uint32_t cap = resident_blocks(kernel, kResolveWarps * kWarp, smem);
    if (cap) grid = std::min(grid, cap);
  }
  grid = std::max(grid, cdiv(pc.n, kResolveWarps * kWarp));
  launch_pdl(kernel, grid, kResolveWarps * kWarp, smem, stream, s, st, b, pc);
}

// The small-step form: up to kSmallK neighbours, the term rows within
// kSmallMaxSmem.
static bool small_fits(const SessionDev &s) {
  return s.k > 0 && s.k <= kSmallK && small_smem_bytes(s.k, s.m, s.n_maps) <= kSmallMaxSmem;
}

template <int T>
static void launch_small_t(const SessionDev &s, const StageDev &st, const BatchDev &b, uint32_t F, cudaStream_t stream,
                           const PendingCommit &pc) {
  const uint32_t grid = std::max(1u, b.i1 - b.i0);
  const size_t smem = small_smem_bytes(s.k, s.m, s.n_maps);
  if (!s.guided)
    launch_pdl(k_resolve_small<T, false, kCostPlain>, grid, T, smem, stream, s, st, b, pc, F);
  else if (T != 128 && st.slow_lut == kLutSigned)
    launch_pdl(k_resolve_small<(T != 128 ? T : 256), true, kCostSigned>, grid, T, smem, stream, s, st, b, pc, F);
  else
    launch_pdl(k_resolve_small<T, true, kCostPlain>, grid, T, smem, stream, s, st, b, pc, F);
}

// Threads per item by the step's items: 512 while every item has an SM, 256
// while the items are resident together, else 128.  F: see k_resolve_small.
static void launch_small(const SessionDev &s, const StageDev &st, const BatchDev &b, bool full, cudaStream_t stream,
                         const PendingCommit &pc) {
  const uint32_t n = b.i1 - b.i0;
  if (full && n <= 152u)
    launch_small_t<512>(s, st, b, s.k, stream, pc);
  else if (full)
    launch_small_t<256>(s, st, b, s.k, stream, pc);
  else
    launch_small_t<128>(s, st, b, kSmallFirst, stream, pc);
}

void launch_resolve_team(const SessionDev &s, const StageDev &st, const BatchDev &b, bool full,
                         cudaStream_t stream, const PendingCommit &pc) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0 && pc.n == 0) return;
  // larger steps of more than one round of neighbours are bound by work per
  // item, not its latency: the early-exit form below (k = m = 50: 2.49
  // against 2.60 ms a 256^2 call; k = m = 8: 1.40 against 1.33).  Costs that
  // have to be looked at in order leave early less often: full scoring
  // (guided inpainting, 250^2 0.53 against 0.58 ms, 256^2 0.53 against 0.54,
  // 512^2 0.90 either way), else the warp form's copy.
  const bool in_order = st.slow_lut == kLutSigned;
  if (small_fits(s) && (full || s.k <= kWarp || in_order)) {
    launch_small(s, st, b, full || in_order, stream, pc);
    return;
  }
  if (in_order) {
    launch_resolve(s, st, b, stream, pc);
    return;
  }
  uint32_t grid = n < 152u * 16u ? n : 152u * 16u;
  grid = std::max(grid, std::min(152u * 16u, cdiv(pc.n, kTeamThreads)));
  if (full && team_full_smem_bytes(s.k, s.m) <= kTeamFullMaxSmem && n <= 152u && pc.n == 0)
    // at most one item per SM of a GB300: twice the threads per item
    launch_pdl(k_resolve_team<kStepWideThreads, true>, grid, kStepWideThreads, team_full_smem_bytes(s.k, s.m), stream,
               s, st, b, pc);
  else if (full && team_full_smem_bytes(s.k, s.m) <= kTeamFullMaxSmem)
    launch_pdl(k_resolve_team<kTeamFullThreads, true>, grid, kTeamFullThreads, team_full_smem_bytes(s.k, s.m), stream, s,
               st, b, pc);
  else
    launch_pdl(k_resolve_team<kTeamThreads, false>, grid, kTeamThreads, team_smem_bytes(s.k, s.m), stream, s, st, b,
               pc);
}

void launch_step_team_full(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0) return;
  const uint32_t grid = n < 608u ? n : 608u;
  const uint32_t cap = exh_key_cap(s, b);
  const size_t smem = std::max<size_t>((size_t)cap * 8, team_full_smem_bytes(s.k, s.m));
  if (n <= 152u)  // at most one item per SM of a GB300
    launch_pdl(k_step_team_full<kStepWideThreads>, grid, kStepWideThreads, smem, stream, s, st, b, cap);
  else
    launch_pdl(k_step_team_full<kTeamFullThreads>, grid, kTeamFullThreads, smem, stream, s, st, b, cap);
}

void launch_commit(const SessionDev &s, const StageDev &st, const BatchDev &b, cudaStream_t stream) {
  const uint32_t n = b.i1 - b.i0;
  if (n == 0) return;
  launch_pdl(k_commit, cdiv(n, 256), 256, 0, stream, s, st, b);
}

void launch_level_switch(const SessionDev &s, uint32_t level, uint32_t n_res, cudaStream_t stream) {
  if (n_res == 0) return;
  launch_pdl(k_level_switch, cdiv(n_res, 256), 256, 0, stream, s, level, n_res);
}

void launch_pad(const uint32_t *src, uint32_t w, uint32_t h, uint32_t levels, uint32_t pitch, uint32_t *dst,
                cudaStream_t stream) {
  const size_t n = (size_t)pitch * (h + 2 * kPad) * levels;
  if (n == 0) return;
  k_pad<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, stream>>>(src, w, h, levels, pitch, dst);
}

static uint32_t pick_grid(uint64_t n) { return (uint32_t)std::min<uint64_t>((n + 255) / 256, 152 * 32); }
void launch_pick_init(uint32_t *un, uint32_t n, const uint32_t *over, uint32_t n_over, cudaStream_t stream) {
  if (n) k_pick_init<<<pick_grid(n), 256, 0, stream>>>(un, n);
  if (n_over) k_pick_over<<<pick_grid(n_over), 256, 0, stream>>>(un, over, n_over);
}
void launch_picks(const PickStage &ps, cudaStream_t stream) {
  if (ps.redo + ps.n_new == 0) return;
  k_pick_draw<<<pick_grid((uint64_t)ps.redo + ps.n_new), 256, 0, stream>>>(ps);
  if (ps.n_new) k_pick_follow<<<pick_grid(ps.len0), 256, 0, stream>>>(ps);
}

void launch_pick_chains(const PickChain *chains, uint32_t n, cudaStream_t stream) {
  if (n) k_pick_chain<<<n, kPickChainThreads, 0, stream>>>(chains);
}

void launch_tree_append(const SessionDev &s, const StageDev &st, uint32_t a0, uint32_t a1, uint32_t pos0,
                        uint32_t nomir_end, cudaStream_t stream) {
  if (a1 <= a0) return;
  launch_pdl(k_tree_append, cdiv(a1 - a0, 256), 256, 0, stream, s, st, a0, a1, pos0, nomir_end);
}

void launch_rank_init(const SessionDev &s, uint32_t n, cudaStream_t stream) {
  if (n == 0) return;
  k_rank_init<<<cdiv(n, 256), 256, 0, stream>>>(s, n);
}

void launch_inpaint_init(const SessionDev &s, const InpaintDev &in, cudaStream_t stream) {
  const uint32_t words = s.wpr * s.H;
  if (words) k_inpaint_init<<<(words + 7) / 8, 256, 0, stream>>>(s, in);
}

void launch_scatter_init(const uint32_t *list, uint32_t n, uint32_t *color, uint4 *state, uint32_t *res,
                         cudaStream_t stream) {
  if (n == 0) return;
  k_scatter_init<<<(n + 127) / 128, 128, 0, stream>>>(list, n, color, state, res);
}

void launch_transform_apply(const uint32_t *buf, size_t n, const uint32_t *texels, const uint4 *maps,
                            uint32_t n_maps, uint32_t *out, int *err, cudaStream_t stream) {
  if (n == 0) return;
  k_transform_apply<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, stream>>>(buf, n, texels, maps,
                                                                                                n_maps, out, err);
}

void launch_debug_maps(const uint32_t *ids, size_t n, const uint32_t *flat, const float *score, size_t n_res,
                       uint32_t *patch_rgba, uint32_t *map_rgba, uint32_t *unc_rgba, cudaStream_t stream) {
  if (n > 0)
    k_id_maps<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, stream>>>(ids, n, patch_rgba, map_rgba);
  if (n_res > 0)
    k_uncertainty<<<(uint32_t)std::min<size_t>((n_res + 255) / 256, 152 * 16), 256, 0, stream>>>(flat, score, n_res, n,
                                                                                                  unc_rgba);
}

void launch_luma_hist(const uint32_t *src, size_t n, uint8_t *luma, uint32_t *hist, cudaStream_t stream) {
  if (n == 0) return;
  k_luma_hist<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 4), 256, 0, stream>>>(src, n, luma, hist);
}

void launch_hist_r(const uint32_t *src, size_t n, uint32_t *hist, cudaStream_t stream) {
  if (n == 0) return;
  k_hist_r<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 4), 256, 0, stream>>>(src, n, hist);
}

void launch_apply_map(const uint8_t *luma, size_t n, const uint8_t *map, uint32_t *out, cudaStream_t stream) {
  if (n == 0) return;
  k_apply_map<<<(uint32_t)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, stream>>>(luma, n, map, out);
}

void launch_resize_v(const uint8_t *src, uint32_t w, uint32_t h, float *tmp, uint32_t nh, const uint4 *taps,
                     const float *wts, cudaStream_t stream) {
  if (w == 0 || nh == 0) return;
  dim3 grid(cdiv(w, 128), nh);
  k_resize_v<<<grid, 128, 0, stream>>>(src, w, h, tmp, nh, taps, wts);
}

void launch_resize_v_jobs(const ResizeJob *jobs, uint32_t n, uint32_t blocks, cudaStream_t stream) {
  if (n == 0 || blocks == 0) return;
  k_resize_v_jobs<<<blocks, 128, 0, stream>>>(jobs, n);
}

void launch_resize_h_jobs(const ResizeJob *jobs, uint32_t n, uint32_t blocks, cudaStream_t stream) {
  if (n == 0 || blocks == 0) return;
  k_resize_h_jobs<<<blocks, 128, 0, stream>>>(jobs, n);
}

void launch_resize_h(const float *tmp, uint32_t w, uint32_t nh, uint8_t *dst, uint32_t nw, const uint4 *taps,
                     const float *wts, cudaStream_t stream) {
  if (nw == 0 || nh == 0) return;
  dim3 grid(cdiv(nw, 128), nh);
  k_resize_h<<<grid, 128, 0, stream>>>(tmp, w, nh, dst, nw, taps, wts);
}

}  // namespace ts

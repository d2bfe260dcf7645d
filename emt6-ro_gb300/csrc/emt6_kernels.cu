// emt6_kernels.cu -- sm_103a kernels of the EMT6-Ro batched simulation step.
//
// One CTA of 96 threads (one warp per substrate field) owns one simulation for
// a whole launch of N steps: the fields, the site-state bytes and the occupied
// list live in shared memory for the launch; per-site cell records (48 B)
// stay in global memory, where the few hundred live cells of each resident
// simulation stay L2-resident.  Three kernels: run_kernel<kTierNarrow> (5 CTAs/SM, a
// window of at most 40 lattice rows on chip) for regions that fit a tile of 32
// slots per lane, run_kernel<kTierWide> (4 CTAs/SM, the whole lattice) for
// larger ones (on the default lattice; smem_layout has the others), and
// run_kernel<kTierLone> (384 threads, 1 CTA/SM) for batches of at most one
// simulation per SM and for the large regions of some others.  Per step (reference
// cadence, src/emt6ro/simulation/simulation.cu:153-166):
//   t % 128 == 0  rebuild the occupied list        (simulation.cu:41-64)
//   t % 32  == 0  ROI + circular fixed-value mask   (diffusion.cu:65-100)
//   diffusion: 23 substeps over free sites + 1 over the ROI (diffusion.cu:135-191),
//     each field in the registers of one warp, or of four (emt6_tiles.cuh)
//   cell update: 8-neighbour vacancy snapshot, Site::step per list entry,
//     at most one division per simulation (simulation.cu:66-110).
// Randomness is Philox keyed by (step, simulation, site, occurrence), so the
// results do not depend on the launch shape, nor on the order in which CTAs
// take simulations: before every chunk of steps three small kernels sort the
// simulations by their region, largest first, so that the CTAs resident on
// an SM run the same tile code (launch_order).
#include <cuda_runtime.h>

#include <cstdint>

#include "emt6_device.cuh"
#include "emt6_kernels.h"
#include "emt6_tiles.cuh"

namespace emt6 {

__device__ unsigned long long g_instr_counts[4];  // decisions, kills, irradiations, divisions
__device__ double g_instr_sum_death_prob;
__device__ unsigned long long g_instr_hist[600];  // irradiation bins, then time-in-repair

constexpr int kThreads = 96;  // one warp per field
// kTierLone: the wide kernel's registers for as many warps as an SM holds.  All
// take part in the cell update, the list and the diffusion of large regions.
constexpr int kThreadsLone = 384;
__host__ __device__ constexpr int threads_of(int tier) { return tier == kTierLone ? kThreadsLone : kThreads; }

struct Misc {
  float4 met[4];  // consumption by metabolic mode
  int roi[5];  // r0, c0, h, w, dist
  uint32_t n, n0;
  int has_multi;
  int edge;  // a cell has divided onto the last row or column
  int winner, target;
  unsigned int ins[4];
  double ins_dp;
  unsigned long long diffused;
  unsigned long long nfs;  // free sites of the current mask
  TileMap tm;    // the region's tile
  int park;      // the narrow kernel cannot take the next step of this simulation
  int w0, wneed;  // first row of the field window on chip (-1: none), the one the region needs
  // behind it, for each warp: reductions, and its rows' list entries per stripe
  __device__ int (*red())[4] { return reinterpret_cast<int (*)[4]>(this + 1); }
  __device__ uint32_t (*stripe())[32] {
    return reinterpret_cast<uint32_t (*)[32]>(red() + (blockDim.x >> 5));
  }
};
constexpr uint32_t kMiscPerWarp = 4 * 4 + 32 * 4;

__host__ __device__ inline uint32_t align_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

// Rows of the field window and entries of the occupied list on chip, by tier of
// launch.  kTierNarrow holds the region's rows (35 at most) with room to move,
// and as many list entries as leave 5 CTAs on an SM; fewer rows or entries would
// only park simulations.  kTierWide holds the whole lattice and 4 CTAs (12 warps,
// 3 on each quarter of the SM; with 3 CTAs one quarter has 3 warps and the CTAs
// wait for it: 23% slower diffusion).  Its list may hold every interior site;
// what does not fit of the entries' clocks lies in the padding of the cell
// records, entry by entry (`held` of them are on chip).  kMinEntries are held on
// any lattice, so the counts are those of lattices up to 53 x 53 sites: larger ones
// have 3 CTAs of the wide tier, and the largest (56 x 62) 4 of the narrow one.
constexpr int kWindowRows = 40;
constexpr uint32_t kEntryBytes = 4 + 4 + 2 + 1, kMinEntries = 1024;

struct SmemLayout {
  uint32_t fld, st, colmask, masks, edge, parts, misc, h0, h1, list, fl, total;
  int rows, plane;    // window rows, floats of a field's window
  int entries, held;  // list capacity, entries with their clocks on chip
};

__host__ __device__ inline SmemLayout smem_layout(int H, int W, int lcap, int tier) {
  SmemLayout L;
  const bool wide = tier != kTierNarrow;
  const int HW = H * W;
  L.rows = wide || H < kWindowRows ? H : kWindowRows;
  L.plane = L.rows * W;
  uint32_t o = 0;
  // the whole-lattice fld region matches the global per-simulation stride
  // (3*HW padded to 32 floats), the st region HW padded to 128 bytes, so
  // whole-stride copies stay inside
  L.fld = o; o += align_up(3u * (uint32_t)L.plane, 32) * 4u;
  L.st = o; o += align_up((uint32_t)HW, 128);
  L.colmask = o; o += 64 * 8;
  L.masks = o; o += 3u * (wide ? kWordsWide : kWordsNarrow) * 32u * 4u;
  L.edge = o; o += 3u * (wide ? kEdgeWide : kEdgeNarrow) * 4u;
  o = align_up(o, 16);
  L.parts = o; o += tier == kTierLone ? 3u * kPartSlots * 8u : 0u;
  L.misc = o; o += align_up(sizeof(Misc) + threads_of(tier) / 32 * kMiscPerWarp, 16);
  // a rebuilt list holds at most the interior, and 128 divisions can follow
  const uint32_t all = align_up((uint32_t)lcap - 128u, 16),
                 room = (tier == kTierLone ? 444u : wide ? 111u : 88u) * 512u;
  const uint32_t left = o < room ? room - o : 0u;
  uint32_t entries = all, held;
  if (wide) {
    held = left > 3u * all ? (left - 3u * all) / 8u : 0u;
  } else {
    held = left / kEntryBytes;
  }
  held = held > kMinEntries ? held & ~15u : kMinEntries;
  if (held > all) held = all;
  if (!wide) entries = held;
  L.entries = (int)entries;
  L.held = (int)held;
  L.h0 = o; o += held * 4u;
  L.h1 = o; o += held * 4u;
  L.list = o; o += entries * 2u;
  L.fl = o; o += entries;
  L.total = o;
  return L;
}

size_t run_kernel_smem(int H, int W, int lcap, int tier) {
  return smem_layout(H, W, lcap, tier).total;
}

// list entries on chip: site index in the low bits, vacant neighbours above
constexpr uint32_t kSiteBits = 12, kSiteMask = (1u << kSiteBits) - 1u;

// ---------------------------------------------------------------------------
// block reductions
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ int block_min(int v, Misc *m) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = __reduce_min_sync(kFull, v);
  if (lane == 0) m->red()[wid][0] = v;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) v = min(v, m->red()[w][0]);
  __syncthreads();
  return v;
}

// ---------------------------------------------------------------------------
// occupied list (simulation.cu:41-64): 32 column stripes, stripe k = columns
// k, k+32, ... < W-1 over rows 0..H-2, stripes concatenated in order.
// Called by all threads, each warp for its share of the rows.  More entries than
// `cap` parks the simulation with an empty list (the wide kernel rebuilds it in full).
// Like compute_roi a function of its own: inlined, the two cost the step kernels'
// loops registers (10,000 simulations of radius 6-14, 150 steps: 21.5 vs 21.7 ms).
// ---------------------------------------------------------------------------
template <int NT>
__device__ __noinline__ void rebuild_list(uint8_t *st, uint16_t *list, Misc *m, int H, int W, int HW, int cap) {
  constexpr int NWARP = NT / 32;
  const int k = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // the state region is padded to 128 bytes
  for (int q = threadIdx.x; q < (HW + 3) / 4; q += NT)
    reinterpret_cast<uint32_t *>(st)[q] &= kStMask * 0x01010101u;
  __syncthreads();
  // warp w counts, then writes, the rows of its share in every stripe
  const int per = (H - 1 + NWARP - 1) / NWARP, ra = min(wid * per, H - 1), rb = min(ra + per, H - 1);
  const int c0 = k < W - 1, c1 = k + 32 < W - 1;
  uint32_t cnt = 0;
#pragma unroll 4
  for (int r = ra; r < rb; ++r) {
    const uint8_t *q = st + r * W + k;
    cnt += (c0 && q[0] == kOccupied) + (c1 && q[32] == kOccupied);
  }
  m->stripe()[wid][k] = cnt;
  __syncthreads();
  uint32_t before = 0, all = 0;  // of this stripe: earlier rows; all rows
#pragma unroll
  for (int w = 0; w < NWARP; ++w) {
    const uint32_t v = m->stripe()[w][k];
    if (w < wid) before += v;
    all += v;
  }
  uint32_t incl = all;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (k >= o) incl += y;
  }
  uint32_t off = incl - all + before;
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  const bool fits = total <= (uint32_t)cap;
  if (fits) {
#pragma unroll 4
    for (int r = ra; r < rb; ++r) {
      const int q = r * W + k;
      if (c0 && st[q] == kOccupied) {
        list[off++] = (uint16_t)q;
        st[q] = kOccupied | kStRebuilt;
      }
      if (c1 && st[q + 32] == kOccupied) {
        list[off++] = (uint16_t)(q + 32);
        st[q + 32] = kOccupied | kStRebuilt;
      }
    }
  }
  if (threadIdx.x == 0) {
    m->n = m->n0 = fits ? total : 0u;
    m->has_multi = 0;
    if (!fits) m->park = 1;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// ROI + mask (diffusion.cu:16-100).  colmask[j] bit i = site (i, j) of the
// (h+2) x (w+2) region is free (not held at the external level): its distance
// from the region's centre is below dist.  The squared distances are multiples
// of 1/4 and exact, so they compare with dist^2 as their rounded roots do with
// dist; a column's free rows are an interval, found from the root and moved to
// the exact bound.  Called by threads 0..63.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void build_colmask(uint64_t *colmask, int h, int w, int dist) {
  if (threadIdx.x < 64) {
    const int j = threadIdx.x, mh = h + 2, mw = w + 2;
    uint64_t bits = 0;
    if (h > 0 && w > 0 && j < mw) {
      const float mr = mh / 2.f - 1.f, dc = (float)(j + 1) - mw / 2.f;  // row i is i - mr away
      const float lim = (float)(dist * dist) - dc * dc;
      if (lim > 0.f) {
        const float root = sqrtf(lim);
        int lo = max((int)ceilf(mr - root) - 1, 0), hi = min((int)floorf(mr + root) + 1, mh - 1);
        while (lo <= hi && (lo - mr) * (lo - mr) >= lim) ++lo;
        while (hi >= lo && (hi - mr) * (hi - mr) >= lim) --hi;
        if (lo <= hi) bits = (~0ull >> (63 - hi)) & (~0ull << lo);
      }
    }
    colmask[j] = bits;
  }
}

// row of site s: s / W for s < 4096 and W < 64 (inv = ceil(2^20 / W): the
// product's error s (inv W - 2^20) / (2^20 W) stays below 1 / W)
__device__ __forceinline__ int row_of(int s, uint32_t inv) { return (int)((uint32_t)s * inv >> 20); }

// The occupied sites are all in the list (rebuilt, then appended to), but for cells
// that divided onto a vacant border site of the last row or column (m->edge): the
// list leaves them out at its next rebuild (simulation.cu:50-53), the region does not.
template <int NT>
__device__ __noinline__ void compute_roi(const uint8_t *st, const uint16_t *list, uint64_t *colmask, Misc *m,
                            int H, int W) {
  constexpr int NWARP = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t n = m->n, all = n + (m->edge ? H + W - 1 : 0), inv = ((1u << 20) + W - 1) / W;
  const auto site = [&](uint32_t e) -> int {  // of the list, the last row, the last column
    if (e < n) return list[e] & kSiteMask;
    const int q = (int)(e - n);
    return q < W ? (H - 1) * W + q : (q - W) * W + W - 1;
  };
  int v[4] = {H, W, 0, 0};
  for (uint32_t e = threadIdx.x; e < all; e += NT) {
    const int s = site(e);
    if ((st[s] & kStMask) == kOccupied) {
      const int r = row_of(s, inv), c = s - r * W;
      v[0] = min(v[0], r); v[1] = min(v[1], c);
      v[2] = max(v[2], r); v[3] = max(v[3], c);
    }
  }
  v[0] = __reduce_min_sync(kFull, v[0]);
  v[1] = __reduce_min_sync(kFull, v[1]);
  v[2] = __reduce_max_sync(kFull, v[2]);
  v[3] = __reduce_max_sync(kFull, v[3]);
  if (lane == 0)
    for (int k = 0; k < 4; ++k) m->red()[wid][k] = v[k];
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NWARP; ++w) {
    v[0] = min(v[0], m->red()[w][0]);
    v[1] = min(v[1], m->red()[w][1]);
    v[2] = max(v[2], m->red()[w][2]);
    v[3] = max(v[3], m->red()[w][3]);
  }
  __syncthreads();
  if (v[2] == 0 && v[3] == 0) {
    if (threadIdx.x == 0) m->roi[0] = m->roi[1] = m->roi[2] = m->roi[3] = m->roi[4] = 0;
    if (threadIdx.x < 64) colmask[threadIdx.x] = 0;
    __syncthreads();
    return;
  }
  const int midr = v[0] + (v[2] - v[0] + 1) / 2;
  const int midc = v[1] + (v[3] - v[1] + 1) / 2;
  int far = 0;  // largest squared distance
  for (uint32_t e = threadIdx.x; e < all; e += NT) {
    const int s = site(e);
    if ((st[s] & kStMask) == kOccupied) {
      const int r = row_of(s, inv), c = s - r * W;
      far = max(far, (midr - r) * (midr - r) + (midc - c) * (midc - c));
    }
  }
  far = __reduce_max_sync(kFull, far);
  if (lane == 0) m->red()[wid][0] = far;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NWARP; ++w) far = max(far, m->red()[w][0]);
  const int dist = (int)ceilf(sqrtf((float)far));
  const int sub_r = (midr <= dist) ? 1 : midr - dist;
  const int sub_c = (midc <= dist) ? 1 : midc - dist;
  const int sub_w = (midc + dist >= W - 1) ? W - 1 - sub_c : midc + dist - sub_c + 1;
  const int sub_h = (midr + dist >= H - 1) ? H - 1 - sub_r : midr + dist - sub_r + 1;
  if (threadIdx.x == 0) {
    m->roi[0] = sub_r; m->roi[1] = sub_c; m->roi[2] = sub_h; m->roi[3] = sub_w; m->roi[4] = dist;
  }
  build_colmask(colmask, sub_h, sub_w, dist);
  __syncthreads();
}

// The tile of the current region, its free-site count, and the field window
// it needs.  Block mode: an unclipped ROI of distance d (2d + 1 rows and
// columns) has its free sites in region rows and columns 1..2d, surrounded by
// fixed sites, so a tile holding just that block suffices, with every slot and
// neighbour outside it at the external level (the ROI's last row and column,
// 2d + 1, only change in the final substep).  Any other region (clipped
// against the lattice edge, where ring sites can be free and have zero
// neighbours outside the region) is held whole, its ring included, with zero
// around it.  A tile without CE (RE) needs one spare column (row) of constant
// slots: 2d and 8C are even, so a block that leaves any leaves two, and the
// ROI's last column is one of them.  Called by warp 0.
__device__ void tile_mapping(const uint64_t *colmask, Misc *m, uint32_t layouts, int tiles, int H,
                             int rows) {
  const int lane = threadIdx.x & 31;
  const int h = m->roi[2], w = m->roi[3], d = m->roi[4];
  const uint64_t c0 = colmask[lane], c1 = colmask[lane + 32];
  const uint64_t any = c0 | c1;
  const uint32_t rlo = __reduce_or_sync(kFull, (uint32_t)any);
  const uint32_t rhi = __reduce_or_sync(kFull, (uint32_t)(any >> 32));
  const uint32_t clo = __ballot_sync(kFull, c0 != 0), chi = __ballot_sync(kFull, c1 != 0);
  const uint32_t nfs = __reduce_add_sync(kFull, (uint32_t)(__popcll(c0) + __popcll(c1)));
  if (lane) return;
  m->nfs = nfs;
  int need = max(m->w0, 0);  // an empty region needs no other window
  const uint64_t ra = ((uint64_t)rhi << 32) | rlo, ca = ((uint64_t)chi << 32) | clo;
  TileMap tm = {-1, 1, 1, 0, 0, 0};
  if (h == 0 || w == 0) {
    tm.tile = 0;  // never diffused
  } else {
    const uint32_t bit = d <= 16 ? kLayoutBands : kLayoutWideBands;
    const bool block = h == 2 * d + 1 && w == h && (layouts & bit) && !((ra | ca) & 1ull) &&
                       !((ra | ca) >> (2 * d + 1));
    const bool exact = !block || (layouts & kLayoutRing);
    const int nr = block ? 2 * d : h + 2, nc = block ? 2 * d : w + 2;
#pragma unroll
    for (int k = 0; k < kNumTiles; ++k) {
      const TileShape t = tile_shape(k);
      if (tm.tile < 0 && nr + (t.RE && exact ? 0 : 1) <= 4 * t.R &&
          nc + (t.CE && exact ? 0 : 1) <= 8 * t.C) {
        tm.tile = k;
        tm.C = t.C;
        tm.R = t.R;
        tm.off = block;
        tm.xrow = block && nr == 4 * t.R;
        tm.xcol = block && nc == 8 * t.C;
      }
    }
    // rows r0 - 1 .. r0 + h, one more on each side for cells that divide
    // across the ring before the next ROI
    const int lo = max(m->roi[0] - 2, 0), hi = min(m->roi[0] + h + 1, H - 1);
    if (m->w0 < 0 || lo < m->w0 || hi >= m->w0 + rows)
      need = min(max((lo + hi + 1 - rows) / 2, 0), H - rows);
    if (hi - lo + 1 > rows) tm.tile = -1;
  }
  m->wneed = need;
  m->tm = tm;
  if (tm.tile < 0 || tm.tile >= tiles) m->park = 1;
}

// The slot bits of the region's tile (emt6_tiles.cuh), warp k builds kind k.
template <bool WIDE>
__device__ void build_masks(uint32_t *masks, const uint64_t *colmask, const Misc *m) {
  constexpr int WORDS = WIDE ? kWordsWide : kWordsNarrow;
  const int kind = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (kind > 2) return;
  const int C = m->tm.C, R = m->tm.R, off = m->tm.off, h = m->roi[2], w = m->roi[3];
  const int r0 = (lane >> 3) * R + off, c0 = (lane & 7) * C + off;
  uint32_t bits = 0;
  int q = 0;
  for (int i = 0; i < R; ++i)
    for (int c = 0; c < C; ++c) {
      const int row = r0 + i, col = c0 + c;
      bool on;
      if (kind == kFreeBits) on = col < w + 2 && ((colmask[col] >> row) & 1ull);
      else if (kind == kRoiBits) on = row >= 1 && row <= h && col >= 1 && col <= w;
      else on = row < h + 2 && col < w + 2;
      bits |= (on ? 1u : 0u) << slot_bit(q % 28);
      if (++q % 28 == 0 || q == C * R) {
        masks[(kind * WORDS + (q - 1) / 28) * 32 + lane] = bits;
        bits = 0;
      }
    }
}

// One diffusion step of the region: warp w diffuses field w.  `fld` is the
// window of rows from m->w0.
template <bool WIDE>
__device__ __forceinline__ void diffuse_step(float *fld, int plane, const uint32_t *masks,
                                             float *edge, const Misc *m, const KParams &p) {
  const int h = m->roi[2], w = m->roi[3];
  if (h == 0 || w == 0) return;
  // the broadcast makes the field index warp-uniform for the compiler, so the
  // coefficients come from the constant bank instead of per-lane registers
  const int field = __shfl_sync(kFull, threadIdx.x >> 5, 0);
  const TileMap tm = m->tm;
  const int r0 = m->roi[0] - m->w0, c0 = m->roi[1];
  float *f = fld + field * plane;
  float *e = edge + field * (WIDE ? kEdgeWide : kEdgeNarrow);
  const float ext = p.ext[field], ca = p.da[field], cb = p.db[field], cd = p.dd[field];
#define EMT6_TILE(K)                                                                              \
  case K:                                                                                         \
    diffuse_tile<tile_shape(K).C, tile_shape(K).R, tile_shape(K).RE, tile_shape(K).CE>(           \
        f, masks, WIDE ? kWordsWide : kWordsNarrow, e, tm, r0, c0, w, p.W, ext, ca, cb, cd, p.nfree); \
    break;
#define EMT6_LARGE(K)                                                                             \
  case K:                                                                                         \
    diffuse_large<tile_shape(K).C, tile_shape(K).R, tile_shape(K).RE, tile_shape(K).CE>(          \
        f, masks, kWordsWide, e, &m->tm, r0, c0, w, p.W, ext, ca, cb, cd, p.nfree);               \
    break;
  switch (tm.tile) {
    EMT6_TILE(0) EMT6_TILE(1) EMT6_TILE(2) EMT6_TILE(3) EMT6_TILE(4) EMT6_TILE(5)
    EMT6_TILE(6) EMT6_TILE(7) EMT6_TILE(8) EMT6_TILE(9) EMT6_TILE(10) EMT6_TILE(11)
    default:
      if constexpr (WIDE) {
        switch (tm.tile) {
          EMT6_TILE(12) EMT6_TILE(13) EMT6_TILE(14) EMT6_TILE(15) EMT6_LARGE(16)
          EMT6_LARGE(17) EMT6_LARGE(18) EMT6_LARGE(19) EMT6_LARGE(20)
          default: break;
        }
      }
      break;
  }
#undef EMT6_TILE
#undef EMT6_LARGE
  static_assert(kNumTiles == 21 && kNarrowTiles == 12, "every tile has a case above");
}

// The same of a large region by all 12 warps of the lone tier.
constexpr int kPartTiles = 16;  // from 72 slots per lane on (diffuse_parts)
__device__ __forceinline__ void diffuse_by_parts(float *fld, int plane, const uint64_t *colmask,
                                                 float2 *slots, const Misc *m, const KParams &p) {
  static_assert(kThreadsLone == 384, "four warps per field");
  const int wid = __shfl_sync(kFull, threadIdx.x >> 5, 0), field = wid >> 2, part = wid & 3;
  const int h = m->roi[2], w = m->roi[3], r0 = m->roi[0] - m->w0, c0 = m->roi[1];
  const float ext = p.ext[field], ca = p.da[field], cb = p.db[field], cd = p.dd[field];
  float *f = fld + field * plane;
  slots += field * kPartSlots;
  if (h + 2 <= 4 * 13)
    diffuse_parts<13>(f, colmask, slots, part, 1 + field, r0, c0, h, w, p.W, ext, ca, cb, cd, p.nfree);
  else
    diffuse_parts<14>(f, colmask, slots, part, 1 + field, r0, c0, h, w, p.W, ext, ca, cb, cd, p.nfree);
}

// The class (kRegion*) of a region: what tile_mapping's tiles hold of it.
__host__ __device__ inline int class_of(int h, int w, int d, int H, int W) {
  constexpr TileShape small = tile_shape(kPartTiles - 1), medium = tile_shape(kPartTiles),
                      largest = tile_shape(kNumTiles - 2);
  static_assert(small.RE && !small.CE && !medium.RE && !medium.CE && largest.RE && !largest.CE &&
                    4 * largest.R >= 56 && 8 * largest.C - 1 == kLargestWidth,
                "what the tiles hold");
  const bool block = h == 2 * d + 1 && w == h;
  const bool next = block && h + 2 <= H - 2 && w + 2 <= W - 2;  // a block one site larger, too
  const int nr = block ? 2 * d : h + 2, nc = block ? 2 * d : w + 2;
  const int grown = next ? w + 1 : (w + 2 < W - 2 ? w + 2 : W - 2) + 2;
  if (h > 0 && (nc > kLargestWidth || grown > kLargestWidth)) return kRegionLargest;
  if (nr > 4 * medium.R - 1 || nc > 8 * medium.C - 1) return kRegionLarge;
  return nr > 4 * small.R || nc > 8 * small.C - 1 ? kRegionMedium : kRegionSmall;
}

int region_class(const int32_t roi[5], int H, int W) { return class_of(roi[2], roi[3], roi[4], H, W); }

// Field window (rows w0 .. w0 + rows - 1 of the three planes) from and to
// global memory.  The whole lattice is one contiguous copy of 16-byte words
// (strides are padded); a window's rows start at any 4-byte word.
__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int NT>
__device__ __forceinline__ void load_window(float *fld, const float *g, int w0, int plane, int W,
                                            int HW, uint32_t fstride) {
  if (plane == HW) {
    for (uint32_t q = threadIdx.x; q < fstride / 4; q += NT) cp_async16(fld + 4 * q, g + 4 * q);
  } else {
    for (int k = 0; k < 3; ++k)
      for (int q = threadIdx.x; q < plane; q += NT)
        cp_async4(fld + k * plane + q, g + k * HW + w0 * W + q);
  }
  cp_async_wait();
}

template <int NT>
__device__ __forceinline__ void store_window(const float *fld, float *g, int w0, int plane, int W,
                                             int HW, uint32_t fstride) {
  if (plane == HW) {
    for (uint32_t q = threadIdx.x; q < fstride / 4; q += NT)
      reinterpret_cast<float4 *>(g)[q] = reinterpret_cast<const float4 *>(fld)[q];
  } else {
    for (int k = 0; k < 3; ++k)
      for (int q = threadIdx.x; q < plane; q += NT) g[k * HW + w0 * W + q] = fld[k * plane + q];
  }
}

// ---------------------------------------------------------------------------
// Site::step (site/site.h:62-82) of one cell, from its record in global memory;
// returns ready-to-divide.  The rare parts are functions of their own: their
// exponentials and Philox rounds are ten times the code of the common path.
// ---------------------------------------------------------------------------
// the survival decision of a cell whose repair ended; true if it dies
__device__ __noinline__ bool repair_kills(const KParams &p, Misc *m, float irr, float tir, uint32_t s,
                                          uint32_t t, uint32_t sim, uint32_t occ, uint32_t epoch) {
  DCell c{};
  c.irr = irr;
  const float dp = death_prob(c, p);
  atomicAdd(&m->ins[0], 1u);
  atomicAdd(&m->ins_dp, (double)dp);
  int bi = (int)(irr / 0.1f);
  bi = bi < 0 ? 0 : (bi >= 300 ? 299 : bi);
  int bj = (int)(tir / 0.1f);
  bj = bj < 0 ? 0 : (bj >= 300 ? 299 : bj);
  atomicAdd(&g_instr_hist[bi], 1ull);
  atomicAdd(&g_instr_hist[300 + bj], 1ull);
  const float u = u01(draw(p, t, sim, s, occ, 1, epoch).x);
  if (u < dp) atomicAdd(&m->ins[1], 1u);
  return u < dp;
}

__device__ __noinline__ bool step_site(const KParams &p, float *lv, int plane, uint8_t *st,
                                       float4 *rec, int s, uint32_t vac, float dose, uint32_t t,
                                       uint32_t sim, uint32_t occ, uint32_t epoch, Misc *m,
                                       bool *died) {
  DCell c = load_cell(rec);
  const uint32_t mp0 = c.mode | (c.phase << 8);
  const float l0 = lv[0], l1 = lv[plane], l2 = lv[2 * plane];
  *died = true;
  if (!update_state(c, l0, l1, l2, p, vac)) {
    *st = (*st & ~kStMask) | kVacant;
    return false;
  }
  if (dose > 0) {
    irradiate(c, dose, p);
    atomicAdd(&m->ins[2], 1u);
  }
  lv[0] = l0 - met_of(p, c.mode, 0);
  lv[plane] = l1 - met_of(p, c.mode, 1);
  lv[2 * plane] = l2 - met_of(p, c.mode, 2);
  const bool cc = progress_clock(c, p);
  bool dead = false;
  if (repair_pre(c, p, cc)) {
    dead = repair_kills(p, m, c.irr, c.tir, (uint32_t)s, t, sim, occ, epoch);
    if (!dead) {
      c.irr = 0.f;
      c.tir = 0.f;
      c.delay = 0.f;
    }
  }
  // the cycle times (t0..t4) never change here: store the clocks and, when
  // they changed, mode and phase (same memory contents as a full store)
  rec[0] = make_float4(c.prolif, c.tir, c.irr, c.delay);
  const uint32_t mp = c.mode | (c.phase << 8);
  if (mp != mp0) reinterpret_cast<uint32_t *>(rec + 2)[1] = mp;
  if (dead) *st = (*st & ~kStMask) | kVacant;
  *died = dead;
  return !dead && c.phase == 4;
}

// ---------------------------------------------------------------------------
// Hot entries.  Between two list rebuilds, what a step needs of a listed cell
// is on chip, by list entry: its running clock h0, the threshold h1 of that
// clock's next event, and a flag word fl.  The 48-byte record in global memory
// is loaded (a scattered access of about 900 cycles, L2) only for events: a
// phase change, the end of a repair, a dose, a death, a division.
//   fl: mode (2 bits) | class << 2 | kT | kG | kOld
//   class 0-4: the cell's phase.  Its clock is the proliferation time, or,
//     with kT, the time in repair (the proliferation time then stands still).
//     h1: the smaller of the phase's end and the age limit t4 - dt (kOld:
//     reached, the cell dies in the next step); with kT the repair delay.
//     kG (with kT): the G1/S check's clock condition.
//   kSlow: any other record (stepped from global memory)
//   kGone: no cell, or a site listed more than once (stepped in list order)
// Entries of class kSlow and kGone have, in h0's place, kReady | occurrence of
// a cell that is ready to divide, or 0.
// ---------------------------------------------------------------------------
constexpr uint32_t kT = 32u, kG = 64u, kOld = 128u, kReady = 0x100u;
constexpr uint32_t kClass = 7u << 2, kSlow = 6u << 2, kGone = 7u << 2;

struct Hot {
  float *h0, *h1;
  uint8_t *fl;
  float4 *cells;  // the simulation's records
  uint32_t held;  // entries from here on have their clocks in the records' padding
  __device__ __forceinline__ float2 *spill(uint32_t e) const {
    return reinterpret_cast<float2 *>(cells + 3 * e + 2) + 1;
  }
  __device__ __forceinline__ float clock(uint32_t e) const { return e < held ? h0[e] : spill(e)->x; }
  __device__ __forceinline__ void set(uint32_t e, float clk, float thr) const {
    if (e < held) {
      h0[e] = clk;
      h1[e] = thr;
    } else {
      *spill(e) = make_float2(clk, thr);
    }
  }
  __device__ __forceinline__ void idle(uint32_t e, uint32_t cls, uint32_t ready) const {
    fl[e] = (uint8_t)cls;
    set(e, __uint_as_float(ready), 0.f);
  }
  // kReady | occurrence of a cell that is ready to divide, else 0
  __device__ __forceinline__ uint32_t ready(uint32_t e) const {
    const uint32_t cls = fl[e] & kClass;
    return cls < kSlow ? (cls == 16u ? kReady : 0u) : __float_as_uint(clock(e));
  }
};

__device__ __forceinline__ void classify(const KParams &p, const DCell &c, const Hot &h, uint32_t e) {
  const float tc = c.phase == 0 ? c.t0 : c.phase == 1 ? c.t1 : c.phase == 2 ? c.t2 : c.phase == 3 ? c.t3 : c.t4;
  const float lim = c.t4 - p.dt_h;
  const bool old = c.prolif >= lim;
  uint32_t f = kSlow;
  float h0 = 0.f, h1 = 0.f;
  if (c.mode <= 3 && c.phase <= 4) {
    if (c.tir == 0) {
      // (the G1/S check reads the end of phase 0 itself)
      if (c.phase != 0 || tc <= lim) {
        f = c.mode | (c.phase << 2) | (old ? kOld : 0u);
        h0 = c.prolif;
        h1 = fminf(tc, lim);
      }
    } else if (!old) {
      f = c.mode | (c.phase << 2) | kT | (c.prolif > c.t0 - p.dt2_h ? kG : 0u);
      h0 = c.tir;
      h1 = c.delay;
    }
  }
  h.set(e, h0, h1);
  h.fl[e] = (uint8_t)f;
}

// the cell of a hot entry, its clock and flags merged into the global record
__device__ __forceinline__ DCell merged_cell(const float4 *rec, const Hot &h, uint32_t e) {
  DCell c = load_cell(rec);
  const uint32_t f = h.fl[e];
  if ((f & kClass) < kSlow) {
    (f & kT ? c.tir : c.prolif) = h.clock(e);
    c.mode = f & 3u;
    c.phase = (f & kClass) >> 2;
  }
  return c;
}

// clocks, mode and phase of a cell (the cycle times never change)
__device__ __forceinline__ void store_clocks(float4 *rec, const DCell &c) {
  rec[0] = make_float4(c.prolif, c.tir, c.irr, c.delay);
  reinterpret_cast<uint32_t *>(rec + 2)[1] = c.mode | (c.phase << 8);
}

// a new cell's record; the padding may hold an entry's clocks
__device__ __forceinline__ void store_fresh(float4 *rec, const DCell &c) {
  store_clocks(rec, c);
  rec[1] = make_float4(c.t0, c.t1, c.t2, c.t3);
  reinterpret_cast<float *>(rec + 2)[0] = c.t4;
}

template <int NT>
__device__ __noinline__ void gather_cells(const KParams &p, const uint8_t *st, const uint16_t *list,
                                          const float4 *cells, const Hot h, uint32_t n) {
  // four entries of a thread at a time, so their records' loads overlap
  constexpr int U = 4;
  for (uint32_t e0 = threadIdx.x; e0 < n; e0 += NT * U) {
    DCell c[U];
    bool on[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t e = min(e0 + u * NT, n - 1);
      const int s = list[e] & kSiteMask;
      on[u] = (st[s] & (kStMask | kStMulti)) == kOccupied;
      c[u] = load_cell(cells + 3 * s);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t e = e0 + u * NT;
      if (e >= n) break;
      if (on[u]) classify(p, c[u], h, e);
      else h.idle(e, kGone, 0);
    }
  }
}

template <int NT>
__device__ __noinline__ void scatter_cells(const uint16_t *list, float4 *cells, const Hot h, uint32_t n) {
  for (uint32_t e = threadIdx.x; e < n; e += NT) {
    const uint32_t f = h.fl[e];
    if ((f & kClass) >= kSlow) continue;
    float *rec = reinterpret_cast<float *>(cells + 3 * (list[e] & kSiteMask));
    rec[f & kT ? 1 : 0] = h.clock(e);
    reinterpret_cast<uint32_t *>(rec)[9] = (f & 3u) | ((f & kClass) << 6);
  }
}

// An event of hot entry e (levels and running clock already advanced): the
// cell dies of its levels or age (!alive), its repair ends (kT), or its clock
// reached the threshold.  Returns whether the cell died.
__device__ __noinline__ bool cell_event(const KParams &p, Misc *m, float4 *rec, uint8_t *st,
                                        const Hot h, uint32_t e, bool alive, int s, uint32_t t,
                                        uint32_t sim, uint32_t epoch) {
  DCell c = merged_cell(rec, h, e);
  bool dead = !alive;
  if (alive) {
    bool decide = (h.fl[e] & kT) != 0;
    if (!decide) {
      const uint32_t cur = c.phase;
      const float tc = cur == 0 ? c.t0 : cur == 1 ? c.t1 : cur == 2 ? c.t2 : cur == 3 ? c.t3 : c.t4;
      const bool next = c.prolif > tc;
      c.phase = cur + (next ? 1u : 0u);
      decide = repair_pre(c, p, next & (c.phase != 4));
    }
    if (decide) {
      dead = repair_kills(p, m, c.irr, c.tir, (uint32_t)s, t, sim, 0, epoch);
      if (!dead) c.irr = c.tir = c.delay = 0.f;
    }
  }
  store_clocks(rec, c);
  if (dead) {
    *st = (*st & ~kStMask) | kVacant;
    h.idle(e, kGone, 0);
  } else {
    classify(p, c, h, e);
    if (c.phase == 4 && h.fl[e] == kSlow) h.idle(e, kSlow, kReady);
  }
  return dead;
}

// Entry e stepped from its global record: class kSlow, and every entry of a
// step with a dose.  Returns bit 0: ready to divide, bit 1: died.
__device__ __noinline__ uint32_t step_entry(const KParams &p, Misc *m, float *lv, int plane,
                                            float4 *rec, uint8_t *st, const Hot h, uint32_t e, int s,
                                            uint32_t vac, float dose, uint32_t t, uint32_t sim,
                                            uint32_t epoch) {
  if ((h.fl[e] & kClass) < kSlow) store_clocks(rec, merged_cell(rec, h, e));
  bool died;
  const bool ready = step_site(p, lv, plane, st, rec, s, vac, dose, t, sim, 0, epoch, m, &died);
  if (died) {
    h.idle(e, kGone, 0);
    return 2u;
  }
  classify(p, load_cell(rec), h, e);
  if (ready && h.fl[e] == kSlow) h.idle(e, kSlow, kReady);
  return ready ? 1u : 0u;
}

// occurrence index of list entry e of a multi-listed site (entries before e
// with the same site): 0 in the rebuilt part, else rebuilt-bit + tail count.
__device__ __forceinline__ uint32_t occurrence(const uint16_t *list, const uint8_t *st, uint32_t e,
                                               uint32_t n0) {
  const int lane = threadIdx.x & 31;
  const uint32_t s = list[e] & kSiteMask;
  if (e < n0) return 0;
  uint32_t k = (st[s] & kStRebuilt) ? 1u : 0u;
  for (uint32_t b = n0; b < e; b += 32) {
    const uint32_t q = b + lane;
    k += __popc(__ballot_sync(kFull, q < e && (list[q] & kSiteMask) == s));
  }
  return k;
}

// diffused site-substeps of `steps` steps with the current ROI: free sites x free
// substeps + the final ROI pass
__device__ __forceinline__ void count_diffused(Misc *m, const KParams &p, uint32_t steps) {
  if (m->roi[2] > 0)
    m->diffused += steps * (m->nfs * (unsigned long long)p.nfree +
                            (unsigned long long)m->roi[2] * (unsigned long long)m->roi[3]);
}

// ---------------------------------------------------------------------------
// the fused step kernel
// ---------------------------------------------------------------------------
// kTierNarrow: regions that fit a tile of at most 32 slots per lane (discs up
// to distance 16, clipped regions up to 32 x 32), 5 CTAs/SM.  A simulation it
// cannot hold (region, window or list) is parked at the start of that step for
// kTierWide: any simulation, 4 CTAs/SM.  kTierLone: any simulation, one CTA of 384
// threads per SM, for batches that leave SMs idle otherwise, and for regions that
// the wide tier is slower on (emt6_batch::prepare_launch): a step's latency instead
// of the SM's throughput (one disc of radius 10, 300 steps: 1.39 vs 1.46 ms with the
// other tiers side by side, 100 of them 1.41 vs 1.47; 152 of radius 24, 200 steps:
// 3.01 vs 5.92).
template <int TIER>
__global__ void __launch_bounds__(threads_of(TIER), TIER == kTierLone ? 1 : TIER == kTierWide ? 4 : 5)
    run_kernel(const __grid_constant__ RunArgs a, uint32_t t_end) {
  constexpr int NT = threads_of(TIER);
  constexpr bool WIDE = TIER != kTierNarrow;
  extern __shared__ __align__(16) uint8_t sm[];
  const KParams &p = a.p;
  const int H = p.H, W = p.W, HW = p.HW;
  const SmemLayout L = smem_layout(H, W, p.lcap, TIER);
  float *fld = reinterpret_cast<float *>(sm + L.fld);
  uint8_t *st = sm + L.st;
  uint16_t *list = reinterpret_cast<uint16_t *>(sm + L.list);
  Hot hot = {reinterpret_cast<float *>(sm + L.h0), reinterpret_cast<float *>(sm + L.h1), sm + L.fl,
             nullptr, (uint32_t)L.held};
  uint64_t *colmask = reinterpret_cast<uint64_t *>(sm + L.colmask);
  uint32_t *masks = reinterpret_cast<uint32_t *>(sm + L.masks);
  float *edge = reinterpret_cast<float *>(sm + L.edge);
  Misc *m = reinterpret_cast<Misc *>(sm + L.misc);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int plane = L.plane, rows = L.rows, tiles = WIDE ? kNumTiles : kNarrowTiles;

  if (tid < 4) m->met[tid] = make_float4(p.met[tid][0], p.met[tid][1], p.met[tid][2], 0.f);
  for (int64_t item = blockIdx.x;; item += gridDim.x) {
    int64_t sim;
    if (a.queue) {
      // persistent CTAs: take the next simulation from the work queue
      __syncthreads();
      if (tid == 0) m->winner = (int)atomicAdd(a.ticket, 1u);
      __syncthreads();
      const int64_t ticket = m->winner;
      if (ticket >= a.nsims) break;
      sim = a.order[ticket];
    } else {
      if (item >= a.nsims) break;
      sim = a.order ? a.order[item] : item;
    }
    if (a.tier_of && a.tier_of[sim] != TIER) continue;  // another concurrent launch's
    const uint32_t horizon = a.horizon ? a.horizon[sim] : 0xFFFFFFFFu;
    const uint32_t t_stop = t_end < horizon ? t_end : horizon;
    const uint32_t step0 = a.step[sim];
    // nothing to do for a simulation already at its target step
    if (step0 >= t_stop) continue;
    const int4 meta = a.meta[sim];
    if (!WIDE && meta.x >= L.entries) continue;  // the list does not fit: the wide tier's

    // ---- load the simulation into shared memory (its fields when the window
    //      is known) ----
    float *gfld = a.fld + sim * a.fstride;
    const uint4 *gs = reinterpret_cast<const uint4 *>(a.st + sim * a.sstride);
    for (uint32_t q = tid; q < a.sstride / 16; q += NT) cp_async16(st + 16 * q, gs + q);
    const uint16_t *gl = a.list + sim * a.lstride;
    for (int q = tid; q < meta.x; q += NT) list[q] = gl[q];
    if (tid == 0) {
      m->n = (uint32_t)meta.x;
      m->n0 = (uint32_t)meta.y;
      m->has_multi = meta.z;
      m->edge = meta.w;
      for (int k = 0; k < 5; ++k) m->roi[k] = a.roi[sim * 8 + k];
      m->ins[0] = m->ins[1] = m->ins[2] = m->ins[3] = 0;
      m->ins_dp = 0.0;
      m->diffused = 0;
      m->park = 0;
      m->w0 = -1;
    }
    cp_async_wait();
    float4 *cells = a.cell + sim * (int64_t)HW * 3;
    hot.cells = cells;
    const int32_t prot = a.sim_protocol[sim];
    const float *doses = a.doses + (int64_t)prot * p.bins;
    __syncthreads();

    uint32_t t = step0;
    bool dirty = true;    // site states changed since the last vacancy snapshot
    bool onchip = false;  // the hot entries hold the cells' clocks
    uint32_t bin = t / p.res, in_bin = t % p.res;  // dose bin of step t, steps into it
    uint32_t since = t;   // steps before it are in m->diffused
    for (; t < t_stop; ++t) {
      if (t % 128 == 0) {
        if (onchip) scatter_cells<NT>(list, cells, hot, m->n);
        onchip = false;
        __syncthreads();
        rebuild_list<NT>(st, list, m, H, W, HW, L.entries);
        dirty = true;
      }
      if (t % 32 == 0 || t == step0) {
        if (tid == 0) count_diffused(m, p, t - since);
        since = t;
        if (t % 32 == 0) {
          compute_roi<NT>(st, list, colmask, m, H, W);
        } else {
          // launch start between ROI updates: the mask of the stored ROI
          build_colmask(colmask, m->roi[2], m->roi[3], m->roi[4]);
          __syncthreads();
        }
        if (wid == 0) tile_mapping(colmask, m, p.layouts, tiles, H, rows);
        __syncthreads();
        if (WIDE || !m->park) build_masks<WIDE>(masks, colmask, m);
        const int w0 = m->w0, need = m->wneed;
        if (w0 != need) {
          // (another) window of the fields; a parked simulation needs none
          if (w0 >= 0) store_window<NT>(fld, gfld, w0, plane, W, HW, a.fstride);
          __syncthreads();
          if (WIDE || !m->park) {
            load_window<NT>(fld, gfld, need, plane, W, HW, a.fstride);
            if (tid == 0) m->w0 = need;
          } else if (tid == 0) {
            m->w0 = -1;
          }
        }
        __syncthreads();
      }
      if (!WIDE && t == step0 && t % 32 != 0) {
        // between ROI updates cells may lie beyond the ROI, and beyond the
        // window chosen for it
        const int fo = m->w0 * W;
        for (uint32_t e = tid; e < m->n; e += NT) {
          const int s = list[e] & kSiteMask;
          if ((st[s] & kStMask) == kOccupied && (s < fo || s >= fo + plane)) m->park = 1;
        }
        __syncthreads();
      }
      // a simulation the narrow tier cannot hold is left for the wide one; the
      // state stored is the state at the start of step t (the list rebuild and
      // ROI above are recomputed identically there)
      if (!WIDE && (m->park || m->n >= (uint32_t)L.entries)) break;
      const uint32_t n = m->n;
      const int fo = m->w0 * W;
      if (!onchip) gather_cells<NT>(p, st, list, cells, hot, n);
      onchip = true;
      // vacancy snapshot (simulation.cu:79-83), before any site changes: kept
      // from the last step unless a site state or the list changed there
      if (dirty)
        for (uint32_t e = tid; e < n; e += NT) {
          const int s = list[e] & kSiteMask;
          const uint32_t vac =
              ((st[s - W - 1] & kStMask) == kVacant) + ((st[s - W + 1] & kStMask) == kVacant) +
              ((st[s + W - 1] & kStMask) == kVacant) + ((st[s + W + 1] & kStMask) == kVacant) +
              ((st[s - 1] & kStMask) == kVacant) + ((st[s + 1] & kStMask) == kVacant) +
              ((st[s - W] & kStMask) == kVacant) + ((st[s + W] & kStMask) == kVacant);
          list[e] = (uint16_t)(s | (vac << kSiteBits));
        }
      dirty = false;
      if (TIER == kTierLone && m->tm.tile >= kPartTiles)
        diffuse_by_parts(fld, plane, colmask, reinterpret_cast<float2 *>(sm + L.parts), m, p);
      else if (NT == kThreads || wid < 3)
        diffuse_step<WIDE>(fld, plane, masks, edge, m, p);
      __syncthreads();

      // ---- cell update (simulation.cu:84-96) ----
      // may_divide: some cell is ready and may find a vacant neighbour.  A
      // ready cell whose 8 neighbours were all taken at the vacancy snapshot
      // can only find one if a neighbour dies in this step (divisions fill
      // sites only after the arbitration), so the arbitration runs only when
      // a ready cell had a vacant neighbour or some cell died.
      bool may_divide = false;
      const float dose = (in_bin == 0 && t < p.length && bin < p.bins) ? doses[bin] : 0.f;
      if (++in_bin == p.res) {
        in_bin = 0;
        ++bin;
      }
      {
        // A thread steps the entries it gathered: no other thread touches them
        // before the barrier below.  The loop is what the kernel issues most
        // outside the substeps, so conditions are combined without branches and
        // a mode's consumption comes from a table on chip.
        float2 ahead = make_float2(0.f, 0.f);  // clocks of the next entry, if not on chip
        for (uint32_t e = tid; e < n; e += NT) {
          float clk = ahead.x, thr = ahead.y;
          const bool here = !WIDE || e < hot.held;
          if (here) {
            clk = hot.h0[e];
            thr = hot.h1[e];
          }
          if (WIDE && e + NT >= hot.held && e + NT < n) ahead = *hot.spill(e + NT);
          const uint32_t f = hot.fl[e], cls = f & kClass, le = list[e];
          const int s = le & kSiteMask;
          float *lv = fld + (s - fo);  // the site in the field window
          if (cls >= kSlow || dose > 0) {
            if (cls == kGone) continue;
            const uint32_t r = step_entry(p, m, lv, plane, cells + 3 * s, st + s, hot, e, s,
                                          le >> kSiteBits, dose, t, (uint32_t)sim, a.epoch);
            may_divide |= ((r & 1u) && (le >> kSiteBits) != 0) || (r & 2u);
            continue;
          }
          const float l0 = lv[0], l1 = lv[plane], l2 = lv[2 * plane];
          // update_state, progress_clock and repair_pre (emt6_device.cuh)
          const bool rep = (f & kT) != 0;
          const bool late = rep ? (f & kG) != 0 : clk > thr - p.dt2_h;
          const bool g1s = late & (cls == 0) & (le < (2u << kSiteBits));
          const bool q = (l2 < p.quiescence_gi) & !g1s;
          const bool d = (l2 < p.death_gi) & ((cls & (4u | 16u)) == 0);  // phases G1, G2 only
          const bool a0 = (l0 >= p.met[0][0]) & (l1 >= p.met[0][1]) & q;
          const bool a1 = (l0 >= p.met[1][0]) & (l1 >= p.met[1][1]) & q;
          const bool a2 = (l0 >= p.met[2][0]) & (l1 >= p.met[2][1]) & d;
          const bool a3 = (l0 >= p.met[3][0]) & (l1 >= p.met[3][1]) & d;
          const bool grows = a0 | a1, alive = (grows | a2 | a3) & !(f & kOld);
          const uint32_t mode = grows ? (a0 ? 0u : 1u) : (a2 ? 2u : 3u);
          const float4 use = m->met[mode];
          const float next = clk + p.dt_h;
          const bool moves = rep ? clk > 0 : grows;
          if (alive) {
            lv[0] = l0 - use.x;
            lv[plane] = l1 - use.y;
            lv[2 * plane] = l2 - use.z;
            hot.fl[e] = (uint8_t)((f & ~3u) | mode);
            if (moves) *(here ? hot.h0 + e : &hot.spill(e)->x) = next;
          }
          bool ready = alive & (cls == 16);
          if (!alive | (moves & (next >= thr))) {
            const bool died = cell_event(p, m, cells + 3 * s, st + s, hot, e, alive, s, t,
                                         (uint32_t)sim, a.epoch);
            ready = hot.ready(e) != 0;
            may_divide |= died;
          }
          may_divide |= ready & (le >= (1u << kSiteBits));
        }
      }
      if (m->has_multi && wid == 0) {
        // sites listed more than once: every entry steps the site, in list order
        const uint32_t n0 = m->n0;
        for (uint32_t b = 0; b < n; b += 32) {
          const uint32_t e = b + lane;
          const bool mult = e < n && (st[list[e] & kSiteMask] & kStMulti);
          uint32_t bal = __ballot_sync(kFull, mult);
          while (bal) {
            const int bit = __ffs(bal) - 1;
            bal &= bal - 1;
            const uint32_t ee = b + bit;
            const uint32_t occ = occurrence(list, st, ee, n0);
            if (lane == 0) {
              const int s = list[ee] & kSiteMask;
              uint32_t res = 0;
              if ((st[s] & kStMask) == kOccupied) {
                const uint32_t vac = list[ee] >> kSiteBits;
                bool died;
                const bool ready = step_site(p, fld + (s - fo), plane, st + s, cells + 3 * s, s, vac,
                                             dose, t, (uint32_t)sim, occ, a.epoch, m, &died);
                if (ready) {
                  if (occ > 127) atomicOr(a.err, 4u);
                  res = kReady | (occ & 0x7fu);
                }
                may_divide |= (ready & (vac != 0)) | died;
              }
              hot.idle(ee, kGone, res);
            }
            __syncwarp();
          }
        }
      }
      // most steps have no cell that may divide: skip the arbitration then
      if (!__syncthreads_or(may_divide)) continue;
      dirty = true;  // a death or division is possible only here

      // ---- division arbitration: lowest list index with a vacant target ----
      int best = 0x7fffffff, best_target = -1;
      for (uint32_t e = tid; e < n; e += NT) {
        const uint32_t ready = hot.ready(e);
        if (ready) {
          const int s = list[e] & kSiteMask;
          // a cell none of whose neighbours is vacant now cannot divide,
          // whatever the draw: skip the draw (interior cells stay ready)
          const bool open = ((st[s - W - 1] & kStMask) == kVacant) |
                            ((st[s - W] & kStMask) == kVacant) |
                            ((st[s - W + 1] & kStMask) == kVacant) |
                            ((st[s - 1] & kStMask) == kVacant) |
                            ((st[s + 1] & kStMask) == kVacant) |
                            ((st[s + W - 1] & kStMask) == kVacant) |
                            ((st[s + W] & kStMask) == kVacant) |
                            ((st[s + W + 1] & kStMask) == kVacant);
          if (!open) continue;
          const float u = u01(draw(p, t, (uint32_t)sim, (uint32_t)s, ready & 0x7fu, 0, a.epoch).x);
          const int tg = choose_neighbour(s, W, u);
          if ((st[tg] & kStMask) == kVacant) {
            best = (int)e;
            best_target = tg;
            break;
          }
        }
      }
      const int win = block_min<NT>(best, m);
      if (win != 0x7fffffff && best == win) {
        m->winner = win;
        m->target = best_target;
      }
      __syncthreads();
      if (win != 0x7fffffff && wid == 0) {
        // divideCell (cell-division.h:10-30) with five Philox normals; lanes
        // 0..2 each evaluate one Box-Muller pair
        float za = 0.f, zb = 0.f;
        if (lane < 3) {
          const uint4 r = draw(p, t, (uint32_t)sim, 0xFFFFu, 0, lane == 2 ? 3 : 2, a.epoch);
          if (lane == 0) box_muller(r.x, r.y, &za, &zb);
          else if (lane == 1) box_muller(r.z, r.w, &za, &zb);
          else box_muller(r.x, r.y, &za, &zb);
        }
        float z[5];
        z[0] = __shfl_sync(kFull, za, 0);
        z[1] = __shfl_sync(kFull, zb, 0);
        z[2] = __shfl_sync(kFull, za, 1);
        z[3] = __shfl_sync(kFull, zb, 1);
        z[4] = __shfl_sync(kFull, za, 2);
        if (lane == 0) {
          const uint32_t pe = (uint32_t)m->winner;
          const int parent = list[pe] & kSiteMask, child = m->target;
          DCell pc = merged_cell(cells + 3 * parent, hot, pe);
          pc.phase = 0;
          pc.prolif = 0.f;
          store_clocks(cells + 3 * parent, pc);
          if ((hot.fl[pe] & kClass) != kGone) classify(p, pc, hot, pe);
          const DCell cc = make_child(pc, z, p);
          store_fresh(cells + 3 * child, cc);
          const uint8_t sv = st[child];
          const bool listed = (sv & (kStRebuilt | kStTail)) != 0;
          st[child] = (uint8_t)((sv & (kStRebuilt | kStTail | kStMulti)) | kStTail |
                                (listed ? kStMulti : 0) | kOccupied);
          if (listed) m->has_multi = 1;
          if (child >= HW - W || child % W == W - 1) m->edge = 1;
          // the narrow kernel's window moves with the ROI only: a child beyond
          // it is the wide kernel's
          if (!WIDE && (child < fo || child >= fo + plane)) m->park = 1;
          if (m->n < (uint32_t)L.entries) {
            const uint32_t ce = m->n++;
            list[ce] = (uint16_t)child;
            if (listed) hot.idle(ce, kGone, 0);
            else classify(p, cc, hot, ce);
          } else {
            atomicOr(a.err, 1u);
          }
          m->ins[3] += 1;
        }
      }
      __syncthreads();
    }

    // ---- write the simulation back (nothing changed when the first step parks) ----
    if (!WIDE && t == step0) {
      __syncthreads();
      continue;
    }
    if (tid == 0) count_diffused(m, p, t - since);
    if (onchip) scatter_cells<NT>(list, cells, hot, m->n);
    if (m->w0 >= 0) store_window<NT>(fld, gfld, m->w0, plane, W, HW, a.fstride);
    uint4 *os = reinterpret_cast<uint4 *>(a.st + sim * a.sstride);
    for (uint32_t q = tid; q < a.sstride / 16; q += NT)
      os[q] = reinterpret_cast<const uint4 *>(st)[q];
    uint16_t *ol = a.list + sim * a.lstride;
    for (uint32_t q = tid; q < m->n; q += NT) ol[q] = list[q] & kSiteMask;
    int live = 0;
    for (int q = tid; q < HW; q += NT) live += (st[q] & kStMask) == kOccupied;
#pragma unroll
    for (int o = 16; o; o >>= 1) live += __shfl_xor_sync(kFull, live, o);
    __syncthreads();
    if (lane == 0) m->red()[wid][1] = live;
    __syncthreads();
    if (tid == 0) {
      int tot = 0;
      for (int w2 = 0; w2 < NT / 32; ++w2) tot += m->red()[w2][1];
      a.counts[sim] = (uint32_t)tot;
      a.meta[sim] = make_int4((int)m->n, (int)m->n0, m->has_multi, m->edge);
      for (int k2 = 0; k2 < 5; ++k2) a.roi[sim * 8 + k2] = m->roi[k2];
      a.step[sim] = t;
      if (WIDE && a.seen) {
        const int c = class_of(m->roi[2], m->roi[3], m->roi[4], H, W);
        if (c != kRegionSmall) a.seen[c] = 1;
      }
      if (m->ins[0]) atomicAdd(&g_instr_counts[0], (unsigned long long)m->ins[0]);
      if (m->ins[1]) atomicAdd(&g_instr_counts[1], (unsigned long long)m->ins[1]);
      if (m->ins[2]) atomicAdd(&g_instr_counts[2], (unsigned long long)m->ins[2]);
      if (m->ins[3]) atomicAdd(&g_instr_counts[3], (unsigned long long)m->ins[3]);
      if (m->ins_dp != 0.0) atomicAdd(&g_instr_sum_death_prob, m->ins_dp);
      if (m->diffused) atomicAdd(a.diffused, m->diffused);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// launch order: simulations sorted by the region their next step diffuses
// (largest first), so the CTAs resident on an SM at once mostly run the same
// diffusion tile code and take similar times.  A counting sort over the
// region's (rows, columns) key: count, exclusive scan, scatter.  The order
// inside a key is whatever the atomics give; results do not depend on it
// (every draw is keyed by the simulation, not by the CTA).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t order_key(const RunArgs &a, int64_t sim, uint32_t t_end) {
  const uint32_t hz = a.horizon ? a.horizon[sim] : 0xFFFFFFFFu;
  if (a.step[sim] >= (t_end < hz ? t_end : hz)) return kOrderKeys - 1;  // nothing to do: last
  const int h = a.roi[sim * 8 + 2], w = a.roi[sim * 8 + 3];
  // regions are at most 56 x 62 (lattice limit); the clamps keep any key in
  // [0, kOrderKeys - 2] whatever the stored ROI holds
  const uint32_t nr = (uint32_t)min(max(h + 2, 0), 62), nc = (uint32_t)min(max(w + 2, 0), 63);
  return (kOrderKeys - 2) - (nr * 64u + nc);
}

__global__ void order_count_kernel(const RunArgs a, uint32_t t_end, uint32_t *hist) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.nsims;
       i += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(&hist[order_key(a, i, t_end)], 1u);
}

static_assert(kOrderKeys == 4 * 1024, "order_scan_kernel scans four counters per thread");

__global__ void __launch_bounds__(1024) order_scan_kernel(uint32_t *hist) {
  // kOrderKeys = 4 x 1024 counters: each thread scans four, then the block
  __shared__ uint32_t part[1024];
  const int t = threadIdx.x;
  uint32_t v[4], run = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = run;
    run += hist[4 * t + k];
  }
  part[t] = run;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const uint32_t add = t >= o ? part[t - o] : 0u;
    __syncthreads();
    part[t] += add;
    __syncthreads();
  }
  const uint32_t base = part[t] - run;
#pragma unroll
  for (int k = 0; k < 4; ++k) hist[4 * t + k] = base + v[k];
}

// The tier expected to hold a simulation, from its stored region and list
// (or, until its first step, its tumour's cells): a wrong guess only costs time, the launch
// after the concurrent ones takes what they leave.  A region at the narrow
// tiles' limit is given to the wide tier, which runs it nearly as fast: it may
// grow in the next steps, and what is left for the last launch runs alone.  Regions
// from class `lone` on (unless 0) go to the lone tier.
__device__ __forceinline__ uint8_t expected_tier(const RunArgs &a, int64_t sim, int lone) {
  const int *roi = a.roi + sim * 8;
  const int h = roi[2], w = roi[3], d = roi[4];
  const int n = (a.step[sim] == 0 ? roi[5] : a.meta[sim].x) + 64;
  const bool small = (h == 2 * d + 1 && w == h) ? d <= 15 : h + 2 <= 30 && w + 2 <= 30;
  if (lone && class_of(h, w, d, a.p.H, a.p.W) >= lone) return kTierLone;
  if (small && n < smem_layout(a.p.H, a.p.W, a.p.lcap, kTierNarrow).entries)
    return kTierNarrow;
  return kTierWide;
}

__global__ void order_scatter_kernel(const RunArgs a, uint32_t t_end, uint32_t *hist,
                                     int64_t *out, uint8_t *tier, int lone) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.nsims;
       i += (int64_t)gridDim.x * blockDim.x) {
    out[atomicAdd(&hist[order_key(a, i, t_end)], 1u)] = i;
    if (tier) tier[i] = expected_tier(a, i, lone);
  }
}

// Tiers of a batch that is resident at once, by one block.  The lone tier takes whole
// SMs, and the wide one would crowd on what is left of them; where its simulations
// would be more than two to an SM there (`sms` SMs, 0: no such rule), they go to the
// lone tier, too (260 discs of radius 22 to 24, 300 steps: 9.0 ms, 10.3 on the wide tier
// alone; crowded they took 12.1).
constexpr int kTierThreads = 1024;
__global__ void __launch_bounds__(kTierThreads) tier_kernel(const RunArgs a, uint8_t *tier, int lone,
                                                            bool narrow, int sms) {
  __shared__ int count[kTiers];
  if (threadIdx.x < kTiers) count[threadIdx.x] = 0;
  __syncthreads();
  if (lone && sms)
    for (int64_t i = threadIdx.x; i < a.nsims; i += kTierThreads)
      atomicAdd(&count[expected_tier(a, i, lone)], 1);
  __syncthreads();
  const bool crowded = count[kTierWide] > 2 * max(sms - count[kTierLone], 0);
  for (int64_t i = threadIdx.x; i < a.nsims; i += kTierThreads) {
    uint8_t t = expected_tier(a, i, lone);
    if (t == kTierWide && crowded) t = kTierLone;
    tier[i] = t == kTierNarrow && !narrow ? (uint8_t)kTierWide : t;
  }
}

// ---------------------------------------------------------------------------
// reset: expand the initial tumours into every simulation
// ---------------------------------------------------------------------------
__global__ void reset_kernel(const ResetArgs a) {
  for (int64_t sim = blockIdx.x; sim < a.nsims; sim += gridDim.x) {
    const int t = a.sim_tumor[sim];
    const float4 *sf = reinterpret_cast<const float4 *>(a.tpl_fld + (int64_t)t * a.fstride);
    float4 *df = reinterpret_cast<float4 *>(a.fld + sim * a.fstride);
    for (uint32_t q = threadIdx.x; q < a.fstride / 4; q += blockDim.x) df[q] = sf[q];
    const uint4 *ss = reinterpret_cast<const uint4 *>(a.tpl_st + (int64_t)t * a.sstride);
    uint4 *ds = reinterpret_cast<uint4 *>(a.st + sim * a.sstride);
    for (uint32_t q = threadIdx.x; q < a.sstride / 16; q += blockDim.x) ds[q] = ss[q];
    const float4 *sc = a.tpl_cell + (int64_t)t * a.HW * 3;
    float4 *dc = a.cell + sim * (int64_t)a.HW * 3;
    for (int q = threadIdx.x; q < a.HW * 3; q += blockDim.x) dc[q] = sc[q];
    if (threadIdx.x == 0) {
      a.meta[sim] = make_int4(0, 0, 0, 0);
      for (int k = 0; k < 8; ++k) a.roi[sim * 8 + k] = a.tpl_roi[t * 8 + k];
      a.step[sim] = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// unit hooks: run the device functions above on caller-provided inputs
// ---------------------------------------------------------------------------
__global__ void test_philox_kernel(const uint4 *ctr, const uint2 *key, uint4 *out, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = philox4x32_10(ctr[i], key[i].x, key[i].y);
}

__global__ void test_math_kernel(const float *x, float *ex, const double *u, double *lg, double *sn,
                                 double *cs, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) {
    ex[i] = dexpf(x[i]);
    lg[i] = log_core(u[i] > 0 ? u[i] : 1.0);
    double s, c;
    double v = u[i] - floor(u[i]);
    sincos2pi(v, &s, &c);
    sn[i] = s;
    cs[i] = c;
  }
}

__global__ void test_site_step_kernel(const KParams p, float4 *cells, float *lv, uint8_t *state,
                                      const uint32_t *vac, const float *dose, const float *draws,
                                      int32_t *ready, int32_t *used, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  ready[i] = 0;
  used[i] = 0;
  if (state[i] != kOccupied) return;
  DCell c = load_cell(cells + 3 * i);
  float l0 = lv[3 * i], l1 = lv[3 * i + 1], l2 = lv[3 * i + 2];
  if (!update_state(c, l0, l1, l2, p, vac[i])) {
    state[i] = kVacant;
    store_cell(cells + 3 * i, c);
    return;
  }
  if (dose[i] > 0) irradiate(c, dose[i], p);
  l0 -= met_of(p, c.mode, 0);
  l1 -= met_of(p, c.mode, 1);
  l2 -= met_of(p, c.mode, 2);
  lv[3 * i] = l0; lv[3 * i + 1] = l1; lv[3 * i + 2] = l2;
  const bool cc = progress_clock(c, p);
  bool dead = false;
  if (repair_pre(c, p, cc)) {
    used[i] = 1;
    if (draws[i] < death_prob(c, p)) dead = true;
    else { c.irr = 0.f; c.tir = 0.f; c.delay = 0.f; }
  }
  store_cell(cells + 3 * i, c);
  if (dead) state[i] = kVacant;
  else ready[i] = c.phase == 4;
}

__global__ void test_choose_kernel(const float *u, int r, int c, int W, int32_t *rc, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) {
    int s = choose_neighbour(r * W + c, W, u[i]);
    rc[2 * i] = s / W;
    rc[2 * i + 1] = s % W;
  }
}

__global__ void test_divide_kernel(const KParams p, float4 *parents, const float *z,
                                   float4 *children, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  DCell pc = load_cell(parents + 3 * i);
  pc.phase = 0;
  pc.prolif = 0.f;
  store_cell(parents + 3 * i, pc);
  float zz[5] = {z[5 * i], z[5 * i + 1], z[5 * i + 2], z[5 * i + 3], z[5 * i + 4]};
  store_cell(children + 3 * i, make_child(pc, zz, p));
}

__global__ void test_normals_kernel(const KParams p, const uint32_t *step, const uint32_t *sim,
                                    uint32_t epoch, float *z, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint4 r1 = draw(p, step[i], sim[i], 0xFFFFu, 0, 2, epoch);
  const uint4 r2 = draw(p, step[i], sim[i], 0xFFFFu, 0, 3, epoch);
  float unused;
  box_muller(r1.x, r1.y, &z[5 * i], &z[5 * i + 1]);
  box_muller(r1.z, r1.w, &z[5 * i + 2], &z[5 * i + 3]);
  box_muller(r2.x, r2.y, &z[5 * i + 4], &unused);
}

// one CTA: list rebuild, ROI on a lattice, or one diffusion step with the
// narrow (WIDE = false) or wide kernel's tiles
template <bool WIDE>
__global__ void __launch_bounds__(kThreads, WIDE ? 4 : 5)
    test_block_kernel(const KParams p, int mode, float *gfld, const uint8_t *gst, int32_t *roi,
                      uint8_t *mask, uint16_t *glist, uint32_t *gn) {
  constexpr int NT = kThreads;
  extern __shared__ __align__(16) uint8_t sm[];
  const int HW = p.HW;
  const SmemLayout L = smem_layout(p.H, p.W, p.lcap, WIDE ? kTierWide : kTierNarrow);
  float *fld = reinterpret_cast<float *>(sm + L.fld);
  uint8_t *st = sm + L.st;
  uint16_t *list = reinterpret_cast<uint16_t *>(sm + L.list);
  uint64_t *colmask = reinterpret_cast<uint64_t *>(sm + L.colmask);
  uint32_t *masks = reinterpret_cast<uint32_t *>(sm + L.masks);
  float *edge = reinterpret_cast<float *>(sm + L.edge);
  Misc *m = reinterpret_cast<Misc *>(sm + L.misc);
  for (int q = threadIdx.x; q < HW; q += NT) st[q] = gst ? gst[q] : 0;
  if (threadIdx.x == 0) {
    m->park = 0;
    m->w0 = -1;
    m->edge = 1;
  }
  __syncthreads();
  if (mode < 2) rebuild_list<NT>(st, list, m, p.H, p.W, HW, L.entries);
  if (mode == 0) {
    for (uint32_t q = threadIdx.x; q < m->n; q += NT) glist[q] = list[q];
    if (threadIdx.x == 0) *gn = m->n;
  } else if (mode == 1) {
    compute_roi<NT>(st, list, colmask, m, p.H, p.W);
    if (threadIdx.x == 0)
      for (int k = 0; k < 5; ++k) roi[k] = m->roi[k];
    const int mh = m->roi[2] + 2, mw = m->roi[3] + 2;
    if (m->roi[2] > 0)
      for (int q = threadIdx.x; q < mh * mw; q += NT) {
        int i = q / mw, j = q % mw;
        mask[q] = ((colmask[j] >> i) & 1ull) ? 0 : 1;
      }
  } else {
    if (threadIdx.x == 0)
      for (int k = 0; k < 5; ++k) m->roi[k] = roi[k];
    __syncthreads();
    build_colmask(colmask, m->roi[2], m->roi[3], m->roi[4]);
    __syncthreads();
    if (threadIdx.x < 32)
      tile_mapping(colmask, m, p.layouts, WIDE ? kNumTiles : kNarrowTiles, p.H, L.rows);
    __syncthreads();
    if (threadIdx.x == 0) {
      *gn = (WIDE || !m->park) ? 0u : 1u;
      m->w0 = m->wneed;
    }
    __syncthreads();
    if (!WIDE && m->park) return;
    build_masks<WIDE>(masks, colmask, m);
    for (int q = threadIdx.x; q < 3 * L.plane; q += NT)
      fld[q] = gfld[q / L.plane * HW + m->w0 * p.W + q % L.plane];
    __syncthreads();
    diffuse_step<WIDE>(fld, L.plane, masks, edge, m, p);
    __syncthreads();
    for (int q = threadIdx.x; q < 3 * L.plane; q += NT)
      gfld[q / L.plane * HW + m->w0 * p.W + q % L.plane] = fld[q];
  }
}

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------
// the dynamic shared-memory limit is raised once per device and size (the
// attribute call is kept out of CUDA-graph captures)
static size_t g_smem_set[3][64];

using RunKernel = void (*)(RunArgs, uint32_t);
static RunKernel kernel_of(int tier) {
  return tier == kTierNarrow ? run_kernel<kTierNarrow>
         : tier == kTierWide ? run_kernel<kTierWide> : run_kernel<kTierLone>;
}

static cudaError_t ensure_smem(int tier, size_t smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) dev = 63;
  if (g_smem_set[tier][dev] >= smem) return cudaSuccess;
  const RunKernel k = kernel_of(tier);
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // all ask for the same split of the L1, so that their CTAs share SMs
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e == cudaSuccess) g_smem_set[tier][dev] = smem;
  return e;
}

cudaError_t launch_run(const RunArgs &a, uint32_t t_end, int tier, int grid, cudaStream_t stream) {
  const size_t smem = run_kernel_smem(a.p.H, a.p.W, a.p.lcap, tier);
  cudaError_t e = ensure_smem(tier, smem);
  if (e != cudaSuccess) return e;
  kernel_of(tier)<<<grid, threads_of(tier), smem, stream>>>(a, t_end);
  return cudaGetLastError();
}

cudaError_t launch_order(const RunArgs &a, uint32_t t_end, uint32_t *hist, int64_t *out,
                         uint8_t *tier, int lone, cudaStream_t stream) {
  if (a.nsims < 1) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(hist, 0, kOrderKeys * sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  const int64_t blocks = (a.nsims + 255) / 256;
  const int grid = (int)(blocks < 4096 ? blocks : 4096);
  order_count_kernel<<<grid, 256, 0, stream>>>(a, t_end, hist);
  order_scan_kernel<<<1, 1024, 0, stream>>>(hist);
  order_scatter_kernel<<<grid, 256, 0, stream>>>(a, t_end, hist, out, tier, lone);
  return cudaGetLastError();
}

cudaError_t launch_tiers(const RunArgs &a, uint8_t *tier, int lone, bool narrow, int sms,
                         cudaStream_t stream) {
  tier_kernel<<<1, kTierThreads, 0, stream>>>(a, tier, lone, narrow, sms);
  return cudaGetLastError();
}

cudaError_t launch_reset(const ResetArgs &a, cudaStream_t stream) {
  int grid = (int)(a.nsims < 65535 * 8 ? a.nsims : 65535 * 8);
  if (grid < 1) return cudaSuccess;
  reset_kernel<<<grid, 256, 0, stream>>>(a);
  return cudaGetLastError();
}

int max_ctas_per_sm(const KParams &p, int tier) {
  const size_t smem = run_kernel_smem(p.H, p.W, p.lcap, tier);
  int n = 0;
  if (ensure_smem(tier, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_of(tier), threads_of(tier), smem) !=
          cudaSuccess)
    return 0;
  return n;
}

cudaError_t instr_read(unsigned long long counts[4], double *sum_dp, unsigned long long *hist) {
  cudaError_t e = cudaMemcpyFromSymbol(counts, g_instr_counts, sizeof(unsigned long long) * 4);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyFromSymbol(sum_dp, g_instr_sum_death_prob, sizeof(double));
  if (e != cudaSuccess) return e;
  if (hist) e = cudaMemcpyFromSymbol(hist, g_instr_hist, sizeof(unsigned long long) * 600);
  return e;
}

cudaError_t instr_reset() {
  unsigned long long z[600] = {0};
  double zd = 0.0;
  cudaError_t e = cudaMemcpyToSymbol(g_instr_counts, z, sizeof(unsigned long long) * 4);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyToSymbol(g_instr_sum_death_prob, &zd, sizeof(double));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(g_instr_hist, z, sizeof(z));
}

// FP32 issue-rate probe: 8 independent FMA chains per thread, register only
__global__ void __launch_bounds__(256) fma_probe_kernel(float *out, float a, float b, int iters) {
  float x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = a * (threadIdx.x + k);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = fmaf(x[k], b, a);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += x[k];
  if (s == 1234.5f) out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

cudaError_t fp32_peak(int device, double *tflops) {
  int sms = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, threads = 256, iters = 8192;
  float *out = nullptr;
  e = cudaMalloc(&out, sizeof(float) * blocks * threads);
  if (e != cudaSuccess) return e;
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  double best = 0;
  for (int rep = 0; rep < 12; ++rep) {
    cudaEventRecord(t0);
    fma_probe_kernel<<<blocks, threads>>>(out, 1.0001f, 0.9999f, iters);
    cudaEventRecord(t1);
    e = cudaEventSynchronize(t1);
    if (e != cudaSuccess) break;
    float ms = 0;
    cudaEventElapsedTime(&ms, t0, t1);
    const double flop = 2.0 * 8 * (double)iters * blocks * threads;
    if (rep >= 2 && ms > 0) best = fmax(best, flop / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  cudaFree(out);
  *tflops = best;
  return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t launch_test_philox(const uint4 *c, const uint2 *k, uint4 *o, int64_t n) {
  test_philox_kernel<<<(unsigned)((n + 127) / 128), 128>>>(c, k, o, n);
  return cudaGetLastError();
}
cudaError_t launch_test_math(const float *x, float *ex, const double *u, double *lg, double *sn,
                             double *cs, int64_t n) {
  test_math_kernel<<<(unsigned)((n + 127) / 128), 128>>>(x, ex, u, lg, sn, cs, n);
  return cudaGetLastError();
}
cudaError_t launch_test_site_step(const KParams &p, float4 *cells, float *lv, uint8_t *state,
                                  const uint32_t *vac, const float *dose, const float *draws,
                                  int32_t *ready, int32_t *used, int64_t n) {
  test_site_step_kernel<<<(unsigned)((n + 127) / 128), 128>>>(p, cells, lv, state, vac, dose,
                                                               draws, ready, used, n);
  return cudaGetLastError();
}
cudaError_t launch_test_choose(const float *u, int r, int c, int W, int32_t *rc, int64_t n) {
  test_choose_kernel<<<(unsigned)((n + 127) / 128), 128>>>(u, r, c, W, rc, n);
  return cudaGetLastError();
}
cudaError_t launch_test_divide(const KParams &p, float4 *parents, const float *z, float4 *children,
                               int64_t n) {
  test_divide_kernel<<<(unsigned)((n + 127) / 128), 128>>>(p, parents, z, children, n);
  return cudaGetLastError();
}
cudaError_t launch_test_normals(const KParams &p, const uint32_t *step, const uint32_t *sim,
                                uint32_t epoch, float *z, int64_t n) {
  test_normals_kernel<<<(unsigned)((n + 127) / 128), 128>>>(p, step, sim, epoch, z, n);
  return cudaGetLastError();
}
cudaError_t launch_test_block(const KParams &p, int mode, bool wide, float *fld,
                              const uint8_t *st, int32_t *roi, uint8_t *mask, uint16_t *list,
                              uint32_t *n) {
  wide = wide || mode < 2;  // lists and ROIs of any size
  const size_t smem = run_kernel_smem(p.H, p.W, p.lcap, wide ? kTierWide : kTierNarrow);
  cudaError_t e;
  if (wide) {
    e = cudaFuncSetAttribute(test_block_kernel<true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    test_block_kernel<true><<<1, kThreads, smem>>>(p, mode, fld, st, roi, mask, list, n);
  } else {
    e = cudaFuncSetAttribute(test_block_kernel<false>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    test_block_kernel<false><<<1, kThreads, smem>>>(p, mode, fld, st, roi, mask, list, n);
  }
  return cudaGetLastError();
}

}  // namespace emt6

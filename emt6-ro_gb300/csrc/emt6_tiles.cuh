// emt6_tiles.cuh -- register tiles of the diffusion step, one warp per field (four at
// the end of this file).
//
// A warp holds one field's active block in registers for the whole step (23 +
// 1 substeps): lane = 8 * bw + bl owns the C columns C*bl .. and the R rows
// R*bw .. of an 8C x 4R tile.  Horizontal neighbours across lanes cost two
// shuffles per row and lane, vertical ones two per column, so a lane's C x R
// slots need 2 (C + R) shuffles per substep, and no warp waits for another
// one inside a step.
//
// With H = x_left + x_right and G = b*x + d*H per site (fmaf(d, H, b*x)):
//   x' = a*x + b*(H + x_up + x_down) + d*(H_up + H_down)
//      = fmaf(a, x, fmaf(b, H, G_up + G_down))
// so a site needs its own x and H and the G of the rows above and below: six
// FP32 operations, the last FFMA predicated on the site's free bit, and
// 2 (C + R) / (C R) shuffles.  What bounds it is issue slots (83% busy in a
// diffusion-only loop), so the bits are laid out for the instruction that moves
// seven bits of a register's byte into the seven predicates: 7.6 instructions
// per slot and substep instead of 8.1 with a test per slot (28 slots: 5,230 vs
// 5,690 cycles per simulation step and SM).
#pragma once
#include <cstdint>

#include "emt6_device.cuh"

namespace emt6 {

// How a region is laid on a tile (tile_mapping).  Tile row 0 / column 0 is
// region row / column `off`; slots that hold no free site start at `fill`
// (block mode: the external level) or at the region's own value.
struct TileMap {
  int tile;  // index of tile_shape, or -1
  int C, R;  // its columns and rows per lane
  int off;   // 1: block mode (rows and columns 1..2d of an unclipped disc), 0: whole region
  int xrow, xcol;  // block mode: the ROI's last row / column lies outside the tile
};

// C, R: columns and rows per lane.  RE / CE: the rows / columns may fill the
// tile exactly, at the price of selects that replace what the rotating
// shuffles bring round from the opposite edge; without them one spare row /
// column of constant slots is what comes round.
struct TileShape {
  int C, R;
  bool RE, CE;
};
// Ordered by slots per lane; a region takes the first one it fits.  Discs of
// distance d (2d x 2d blocks) are what fills them: (2,3) d <= 6, (2,4) 7-8,
// (3,5) 9-10, (3,6) 11-12, (4,7) 13-14, (4,8) 15-16, (5,9) 17-18, (5,10)
// 19-20, (6,11) 21-22, (6,12) 23-24, (7,13) 25; the last two hold any other
// region of a 54 x 60 interior.
constexpr int kNumTiles = 21, kNarrowTiles = 12;
__host__ __device__ constexpr TileShape tile_shape(int k) {
  constexpr TileShape shapes[kNumTiles] = {
      {1, 2, false, false}, {2, 3, true, false},   {2, 4, false, false}, {2, 4, true, true},
      {3, 5, false, false}, {3, 5, true, false},   {3, 6, false, false}, {3, 6, true, true},
      {4, 7, false, false}, {4, 7, true, false},   {4, 8, false, false}, {4, 8, true, true},
      {5, 9, true, false},  {5, 10, false, false}, {5, 10, true, true},  {6, 11, true, false},
      {6, 12, false, false}, {6, 12, true, true},  {7, 13, true, false}, {7, 14, true, false},
      {8, 14, true, false}};
  return shapes[k];
}
// Slot bits: slot q = i * C + c of a lane is bit slot_bit(q) of word q / 28,
// seven slots to a byte.  The words of a tile lie in shared memory as
// [kind][word][lane], built with the ROI (build_masks).
enum { kFreeBits = 0, kRoiBits = 1, kInsideBits = 2 };
constexpr int kWordsNarrow = 2, kWordsWide = 4;
__host__ __device__ constexpr int slot_bit(int q) { return (q % 28) / 7 * 8 + q % 7; }

// words of a field's slots for a tile's last row and column (8C + 4R)
constexpr int kEdgeNarrow = 64, kEdgeWide = 120;

template <int C, int R, bool RE, bool CE>
__device__ __forceinline__ void diffuse_tile(float *__restrict__ f, const uint32_t *__restrict__ masks,
                                             int words, float *__restrict__ edge, const TileMap &tm,
                                             int r0, int c0, int w, int W, float ext, float ca,
                                             float cb, float cd, int nfree) {
  const int lane = threadIdx.x & 31, bw = lane >> 3, bl = lane & 7;
  const int left = (lane & 24) | ((bl + 7) & 7), right = (lane & 24) | ((bl + 1) & 7);
  const int up = (lane + 24) & 31, dn = (lane + 8) & 31;
  constexpr int NW = (R * C + 27) / 28;
  const int off = tm.off;
  const float out = off ? ext : 0.f;  // sites beyond the tile
  float *g = f + (r0 - 1 + bw * R + off) * W + (c0 - 1 + bl * C + off);
  // lanes whose up / down / left / right neighbour is outside the tile, as
  // masks the compiler cannot turn back into predicates (all seven are taken)
  uint32_t mt = bw == 0 ? 0u : ~0u, mb = bw == 3 ? 0u : ~0u, ml = bl == 0 ? 0u : ~0u,
           mr = bl == 7 ? 0u : ~0u;
  asm("" : "+r"(mt), "+r"(mb), "+r"(ml), "+r"(mr));
  auto within = [](uint32_t mk, float a, float b) -> float {
    return __uint_as_float((__float_as_uint(a) & mk) | (__float_as_uint(b) & ~mk));
  };
  uint32_t pm[NW];  // sites that change: the free ones, in the last substep the ROI's
  float X[R][C];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) X[i][c] = out;
  if (!off) {
    // whole region: its fixed sites are at the external level
#pragma unroll
    for (int k = 0; k < NW; ++k) pm[k] = masks[(kInsideBits * words + k) * 32 + lane];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (pm[(i * C + c) / 28] & (1u << slot_bit(i * C + c))) X[i][c] = ext;
  }
#pragma unroll
  for (int k = 0; k < NW; ++k) pm[k] = masks[(kFreeBits * words + k) * 32 + lane];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (pm[(i * C + c) / 28] & (1u << slot_bit(i * C + c))) X[i][c] = g[i * W + c];
  const float gout = fmaf(cd, out + out, cb * out);
  for (int s = 0; s <= nfree; ++s) {
    if (s == nfree) {
      // final substep: every site of the ROI
#pragma unroll
      for (int k = 0; k < NW; ++k) pm[k] = masks[(kRoiBits * words + k) * 32 + lane];
      if (RE && bw == 3) {
#pragma unroll
        for (int c = 0; c < C; ++c) edge[C * bl + c] = X[R - 1][c];
      }
      if (CE && bl == 7) {
#pragma unroll
        for (int i = 0; i < R; ++i) edge[8 * C + bw * R + i] = X[i][C - 1];
      }
    }
    float lv[R], rv[R];
    auto hshuffle = [&](int i) {
      lv[i] = __shfl_sync(kFull, X[i][C - 1], left);
      rv[i] = __shfl_sync(kFull, X[i][0], right);
      if (CE) {
        lv[i] = within(ml, lv[i], out);
        rv[i] = within(mr, rv[i], out);
      }
    };
    auto hsum = [&](int i, int c) -> float {
      return (c == 0 ? lv[i] : X[i][c > 0 ? c - 1 : 0]) +
             (c == C - 1 ? rv[i] : X[i][c < C - 1 ? c + 1 : 0]);
    };
    // the band's first and last rows first: their G crosses to other lanes.
    // Tiles of up to 50 slots fetch every row's neighbours at once, larger
    // ones a row ahead (their registers are taken by the tile).
    constexpr bool AHEAD = C * R > 50;
    hshuffle(0);
    if (R > 1) hshuffle(R - 1);
    if (!AHEAD) {
#pragma unroll
      for (int i = 1; i < R - 1; ++i) hshuffle(i);
    } else if (R > 2) {
      hshuffle(1);
    }
    float hb[C], gb[C], hc[C], gc[C], gm[C], gx[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      hc[c] = hsum(0, c);
      gc[c] = fmaf(cd, hc[c], cb * X[0][c]);
      hb[c] = hsum(R - 1, c);
      gb[c] = fmaf(cd, hb[c], cb * X[R - 1][c]);
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      gm[c] = __shfl_sync(kFull, gb[c], up);  // the row above the band
      gx[c] = __shfl_sync(kFull, gc[c], dn);  // the row below it
      if (RE) {
        gm[c] = within(mt, gm[c], gout);
        gx[c] = within(mb, gx[c], gout);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (AHEAD && i + 2 < R - 1) hshuffle(i + 2 < R ? i + 2 : 0);
      float hn[C], gn[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (i + 1 == R) {
          hn[c] = 0.f;
          gn[c] = gx[c];
        } else if (i + 1 == R - 1) {
          hn[c] = hb[c];
          gn[c] = gb[c];
        } else {
          hn[c] = hsum(i + 1 < R ? i + 1 : 0, c);
          gn[c] = fmaf(cd, hn[c], cb * X[i + 1 < R ? i + 1 : 0][c]);
        }
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float t = fmaf(cb, hc[c], gm[c] + gn[c]);
        if (pm[(i * C + c) / 28] & (1u << slot_bit(i * C + c))) X[i][c] = fmaf(ca, X[i][c], t);
        gm[c] = gc[c];
        gc[c] = gn[c];
        hc[c] = hn[c];
      }
    }
  }
  // the last substep's bits are the sites to store
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (pm[(i * C + c) / 28] & (1u << slot_bit(i * C + c))) g[i * W + c] = X[i][c];
  if (RE && (tm.xrow | tm.xcol)) {
    // block mode with 2d = 4R rows (8C columns): the final substep of the
    // ROI's last row (column) n = 2d + 1, outside the tile.  Every site there
    // is fixed (x = ext) and so are its neighbours outside the tile; the
    // tile's last row and column are those before the substep.
    __syncwarp();
    const int n = w;
    const float gfix = fmaf(cd, ext + ext, cb * ext);  // G of an all-fixed row
    float *q = f + (r0 - 1) * W + (c0 - 1);
    if (tm.xrow)
      for (int j = lane + 1; j <= n; j += 32) {  // (n, j)
        const float xl = j >= 2 ? edge[j - 2] : ext, xc = j <= n - 1 ? edge[j - 1] : ext,
                    xr = j <= n - 2 ? edge[j] : ext;
        const float gu = fmaf(cd, xl + xr, cb * xc);
        q[n * W + j] = fmaf(ca, ext, fmaf(cb, ext + ext, gu + gfix));
      }
    if (CE && tm.xcol)
      for (int i = lane + 1; i <= n - 1; i += 32) {  // (i, n); (n, n) is with the row
        const float xu = i >= 2 ? edge[8 * C + i - 2] : ext, xc = edge[8 * C + i - 1],
                    xd = i <= n - 2 ? edge[8 * C + i] : ext;
        const float gu = fmaf(cd, xu + ext, cb * ext), gd = fmaf(cd, xd + ext, cb * ext);
        q[i * W + n] = fmaf(ca, ext, fmaf(cb, xc + ext, gu + gd));
      }
  }
}

// The same as a function of its own, for tiles of 72 slots and more: their
// registers leave no room for the kernel's own variables, which the inlined form
// spills inside the substeps (608 discs of distance 23-25, 300 steps: 13.3 vs
// 15.2 ms).  Smaller tiles are faster inlined, where the coefficients come from
// the constant bank.
template <int C, int R, bool RE, bool CE>
__device__ __noinline__ void diffuse_large(float *f, const uint32_t *masks, int words, float *edge,
                                           const TileMap *tm, int r0, int c0, int w, int W,
                                           float ext, float ca, float cb, float cd, int nfree) {
  diffuse_tile<C, R, RE, CE>(f, masks, words, edge, *tm, r0, c0, w, W, ext, ca, cb, cd, nfree);
}

// A whole region of up to 4 RH x 63 sites by four warps per field: warp `part`
// holds rows RH part .. of it, a lane columns 2 lane and 2 lane + 1 (ring
// included, zero around the region).  The G of a part's first and last row cross
// through shared memory, a barrier of the field's warps per substep: slower per
// SM than one warp per tile, but a lone warp fetches and issues an instruction in
// two cycles, so that a simulation with an SM to itself is done sooner this way
// from 72 slots on (152 discs of radius 24, 200 steps: 3.0 ms, 5.0 with one warp per
// field in the same CTA; of radius 22, 66 slots, 3.1 with one).  `slots` holds
// 2 x 4 x 2 rows of 32 float2.
constexpr int kPartSlots = 2 * 4 * 2 * 32;
template <int RH>
__device__ __forceinline__ void diffuse_parts(float *__restrict__ f, const uint64_t *__restrict__ colmask,
                                              float2 *__restrict__ slots, int part, int barrier, int r0,
                                              int c0, int h, int w, int W, float ext, float ca,
                                              float cb, float cd, int nfree) {
  const int lane = threadIdx.x & 31, base = part * RH, j0 = 2 * lane, j1 = j0 + 1;
  const int left = (lane + 31) & 31, right = (lane + 1) & 31;
  constexpr uint32_t kRows = (1u << RH) - 1u;
  const bool in0 = j0 < w + 2, in1 = j1 < w + 2;
  const uint32_t free0 = in0 ? (uint32_t)(colmask[j0] >> base) & kRows : 0u;
  const uint32_t free1 = in1 ? (uint32_t)(colmask[j1] >> base) & kRows : 0u;
  const uint32_t rows = (uint32_t)((((1ull << h) - 1ull) << 1) >> base) & kRows;
  const uint32_t roi0 = j0 >= 1 && j0 <= w ? rows : 0u, roi1 = j1 <= w ? rows : 0u;
  float *g = f + (r0 - 1 + base) * W + c0 - 1;
  float x0[RH], x1[RH];
#pragma unroll
  for (int i = 0; i < RH; ++i) {
    const bool in = base + i < h + 2;
    x0[i] = in && in0 ? ext : 0.f;
    x1[i] = in && in1 ? ext : 0.f;
    if (free0 >> i & 1u) x0[i] = g[i * W + j0];
    if (free1 >> i & 1u) x1[i] = g[i * W + j1];
  }
#pragma unroll 1
  for (int s = 0; s <= nfree; ++s) {
    const uint32_t u0 = s == nfree ? roi0 : free0, u1 = s == nfree ? roi1 : free1;
    float2 *row = slots + (s & 1) * (4 * 2 * 32) + lane;  // [part][first, last]
    const float ht0 = __shfl_sync(kFull, x1[0], left) + x1[0];
    const float ht1 = x0[0] + __shfl_sync(kFull, x0[0], right);
    const float hb0 = __shfl_sync(kFull, x1[RH - 1], left) + x1[RH - 1];
    const float hb1 = x0[RH - 1] + __shfl_sync(kFull, x0[RH - 1], right);
    const float2 gt = make_float2(fmaf(cd, ht0, cb * x0[0]), fmaf(cd, ht1, cb * x1[0]));
    const float2 gb = make_float2(fmaf(cd, hb0, cb * x0[RH - 1]), fmaf(cd, hb1, cb * x1[RH - 1]));
    row[(part * 2 + 0) * 32] = gt;
    row[(part * 2 + 1) * 32] = gb;
    asm volatile("bar.sync %0, 128;" ::"r"(barrier) : "memory");
    float2 above = make_float2(0.f, 0.f), below = above;
    if (part > 0) above = row[(part * 2 - 1) * 32];
    if (part < 3) below = row[(part * 2 + 2) * 32];
    float gm0 = above.x, gm1 = above.y, gc0 = gt.x, gc1 = gt.y, hc0 = ht0, hc1 = ht1;
#pragma unroll
    for (int i = 0; i < RH; ++i) {
      float hn0 = hb0, hn1 = hb1, gn0 = gb.x, gn1 = gb.y;
      if (i + 1 < RH - 1) {
        hn0 = __shfl_sync(kFull, x1[i + 1], left) + x1[i + 1];
        hn1 = x0[i + 1] + __shfl_sync(kFull, x0[i + 1], right);
        gn0 = fmaf(cd, hn0, cb * x0[i + 1]);
        gn1 = fmaf(cd, hn1, cb * x1[i + 1]);
      } else if (i + 1 == RH) {
        gn0 = below.x;
        gn1 = below.y;
      }
      const float n0 = fmaf(ca, x0[i], fmaf(cb, hc0, gm0 + gn0));
      const float n1 = fmaf(ca, x1[i], fmaf(cb, hc1, gm1 + gn1));
      x0[i] = u0 >> i & 1u ? n0 : x0[i];
      x1[i] = u1 >> i & 1u ? n1 : x1[i];
      gm0 = gc0;
      gm1 = gc1;
      gc0 = gn0;
      gc1 = gn1;
      hc0 = hn0;
      hc1 = hn1;
    }
  }
#pragma unroll
  for (int i = 0; i < RH; ++i) {
    if (roi0 >> i & 1u) g[i * W + j0] = x0[i];
    if (roi1 >> i & 1u) g[i * W + j1] = x1[i];
  }
}

}  // namespace emt6

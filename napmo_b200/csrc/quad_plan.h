// How the FP64 quadrature (quad.cu) is split into partial sums: plain host code,
// without CUDA, so that its bounds can be checked on any machine.
#pragma once

#include <algorithm>
#include <cstddef>

#ifdef __CUDACC__
#define NAPMO_QUAD_FN __host__ __device__ __forceinline__
#else
#define NAPMO_QUAD_FN inline
#endif

namespace napmo {

constexpr int kQuadTile = 128;  // functions of a tile
constexpr int kQuadStage = 16;  // points per stage
// Whole triangle of fragments per warp up to this n.  B200, 66,000 points,
// quadrature / density, us, against the tiled kernels: 40 functions 27 / 17 (35 /
// 27), 48 27 / 17 (43 / 27), 49 to 64 31 / 25 (45 / 33), the last with 255
// registers and 32 bytes spilled in the density; more functions do not fit.
constexpr int kSmallN = 64;
// row tiles of 16 that cover n <= kSmallN, and their upper-triangle fragments
NAPMO_QUAD_FN constexpr int small_tiles(int n) { return (n + 15) / 16; }
NAPMO_QUAD_FN constexpr int small_frags(int rt) { return rt * (rt + 1); }

// Split of an FP64 quadrature into partial sums (quad_plan_slots).
// n <= 64: class 0 holds nch[0] chunks of chunk[0] points, one warp each.
// n > 64: the 128 x 128 tiles of the upper triangle in four classes of equal
// cost (right of the diagonal: full, last column; diagonal: full, last); class
// c has ntile[c] tiles, each split into nch[c] chunks of chunk[c] points, its
// CTAs numbered from first[c], tile fastest; CTA b writes workspace slot b.
struct QuadPlan {
  int ntile[4], nch[4], chunk[4], first[5];
};

// Tile `t` of class `c` (QuadPlan) of nblk x nblk blocks.
NAPMO_QUAD_FN void quad_tile(int c, int t, int nblk, int &mb, int &nb) {
  if (c == 0) {
    nb = 1;
    while (t >= nb) t -= nb++;
    mb = t;
  } else if (c == 1) {
    mb = t;
    nb = nblk - 1;
  } else {
    mb = nb = c == 2 ? t : nblk - 1;
  }
}

// Cost of a stage of one tile: DMMA instructions per k8 step of the busiest
// sub-partition (warps w and w + 4), plus the stage's fixed part (barrier and
// copies, about 4 of them; without it 310 functions x 1,147,600 points take 5.82
// instead of 5.31 ms).
inline int quad_tile_cost(int n, int nblk, int cls) {
  const bool ragged = cls == 1 || cls == 3;
  const int cols = ragged ? n - (nblk - 1) * kQuadTile : kQuadTile;
  const int C = (cols + 7) / 8, R = (cols + 15) / 16;
  const int groups4 = (C + 3) / 4 * 4, frags3 = (C - R + 1 + 2) / 3 * 3;
  return 4 + (cls < 2 ? 2 * groups4 : (R > 4 ? 2 : 1) * frags3);
}

// The split for at most `slots` partial tiles (n > 64) or chunks (n <= 64).
// *bound (optional) receives the most slots that any range of at most npad
// points uses: a shorter range can be cut into more chunks (chunk lengths are
// rounded up to 16 points), up to one per 16 points and the counts below.
inline QuadPlan quad_plan_slots(int n, int npad, int slots, long *bound = nullptr) {
  QuadPlan p = {};
  if (bound) *bound = 0;
  auto split = [&](int c) {  // chunk length and count for at most nch[c] chunks
    if (bound) *bound += (long)p.ntile[c] * std::max(std::min(p.nch[c], npad / kQuadStage), 1);
    int chunk = (npad + p.nch[c] - 1) / p.nch[c];
    chunk = std::max((chunk + kQuadStage - 1) / kQuadStage * kQuadStage, kQuadStage);
    p.chunk[c] = chunk;
    p.nch[c] = (npad + chunk - 1) / chunk;
  };
  if (n <= kSmallN) {
    p.ntile[0] = 1;
    p.nch[0] = slots;
    split(0);
    for (int c = 1; c < 5; ++c) p.first[c] = p.nch[0];
    return p;
  }
  const int nblk = (n + kQuadTile - 1) / kQuadTile;
  p.ntile[0] = (nblk - 1) * (nblk - 2) / 2;
  p.ntile[1] = nblk - 1;
  p.ntile[2] = nblk - 1;
  p.ntile[3] = 1;
  long total = 0;
  int cost[4];
  for (int c = 0; c < 4; ++c) {
    cost[c] = quad_tile_cost(n, nblk, c);
    total += (long)cost[c] * p.ntile[c];
  }
  // chunks in proportion to the cost, so that all CTAs take about as long
  for (int s = slots;; --s) {
    long used = 0;
    bool single = true;
    for (int c = 0; c < 4; ++c) {
      p.nch[c] = (int)std::max<long>((long)s * cost[c] / total, 1);
      used += (long)p.nch[c] * p.ntile[c];
      single = single && p.nch[c] == 1;
    }
    if (used <= slots || single) break;
  }
  for (int c = 0; c < 4; ++c) {
    split(c);
    p.first[c + 1] = p.first[c] + p.nch[c] * p.ntile[c];
  }
  return p;
}

// Slots: n <= 64 (a warp per chunk) four warps per SM; n > 64 (a CTA per slot,
// one CTA per SM at these register counts) two full waves over the 148 SMs for
// a single tile (110 functions x 200,000 points 171 us, 185 with four), four
// otherwise (310 functions x 1,147,600 points 5.31 ms, 5.72 with two).
inline int quad_default_slots(int n) { return n > kSmallN && n <= kQuadTile ? 2 * 148 : 4 * 148; }

// Doubles of workspace for every range of at most npad points.
inline size_t quad_workspace_doubles(int n, int npad) {
  long slots = 0;
  quad_plan_slots(n, npad, quad_default_slots(n), &slots);
  return (size_t)slots *
         (n <= kSmallN ? 128 * small_frags(small_tiles(n)) : kQuadTile * kQuadTile);
}

}  // namespace napmo

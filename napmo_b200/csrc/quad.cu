// FP64 grid quadratures (the plain FP64 path) on the FP64 tensor pipe:
//
//   density     rho[p]     = sum_{mu,nu} phi[mu][p] D[mu][nu] phi[nu][p]
//   quadrature  F[mu][nu]  = sum_p phi[mu][p] wv[p] phi[nu][p]
//               (or sum_p phi[mu][p] wv[p] psi[nu][p] for a second operand psi,
//               upper triangle mirrored as nAPMO does for exchange)
//
// nAPMO computes the density point by point in Python (psi_hybrid.py:144-150)
// and the quadrature by materialising every orbital product
// Psi[n(n+1)/2][N] (src/wavefunction/nwavefunction.cpp:77-107,161-197).  Here
// both are FP64 GEMMs over phi stored basis-major [n][ld] (ld a multiple of
// 128, zero padded), issued as mma.sync m16n8k8 f64 (DMMA: 2048 flops per
// warp instruction, FP64 accumulation).  Both are bound by the FP64 tensor
// pipe (64 FMA per clock and SM, one m16n8k8 per 64 clocks and sub-partition;
// a cuBLAS DGEMM of 8192^3 reaches 35.5 TFLOP/s), so what counts is that no
// instruction is spent on entries nobody needs: work is dropped in 16 x 8
// (quadrature) and 16 x 16 (density) fragments, below the diagonal and beyond
// the last basis function.
//
//   * n <= 64 (kSmallN): every warp holds the whole upper triangle of
//     fragments and works on its own points, straight from global memory to
//     registers; the CTA's 8 warps are summed in shared memory (quadrature).
//     With 128-wide tiles a 25-function molecule spent 16 % of a tile's
//     fragments, and wrote 128 x 128 partial sums per chunk (77 MB).
//   * n > 64: 128 x 128 tiles per CTA from a 4-stage cp.async ring, 8 warps
//     as 2 x 4, each 4 x 4 fragments interleaved over the tile (rows 16 (wr +
//     2 mt), columns 8 (wc + 4 nt)), so that the fragments left of a diagonal
//     or ragged tile are spread over the four sub-partitions.
//
// density: D, symmetric or not, is folded onto block-upper-triangular form at
// 16 x 16 (row tile i takes nu from its own first row on; right of its diagonal
// block D' = D[mu][nu] + D[nu][mu]); T' = D' phi is folded into the per-point
// sum with phi[mu][p] as soon as a row tile is complete; deterministic, no
// atomics.
// quadrature: split-K over points; chunk partials go to a workspace and a
// second kernel adds them in a fixed order and writes both triangles, so F is
// exactly symmetric and bit-reproducible.
//
// Shared-memory rows are padded to a stride of 4 mod 16 doubles, so the
// fragment loads of each half-warp hit 16 distinct banks.
//
// Measured (B200, 1965 MHz; before: whole 128 x 128 tiles for every n):
//   density     H2O (25 functions, 16,500 points)          8.2 ->  4.0 us
//               C12H26 (310 functions, 1,147,600 points)  6.25 -> 4.50 ms
//   quadrature  H2O, both kernels                           87 ->   11 us
//               C8H18 (210 functions, 785,200 points)     2.63 -> 1.78 ms
//               C12H26                                    7.51 -> 5.30 ms
#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>

#include "common.h"
#include "dmma.cuh"
#include "kernels.cuh"
#include "quad_plan.h"

namespace napmo {

namespace {

constexpr int BM = kQuadTile, BN = kQuadTile, NT = 256;
constexpr int BK = kQuadStage;         // points (quadrature) / functions (density) per stage
constexpr int NS = 4;                  // stages of the cp.async ring
constexpr int LDA = BK + 4;            // [row][k] tiles: stride 20 doubles
constexpr int LDB = BN + 4;            // density phi tile [nu][p]: stride 132 doubles

struct QuadSmem {
  double a[NS][BM][LDA];               // phi rows mu0.. over the stage's points
  double b[NS][BN][LDA];               // psi rows nu0..
  double w[NS][BK];                    // wv over the stage's points
};

struct DensSmem {
  double a[NS][BM][LDA];               // D' rows mu0.. over the stage's nu
  double b[NS][BK][LDB];               // phi rows nu over the CTA's 128 points
  double red[2][BN];                   // per-point sums of the two warp rows
};

constexpr size_t kQuadSmem = sizeof(QuadSmem);
constexpr size_t kDensSmem = sizeof(DensSmem);

// 16-byte asynchronous global -> shared copies; src_bytes = 0 fills the
// destination with zeros (rows beyond n) without reading the source.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
               "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr int kWarps = NT / 32;

// ------------------------------------------------------------------ density
// n <= 64: T'[i] = D'[i] phi for 8 points, rho = sum of T' phi.  A warp keeps
// the fragments of D' (row tile i, k8 step kk >= 2 i), formed as they are loaded,
// in registers for all its points.
template <int RT>
__device__ __forceinline__ void density_small_frags(int n, const double *__restrict__ D,
                                                    double (&a)[RT * (RT + 1)][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  int f = 0;
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int kk = 2 * i; kk < 2 * RT; ++kk, ++f)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int mu = 16 * i + g + 8 * (c & 1), nu = 8 * kk + q + 4 * (c >> 1);
        const bool v = mu < n && nu < n;
        a[f][c] = v ? __ldg(D + (long)mu * n + nu) : 0.0;
        if (kk >= 2 * i + 2 && v) a[f][c] += __ldg(D + (long)nu * n + mu);
      }
}

template <int RT>
__device__ __forceinline__ void density_small_points(const double (&a)[RT * (RT + 1)][4], int n,
                                                     int npoint, const double *__restrict__ phi,
                                                     long ld, double *__restrict__ rho, int p0,
                                                     const int *__restrict__ keep) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double b[2 * RT][2];
#pragma unroll
  for (int kk = 0; kk < 2 * RT; ++kk)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int nu = 8 * kk + q + 4 * h;
      b[kk][h] = nu < n ? __ldg(phi + (long)nu * ld + p0 + g) : 0.0;
    }
  double2 fr[RT][2];  // phi[mu] of the accumulator's rows and columns
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int mu = 16 * i + g + 8 * h;
      fr[i][h] = mu < n ? __ldg(reinterpret_cast<const double2 *>(phi + (long)mu * ld + p0 + 2 * q))
                        : make_double2(0.0, 0.0);
    }
  double s0 = 0.0, s1 = 0.0;
  int f = 0;
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int kk = 2 * i; kk < 2 * RT; ++kk, ++f) dmma(acc, a[f], b[kk]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      s0 = fma(acc[2 * h], fr[i][h].x, s0);
      s1 = fma(acc[2 * h + 1], fr[i][h].y, s1);
    }
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (g < 2) {  // lane (g, q) writes point 2 q + g
    const int p = p0 + 2 * q + g;
    if (p < npoint) rho[p] = (keep && !keep[p]) ? 0.0 : (g ? s1 : s0);
  }
}

// The 128-point groups bx, bx + gx, ... of `ngroup` (listed in `groups`, or
// all): warp w takes points 16 w .. 16 w + 15 of each.
template <int RT>
__device__ __forceinline__ void density_small_block(int n, int npoint,
                                                    const double *__restrict__ phi, long ld,
                                                    const double *__restrict__ D,
                                                    double *__restrict__ rho,
                                                    const int *__restrict__ groups, int ngroup,
                                                    int bx, int gx,
                                                    const int *__restrict__ keep) {
  double a[RT * (RT + 1)][4];
  density_small_frags<RT>(n, D, a);
  const int warp = threadIdx.x >> 5;
  for (int gi = bx; gi < ngroup; gi += gx) {
    const int p0 = (groups ? groups[gi] : gi) * BN + 16 * warp;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      density_small_points<RT>(a, n, npoint, phi, ld, rho, p0 + 8 * h, keep);
  }
}

__device__ __forceinline__ void density_small_any(int n, int npoint,
                                                  const double *__restrict__ phi, long ld,
                                                  const double *__restrict__ D,
                                                  double *__restrict__ rho,
                                                  const int *__restrict__ groups, int ngroup,
                                                  int bx, int gx, const int *__restrict__ keep) {
  switch (small_tiles(n)) {
    case 1: density_small_block<1>(n, npoint, phi, ld, D, rho, groups, ngroup, bx, gx, keep); break;
    case 2: density_small_block<2>(n, npoint, phi, ld, D, rho, groups, ngroup, bx, gx, keep); break;
    case 3: density_small_block<3>(n, npoint, phi, ld, D, rho, groups, ngroup, bx, gx, keep); break;
    default: density_small_block<4>(n, npoint, phi, ld, D, rho, groups, ngroup, bx, gx, keep);
  }
}

template <int RT>
__global__ void __launch_bounds__(NT)
density_small_kernel(int n, int npoint, const double *__restrict__ phi, long ld,
                     const double *__restrict__ D, double *__restrict__ rho,
                     const int *__restrict__ groups, int ngroup, const int *__restrict__ keep) {
  density_small_block<RT>(n, npoint, phi, ld, D, rho, groups, ngroup, blockIdx.x, gridDim.x,
                          keep);
}

// n > 64.  Stages of a CTA: block mb of mu takes nu from mb*BM to n (rounded up
// to BK = 16), the blocks one after the other; within a block the nu right of
// the diagonal block come first and the diagonal block's own nu last, in
// descending order, so that row tile i (16 rows) takes every stage up to its
// own one and none after it.  Its phi rows are then in the stage's shared
// memory, where the fold into rho reads them.
struct DensStage {
  int mb, k0;
  int diag;  // the stage's row tile within the diagonal block, or 8 right of it
};
__device__ __forceinline__ void density_stage_next(DensStage &s, int nk) {
  constexpr int SB = BM / BK;                      // stages per 128 functions
  const int k = s.k0 / BK;
  if (s.diag == SB) {                              // right of the diagonal block
    if (k + 1 < nk) {
      s.k0 += BK;
    } else {
      s.diag = SB - 1;                             // a full block: others lie right of it
      s.k0 = (s.mb * SB + s.diag) * BK;
    }
  } else if (s.diag > 0) {
    --s.diag;
    s.k0 -= BK;
  } else {
    ++s.mb;
    if ((s.mb + 1) * SB < nk) {
      s.diag = SB;
      s.k0 = (s.mb + 1) * SB * BK;
    } else {
      s.diag = min(SB, nk - s.mb * SB) - 1;
      s.k0 = (s.mb * SB + s.diag) * BK;
    }
  }
}

// D' of n > 64, [n][fold_ld(n)]: what density_kernel reads, nu from the first
// row of mu's 16-row tile on (the rest is left unset), zero in the padding.  A
// pass of its own, 2.5 us: adding the transposed tile inside density_kernel,
// whose copies of D it doubles, made that 17 % slower (310 functions).
__host__ __device__ constexpr int fold_ld(int n) { return (n + 1) / 2 * 2; }

__device__ __forceinline__ void density_fold_body(int n, const double *__restrict__ D,
                                                  double *__restrict__ out, long e) {
  const int ldd = fold_ld(n);
  const int mu = (int)(e / ldd), nu = (int)(e - (long)mu * ldd);
  if (mu >= n || nu < mu / 16 * 16) return;
  double d = nu < n ? __ldg(D + (long)mu * n + nu) : 0.0;
  if (nu < n && nu / 16 > mu / 16) d += __ldg(D + (long)nu * n + mu);
  out[e] = d;
}

__global__ void __launch_bounds__(NT)
density_fold_kernel(int n, const double *__restrict__ D, double *__restrict__ out) {
  density_fold_body(n, D, out, (long)blockIdx.x * NT + threadIdx.x);
}

// rho of the 128 points p0 .. p0 + 127 (one CTA; see density_kernel) from D'.
__device__ __forceinline__ void density_block(DensSmem &sm, int n, int npoint,
                                              const double *__restrict__ phi, long ld,
                                              const double *__restrict__ D,
                                              double *__restrict__ rho, int p0,
                                              const int *__restrict__ keep) {
  constexpr int SB = BM / BK;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int wr = warp >> 2, wcol = (warp & 3) * 32;
  const int nblk = (n + BM - 1) / BM, ldd = fold_ld(n);
  const int nk = (n + BK - 1) / BK;                 // stages of nu over the whole basis
  int nstage = 0;
  for (int mb = 0; mb < nblk; ++mb) nstage += nk - mb * SB;

  // copies of one stage, 16 bytes each: D' rows (in a diagonal stage only the
  // row tiles that still take it) and phi rows (p0 + c and ld are even)
  auto load_stage = [&](const DensStage &st, int slot) {
    const int rows = st.diag == SB ? BM : 16 * (st.diag + 1);
#pragma unroll
    for (int i = 0; i < (BM * BK / 2) / NT; ++i) {
      const int e = t + NT * i, r = e / (BK / 2), c = (e % (BK / 2)) * 2;
      const int mu = st.mb * BM + r, nu = st.k0 + c;
      const bool v = mu < n && nu < ldd;
      if (r < rows) cp_async16(&sm.a[slot][r][c], D + (v ? (long)mu * ldd + nu : 0), v);
    }
#pragma unroll
    for (int i = 0; i < (BK * BN / 2) / NT; ++i) {
      const int e = t + NT * i, r = e / (BN / 2), c = (e % (BN / 2)) * 2;
      const int nu = st.k0 + r;
      const bool v = nu < n;
      cp_async16(&sm.b[slot][r][c], phi + (v ? (long)nu * ld + p0 + c : 0), v);
    }
  };

  double part[4][2];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) part[nt][0] = part[nt][1] = 0.0;
  double acc[4][4][4];
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[mt][nt][i] = 0.0;

  DensStage ld_st{-1, 0, 0}, st{-1, 0, 0};
  density_stage_next(ld_st, nk);
  density_stage_next(st, nk);
#pragma unroll
  for (int i = 0; i < NS - 1; ++i) {
    if (i < nstage) {
      load_stage(ld_st, i);
      density_stage_next(ld_st, nk);
    }
    cp_async_commit();
  }
  for (int it = 0; it < nstage; ++it) {
    cp_async_wait<NS - 2>();
    __syncthreads();
    auto next_copies = [&] {
      if (it + NS - 1 < nstage) {
        load_stage(ld_st, (it + NS - 1) % NS);
        density_stage_next(ld_st, nk);
      }
      cp_async_commit();
    };
    // half of each sub-partition's warps issue the copies before their
    // products, the other half after the first ones: its pipe does not idle
    if (wr == 0) next_copies();
    const int slot = it % NS;
    const double(*at)[LDA] = sm.a[slot];
    const double(*bt)[LDB] = sm.b[slot];
    const int left = nk - st.mb * SB;             // row tiles of the block
    double b[2][4][2];
#pragma unroll
    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int c = wcol + nt * 8 + g;
        b[kk][nt][0] = bt[8 * kk + q][c];
        b[kk][nt][1] = bt[8 * kk + q + 4][c];
      }
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      if (wr == 1 && mt == 1) next_copies();
      const int i = wr + 2 * mt;                  // row tile within the block
      if (i > st.diag || i >= left) continue;     // warp-uniform
      const int r = 16 * i + g;
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        const double af[4] = {at[r][8 * kk + q], at[r + 8][8 * kk + q], at[r][8 * kk + q + 4],
                              at[r + 8][8 * kk + q + 4]};
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) dmma(acc[mt][nt], af, b[kk][nt]);
      }
      if (i == st.diag) {  // complete: part[p] += sum_mu T'[mu][p] phi[mu][p]
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const double2 f =
                *reinterpret_cast<const double2 *>(&bt[g + 8 * h][wcol + nt * 8 + 2 * q]);
            part[nt][0] = fma(acc[mt][nt][2 * h], f.x, part[nt][0]);
            part[nt][1] = fma(acc[mt][nt][2 * h + 1], f.y, part[nt][1]);
            acc[mt][nt][2 * h] = acc[mt][nt][2 * h + 1] = 0.0;
          }
      }
    }
    density_stage_next(st, nk);
  }
  cp_async_wait<0>();
  // sum over the warp's rows (lanes of equal q), then over the two warp rows
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      double v = part[nt][j];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      part[nt][j] = v;
    }
  if (g == 0) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      sm.red[warp >> 2][wcol + nt * 8 + 2 * q] = part[nt][0];
      sm.red[warp >> 2][wcol + nt * 8 + 2 * q + 1] = part[nt][1];
    }
  }
  __syncthreads();
  if (t < BN && p0 + t < npoint)
    rho[p0 + t] = (keep && !keep[p0 + t]) ? 0.0 : sm.red[0][t] + sm.red[1][t];
}

// groups (optional): the 128-point groups to compute (screened plans; the
// others hold no kept point); keep (optional): rho = 0 at dropped points.
__global__ void __launch_bounds__(NT, 1)
density_kernel(int n, int npoint, const double *__restrict__ phi, long ld,
               const double *__restrict__ D, double *__restrict__ rho,
               const int *__restrict__ groups, const int *__restrict__ keep) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  DensSmem &sm = *reinterpret_cast<DensSmem *>(smem_raw);
  const int p0 = (groups ? groups[blockIdx.x] : (int)blockIdx.x) * BN;
  density_block(sm, n, npoint, phi, ld, D, rho, p0, keep);
}

// --------------------------------------------------------------- quadrature
// Without `blocks` the K range is every point (npoint_pad, chunks of `chunk`
// points); with it (screened plans) the K range is the list of 16-point
// blocks holding a kept point, npoint_pad = 16 x their count and `chunk` a
// multiple of 16 as before.

// n <= 64: each warp accumulates the whole upper triangle of 16 x 8 fragments
// over a chunk of its own; the B fragments of the second operand psi = phi are
// A fragments times the weights (A's rows g and g + 8 are B's columns of two
// fragments), so one set of loads feeds both.  Sums run over the points of a
// chunk and then over the chunks in order.
template <int RT, bool kSame>
__device__ __forceinline__ void quadrature_small_chunk(int n, int npoint_pad,
                                                       const double *__restrict__ phi,
                                                       const double *__restrict__ phib, long ld,
                                                       const double *__restrict__ wv, int chunk,
                                                       double *__restrict__ work,
                                                       const int *__restrict__ blocks, int ck) {
  constexpr int T = small_frags(RT);
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int s_begin = ck * (chunk / 8), s_end = min((ck + 1) * chunk, npoint_pad) / 8;
  if (s_begin >= s_end) return;
  double acc[T][4];
#pragma unroll
  for (int f = 0; f < T; ++f)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[f][c] = 0.0;
  // rows 16 i + g, 16 i + 8 + g of an operand at points p0 + q, p0 + q + 4
  auto load = [&](const double *x, long p0, double (&f)[RT][4]) {
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int r = 16 * i + g + 8 * (c & 1);
        f[i][c] = r < n ? __ldg(x + (long)r * ld + p0 + q + 4 * (c >> 1)) : 0.0;
      }
  };
#pragma unroll (RT <= 2 ? 4 : RT == 3 ? 2 : 1)
  for (int s = s_begin; s < s_end; ++s) {
    const long p0 = blocks ? (long)blocks[s >> 1] * BK + (s & 1) * 8 : 8L * s;
    const double w0 = __ldg(wv + p0 + q), w1 = __ldg(wv + p0 + q + 4);
    double a[RT][4], b[RT][4];
    load(phi, p0, a);
    if (!kSame) load(phib, p0, b);
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      b[i][0] = (kSame ? a[i][0] : b[i][0]) * w0;
      b[i][1] = (kSame ? a[i][1] : b[i][1]) * w0;
      b[i][2] = (kSame ? a[i][2] : b[i][2]) * w1;
      b[i][3] = (kSame ? a[i][3] : b[i][3]) * w1;
    }
    int f = 0;
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 2 * i; j < 2 * RT; ++j, ++f) {
        const double bf[2] = {b[j >> 1][j & 1], b[j >> 1][2 + (j & 1)]};
        dmma(acc[f], a[i], bf);
      }
  }
  double *out = work + (long)ck * (T * 128) + lane;
#pragma unroll
  for (int f = 0; f < T; ++f)
#pragma unroll
    for (int c = 0; c < 4; ++c) out[f * 128 + c * 32] = acc[f][c];
}

template <int RT>
__global__ void __launch_bounds__(NT)
quadrature_small_kernel(int n, int npoint_pad, const double *__restrict__ phi,
                        const double *__restrict__ phib, long ld,
                        const double *__restrict__ wv, int chunk, double *__restrict__ work,
                        const int *__restrict__ blocks) {
  const int ck = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (phi == phib)
    quadrature_small_chunk<RT, true>(n, npoint_pad, phi, phib, ld, wv, chunk, work, blocks, ck);
  else
    quadrature_small_chunk<RT, false>(n, npoint_pad, phi, phib, ld, wv, chunk, work, blocks, ck);
}

// Fragments of one warp in a diagonal tile of R row tiles (16 rows) and C = 2 R
// or 2 R - 1 column tiles (8 columns).  Row tile i has the C - 2 i fragments
// from column 2 i on; row tiles p and R - 1 - p together have twice L = C - R
// + 1, so warp 2 p takes the first L of row p and warp 2 p + 1 the rest of it
// and all of row R - 1 - p (for odd R the middle row is warp R - 1's alone):
// R warps of L fragments each.
struct DiagFrags {
  int r0, r1;      // row tiles of the fragments [0, split) and [split, count)
  int c0, c1;      // their first column tiles
  int split, count;
};
__device__ __forceinline__ DiagFrags diag_frags(int R, int C, int warp) {
  const int L = C - R + 1, p = warp >> 1, last = R - 1 - p;
  if (warp >= R) return DiagFrags{0, 0, 0, 0, 0, 0};
  if ((warp & 1) == 0) return DiagFrags{p, p, 2 * p, 2 * p, L, L};
  return DiagFrags{p, last, 2 * p + L, 2 * last, R - 1 - 2 * p, L};
}

// CTA `cta` of the plan: one tile of F over one chunk of the points, into its
// workspace slot.  Only the 16 x 8 fragments that hold an entry of the upper
// triangle within n are multiplied and written; they are skipped by branches
// around groups of instructions (a predicated-off DMMA still takes its slot in
// the pipe: masking single fragments gained nothing).
__device__ __forceinline__ void quadrature_block(QuadSmem &sm, int n, int npoint_pad,
                                                 const double *__restrict__ phi,
                                                 const double *__restrict__ phib, long ld,
                                                 const double *__restrict__ wv,
                                                 const QuadPlan &plan,
                                                 double *__restrict__ work,
                                                 const int *__restrict__ blocks, int cta) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int g = lane >> 2, q = lane & 3;
  int cls = 0;
  while (cta >= plan.first[cls + 1]) ++cls;
  const int local = cta - plan.first[cls], ck = local / plan.ntile[cls];
  const int chunk = plan.chunk[cls];
  int mb, nb;
  quad_tile(cls, local - ck * plan.ntile[cls], (n + BM - 1) / BM, mb, nb);
  const int mu0 = mb * BM, nu0 = nb * BN;
  const bool same = mb == nb && phi == phib;       // one operand tile serves both
  const int k_begin = ck * chunk;
  const int k_end = min(k_begin + chunk, npoint_pad);
  const int nstage = k_end > k_begin ? (k_end - k_begin) / BK : 0;
  const int ncol = (min(n - nu0, BN) + 7) / 8;     // live column tiles

  // copies of one stage: 128 rows x 16 points of each operand (8 x 16 bytes
  // per row) and the 16 weights; rows beyond n are zero filled
  auto load_stage = [&](int it) {
    const int kv = k_begin + it * BK;
    const int slot = it % NS, k0 = blocks ? blocks[kv / BK] * BK : kv;
#pragma unroll
    for (int i = 0; i < (BM * BK / 2) / NT; ++i) {
      const int e = t + NT * i, r = e / (BK / 2), c = (e % (BK / 2)) * 2;
      const bool va = mu0 + r < n, vb = nu0 + r < n;
      cp_async16(&sm.a[slot][r][c], phi + (va ? (long)(mu0 + r) * ld + k0 + c : 0), va);
      if (!same)
        cp_async16(&sm.b[slot][r][c], phib + (vb ? (long)(nu0 + r) * ld + k0 + c : 0), vb);
    }
    if (t < BK / 2) cp_async16(&sm.w[slot][2 * t], wv + k0 + 2 * t, true);
  };
  // one stage's turn: the stage's data is in, the next copies are issued (by
  // half of the warps before their products, by the other half of each
  // sub-partition's after the first ones, so that its pipe does not idle)
  auto begin_stage = [&](int it) {
    cp_async_wait<NS - 2>();
    __syncthreads();
    if (warp < 4) {
      if (it + NS - 1 < nstage) load_stage(it + NS - 1);
      cp_async_commit();
    }
  };
  auto mid_stage = [&](int it) {
    if (warp >= 4) {
      if (it + NS - 1 < nstage) load_stage(it + NS - 1);
      cp_async_commit();
    }
  };
#pragma unroll
  for (int i = 0; i < NS - 1; ++i) {
    if (i < nstage) load_stage(i);
    cp_async_commit();
  }
  double *out = work + (long)cta * (BM * BN);
  auto store = [&](int r, int c, const double(&v)[4]) {
    double *o = out + (16 * r + g) * BN + 8 * c + 2 * q;
    *reinterpret_cast<double2 *>(o) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2 *>(o + 8 * BN) = make_double2(v[2], v[3]);
  };

  if (mb == nb) {
    constexpr int F = 9;                           // most fragments of a warp (R = 8)
    const int R = (min(n - mu0, BM) + 15) / 16;
    const DiagFrags d = diag_frags(R, ncol, warp);
    double acc[F][4];
    int bo[F];                                     // row of the B tile of fragment f
#pragma unroll
    for (int f = 0; f < F; ++f) {
      bo[f] = 8 * (f < d.split ? d.c0 + f : d.c1 + f - d.split) + g;
      if (f >= d.count) bo[f] = g;
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[f][c] = 0.0;
    }
    for (int it = 0; it < nstage; ++it) {
      begin_stage(it);
      const int slot = it % NS;
      const double(*at)[LDA] = sm.a[slot];
      const double(*bt)[LDA] = same ? sm.a[slot] : sm.b[slot];
      const double *w = sm.w[slot];
#pragma unroll
      for (int kk = 0; kk < BK; kk += 8) {
        const double w0 = w[kk + q], w1 = w[kk + q + 4];
        const double *x0 = &at[16 * d.r0 + g][kk + q], *x1 = &at[16 * d.r1 + g][kk + q];
        const double a0[4] = {x0[0], x0[8 * LDA], x0[4], x0[8 * LDA + 4]};
        const double a1[4] = {x1[0], x1[8 * LDA], x1[4], x1[8 * LDA + 4]};
#pragma unroll
        for (int f3 = 0; f3 < F; f3 += 3) {
          if (f3 >= d.count) continue;             // warp-uniform
#pragma unroll
          for (int f = f3; f < f3 + 3; ++f) {
            const double b[2] = {bt[bo[f]][kk + q] * w0, bt[bo[f]][kk + q + 4] * w1};
            const bool lo = f < d.split;
            const double a[4] = {lo ? a0[0] : a1[0], lo ? a0[1] : a1[1], lo ? a0[2] : a1[2],
                                 lo ? a0[3] : a1[3]};
            dmma(acc[f], a, b);
          }
        }
        if (kk == 0) mid_stage(it);
      }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int f = 0; f < F; ++f)
      if (f < d.count) store(f < d.split ? d.r0 : d.r1, (bo[f] - g) / 8, acc[f]);
    return;
  }
  // off the diagonal: row tile `warp`, all column tiles, in groups of 4
  double acc[BN / 8][4];
#pragma unroll
  for (int j = 0; j < BN / 8; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.0;
  for (int it = 0; it < nstage; ++it) {
    begin_stage(it);
    const int slot = it % NS;
    const double(*bt)[LDA] = sm.b[slot];
    const double *w = sm.w[slot];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 8) {
      const double w0 = w[kk + q], w1 = w[kk + q + 4];
      const double *x = &sm.a[slot][16 * warp + g][kk + q];
      const double a[4] = {x[0], x[8 * LDA], x[4], x[8 * LDA + 4]};
#pragma unroll
      for (int j4 = 0; j4 < BN / 8; j4 += 4) {
        if (j4 >= ncol) continue;                  // uniform
#pragma unroll
        for (int j = j4; j < j4 + 4; ++j) {
          const double b[2] = {bt[8 * j + g][kk + q] * w0, bt[8 * j + g][kk + q + 4] * w1};
          dmma(acc[j], a, b);
        }
      }
      if (kk == 0) mid_stage(it);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int j = 0; j < BN / 8; ++j)
    if (j < ncol) store(warp, j, acc[j]);
}

__global__ void __launch_bounds__(NT, 1)
quadrature_kernel(int n, int npoint_pad, const double *__restrict__ phi,
                  const double *__restrict__ phib, long ld,
                  const double *__restrict__ wv, const QuadPlan plan,
                  double *__restrict__ work, const int *__restrict__ blocks) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  QuadSmem &sm = *reinterpret_cast<QuadSmem *>(smem_raw);
  quadrature_block(sm, n, npoint_pad, phi, phib, ld, wv, plan, work, blocks, blockIdx.x);
}

// Entries of all partial sums, in groups of 32 (a CTA of the reduction each).
__host__ __device__ inline long quad_entry_groups(int n) {
  if (n <= kSmallN) return 4L * small_frags(small_tiles(n));
  const long nblk = (n + BM - 1) / BM;
  return nblk * (nblk + 1) / 2 * (BM * BN / 32);
}

// Adds the chunks' partial sums in a fixed order and writes both triangles of
// F; a CTA owns 32 consecutive entries.  One thread per entry over all chunks
// took 54 us for H2O (592 dependent loads) and 35 us for C8H18.
// n <= 64: chunks in order, staged through shared memory by all 8 warps
// kRedRows at a time while warp 0 adds the rows staged before them.
// n > 64: 8 warps take chunks w, w + 8, ..., then the warps in order.
constexpr int kRedRows = 64;
struct ReduceSmem {
  double row[2][kRedRows][32];
};
__device__ __forceinline__ void quadrature_reduce_block(ReduceSmem &sm, int n,
                                                        const QuadPlan &plan,
                                                        const double *__restrict__ work,
                                                        double *__restrict__ F, long bx) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int mu, nu, nchunk;
  long stride;                          // doubles from one chunk's entry to the next's
  const double *w = work + lane;        // the entry in chunk 0
  if (n <= kSmallN) {
    const int rt = small_tiles(n), c = (int)(bx & 3);
    int f = (int)(bx >> 2), i = 0;
    while (f >= 2 * (rt - i)) f -= 2 * (rt - i++);
    mu = 16 * i + (lane >> 2) + 8 * (c >> 1);
    nu = 8 * (2 * i + f) + 2 * (lane & 3) + (c & 1);
    nchunk = plan.nch[0];
    stride = 128L * small_frags(rt);
    w += bx * 32;
  } else {
    constexpr int G = BM * BN / 32;     // groups per tile
    int tile = (int)(bx / G), cls = 0;
    const int e = (int)(bx % G) * 32 + lane;
    while (tile >= plan.ntile[cls]) tile -= plan.ntile[cls++];
    int mb, nb;
    quad_tile(cls, tile, (n + BM - 1) / BM, mb, nb);
    mu = mb * BM + e / BN;
    nu = nb * BN + e % BN;
    nchunk = plan.nch[cls];
    stride = (long)plan.ntile[cls] * BM * BN;
    w += (long)(plan.first[cls] + tile) * BM * BN + (bx % G) * 32;
  }
  const bool live = mu <= nu && nu < n;
  if (!__syncthreads_or(live)) return;
  double s = 0.0;
  if (n <= kSmallN) {
    constexpr int PER = kRedRows / kWarps;
    double r[PER];
    auto fetch = [&](int k0) {  // rows warp, warp + 8, ... of a round
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int k = k0 + warp + kWarps * i;
        r[i] = k < nchunk ? __ldg(w + k * stride) : 0.0;
      }
    };
    fetch(0);
    for (int k0 = 0, buf = 0; k0 < nchunk; k0 += kRedRows, buf ^= 1) {
#pragma unroll
      for (int i = 0; i < PER; ++i) sm.row[buf][warp + kWarps * i][lane] = r[i];
      __syncthreads();
      if (k0 + kRedRows < nchunk) fetch(k0 + kRedRows);
      if (warp == 0) {
#pragma unroll 16
        for (int i = 0; i < kRedRows; ++i) s += sm.row[buf][i][lane];
      }
    }
  } else {
    if (live) {
#pragma unroll 4
      for (int k = warp; k < nchunk; k += kWarps) s += __ldg(w + k * stride);
    }
    sm.row[0][warp][lane] = s;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int k = 1; k < kWarps; ++k) s += sm.row[0][k][lane];
    }
  }
  if (warp == 0 && live) {
    F[(long)mu * n + nu] = s;
    F[(long)nu * n + mu] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(NT)
quadrature_reduce_kernel(int n, const QuadPlan plan, const double *__restrict__ work,
                         double *__restrict__ F) {
  __shared__ ReduceSmem sm;
  quadrature_reduce_block(sm, n, plan, work, F, blockIdx.x);
}

__global__ void combine_weights_kernel(int npoint, const double *__restrict__ wb,
                                       const double *__restrict__ w, double q,
                                       const double *__restrict__ v,
                                       const double *__restrict__ vext,
                                       double *__restrict__ wv) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npoint) return;
  double pot = v ? q * v[p] : 0.0;
  if (vext) pot += vext[p];
  wv[p] = wb[p] * w[p] * pot;
}

// Scratch of one call: stream-ordered, so safe with any streams and threads, and
// a part of the graph when the stream is capturing.  From a pool of the
// library's own per device, which keeps up to 64 MB between calls until the last
// Fock plan goes (trim_call_scratch).  The default pool returns everything to the
// driver at each synchronisation, and so does one that keeps less than the blocks
// it grows by (with 16 MB the C12H26 build took 14.6 ms instead of 13.5).
struct ScratchPools {
  std::mutex lock;
  std::map<int, cudaMemPool_t> of;  // device -> pool
};
ScratchPools &scratch_pools() {
  static ScratchPools *p = new ScratchPools;  // outlives every static plan
  return *p;
}

cudaError_t call_scratch(void **p, size_t bytes, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  ScratchPools &pools = scratch_pools();
  std::lock_guard<std::mutex> hold(pools.lock);
  cudaMemPool_t &pool = pools.of[dev];
  if (!pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    // neither call touches a stream: allowed while some stream is capturing
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaMemPool_t made = nullptr;
    e = cudaMemPoolCreate(&made, &props);
    unsigned long long keep = 64ull << 20;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    pool = made;
  }
  return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

inline int pad_points(int npoint) { return ((npoint + BN - 1) / BN) * BN; }

}  // namespace

size_t density_workspace_bytes(int, int) { return 0; }

cudaError_t launch_density_f64(int n, int npoint, const double *phi, long ld,
                               const double *D, double *rho, cudaStream_t s,
                               const int *groups, int ngroup, const int *keep) {
  if (npoint <= 0) return cudaSuccess;
  int blocks = (npoint + BN - 1) / BN;
  if (groups) {
    // groups without a kept point are not computed: their rho is 0
    cudaError_t e = cudaMemsetAsync(rho, 0, (size_t)npoint * sizeof(double), s);
    if (e != cudaSuccess) return e;
    blocks = ngroup;
    if (blocks == 0) return cudaSuccess;
  }
  if (n <= kSmallN) {
    // as many CTAs as are resident (registers): each loads D once
    const int rt = small_tiles(n), grid = std::min(blocks, 148 * (rt == 1 ? 4 : 1));
    switch (rt) {
      case 1: density_small_kernel<1><<<grid, NT, 0, s>>>(n, npoint, phi, ld, D, rho, groups, blocks, keep); break;
      case 2: density_small_kernel<2><<<grid, NT, 0, s>>>(n, npoint, phi, ld, D, rho, groups, blocks, keep); break;
      case 3: density_small_kernel<3><<<grid, NT, 0, s>>>(n, npoint, phi, ld, D, rho, groups, blocks, keep); break;
      default: density_small_kernel<4><<<grid, NT, 0, s>>>(n, npoint, phi, ld, D, rho, groups, blocks, keep);
    }
    return cudaGetLastError();
  }
  cudaError_t e = cudaFuncSetAttribute(density_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kDensSmem);
  if (e != cudaSuccess) return e;
  void *fold = nullptr;
  const size_t count = density_fold_doubles(n);
  e = call_scratch(&fold, count * sizeof(double), s);
  if (e != cudaSuccess) return e;
  density_fold_kernel<<<(unsigned)((count + NT - 1) / NT), NT, 0, s>>>(n, D, (double *)fold);
  density_kernel<<<blocks, NT, kDensSmem, s>>>(n, npoint, phi, ld, (const double *)fold, rho,
                                               groups, keep);
  e = cudaGetLastError();
  const cudaError_t ef = cudaFreeAsync(fold, s);
  return e != cudaSuccess ? e : ef;
}

void trim_call_scratch() {
  ScratchPools &pools = scratch_pools();
  std::lock_guard<std::mutex> hold(pools.lock);
  for (auto &p : pools.of)
    if (p.second) cudaMemPoolTrimTo(p.second, 0);
}

size_t density_fold_doubles(int n) { return n > kSmallN ? (size_t)n * fold_ld(n) : 0; }

QuadPlan quad_plan(int n, int npad) { return quad_plan_slots(n, npad, quad_default_slots(n)); }

int quad_plan_items(int n, const QuadPlan &p) {
  return n <= kSmallN ? (p.nch[0] + kWarps - 1) / kWarps : p.first[4];
}

// the split-K quadrature and the sum of its chunks
cudaError_t quadrature_launch(const QuadPlan &plan, int n, int npad, const double *phi,
                              const double *phib, long ld, const double *wv, double *work,
                              double *F, cudaStream_t s, const int *blocks = nullptr) {
  cudaError_t e;
  if (n <= kSmallN) {
    auto kern = small_tiles(n) == 1   ? quadrature_small_kernel<1>
                : small_tiles(n) == 2 ? quadrature_small_kernel<2>
                : small_tiles(n) == 3 ? quadrature_small_kernel<3>
                                      : quadrature_small_kernel<4>;
    // four warps per CTA: the chunks spread over all SMs
    kern<<<(plan.nch[0] + 3) / 4, 128, 0, s>>>(n, npad, phi, phib, ld, wv, plan.chunk[0], work,
                                              blocks);
  } else {
    e = cudaFuncSetAttribute(quadrature_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kQuadSmem);
    if (e != cudaSuccess) return e;
    quadrature_kernel<<<plan.first[4], NT, kQuadSmem, s>>>(n, npad, phi, phib, ld, wv, plan, work,
                                                          blocks);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  quadrature_reduce_kernel<<<(unsigned)quad_entry_groups(n), NT, 0, s>>>(n, plan, work, F);
  return cudaGetLastError();
}

size_t quadrature_workspace_bytes(int n, int npoint) {
  return quad_workspace_doubles(n, pad_points(npoint)) * sizeof(double);
}

cudaError_t launch_quadrature_f64(int n, int npoint, const double *phi, long ld,
                                  const double *wv, double *F, double *work,
                                  cudaStream_t s, const double *phib, const int *blocks,
                                  int nblock) {
  if (!phib) phib = phi;
  if (n <= 0) return cudaSuccess;
  // screened: the K range is the listed 16-point blocks
  const int npad = blocks ? nblock * BK : pad_points(npoint);
  if (npad == 0) return cudaMemsetAsync(F, 0, (size_t)n * n * sizeof(double), s);
  return quadrature_launch(quad_plan(n, npad), n, npad, phi, phib, ld, wv, work, F, s, blocks);
}

// -------------------------------------------------------------- batches
// Persistent batched launches: CTAs take (molecule, tile) items from a device
// work queue until it is empty.  Item i may be taken once *posted > i (the
// batch posts its items when it is built; a producer that never posts makes
// the wait run out): the wait is bounded by q.timeout_ns of %globaltimer,
// after which the CTA records kDeviceTimeout in *q.status and stops.
namespace {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ int queue_pop(const BatchQueue &q) {
  const int i = atomicAdd(q.head, 1);
  if (i >= q.nitems) return -1;
  const volatile int *posted = q.posted;
  if (*posted > i) return i;
  const unsigned long long t0 = globaltimer_ns();
  for (unsigned it = 1;; ++it) {
    if (*posted > i) return i;
    if ((it & 63) == 0 && globaltimer_ns() - t0 > q.timeout_ns) {
      atomicExch(q.status, kDeviceTimeout);
      return -1;
    }
  }
}

// the CTA's next item (all threads), -1 when the queue is done
__device__ __forceinline__ int cta_pop(const BatchQueue &q, int *slot) {
  if (threadIdx.x == 0) *slot = queue_pop(q);
  __syncthreads();
  const int w = *slot;
  __syncthreads();
  return w;
}

// D' of every molecule (blockIdx.y)
__global__ void __launch_bounds__(NT)
density_fold_batch_kernel(const DensBatchArg *__restrict__ args) {
  const DensBatchArg a = args[blockIdx.y];
  if (a.n <= kSmallN) return;
  const long total = (long)a.n * fold_ld(a.n);
  for (long e = (long)blockIdx.x * NT + threadIdx.x; e < total; e += (long)gridDim.x * NT)
    density_fold_body(a.n, a.D, a.fold, e);
}

__global__ void __launch_bounds__(NT, 1)
density_batch_kernel(const DensBatchArg *__restrict__ args, BatchQueue q) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  DensSmem &sm = *reinterpret_cast<DensSmem *>(smem_raw);
  __shared__ int slot;
  for (;;) {
    const int w = cta_pop(q, &slot);
    if (w < 0) break;
    const int4 it = q.items[w];
    const DensBatchArg a = args[it.x];
    if (a.n <= kSmallN) {  // group it.y alone
      density_small_any(a.n, a.npoint, a.phi, a.ld, a.D, a.rho, nullptr, it.y + 1, it.y, 1,
                        a.keep);
      continue;
    }
    density_block(sm, a.n, a.npoint, a.phi, a.ld, a.fold, a.rho, it.y * BN, a.keep);
  }
}

__global__ void __launch_bounds__(NT, 1)
quadrature_batch_kernel(const QuadBatchArg *__restrict__ args, BatchQueue q) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  QuadSmem &sm = *reinterpret_cast<QuadSmem *>(smem_raw);
  __shared__ int slot;
  for (;;) {
    const int w = cta_pop(q, &slot);
    if (w < 0) break;
    const int4 it = q.items[w];
    const QuadBatchArg a = args[it.x];
    if (a.n <= kSmallN) {  // chunks 8 it.y .. 8 it.y + 7, one per warp
      const int ck = kWarps * it.y + (threadIdx.x >> 5), chunk = a.plan.chunk[0];
      switch (small_tiles(a.n)) {
        case 1: quadrature_small_chunk<1, true>(a.n, a.npad, a.phi, a.phi, a.ld, a.wv, chunk, a.work, a.blocks, ck); break;
        case 2: quadrature_small_chunk<2, true>(a.n, a.npad, a.phi, a.phi, a.ld, a.wv, chunk, a.work, a.blocks, ck); break;
        case 3: quadrature_small_chunk<3, true>(a.n, a.npad, a.phi, a.phi, a.ld, a.wv, chunk, a.work, a.blocks, ck); break;
        default: quadrature_small_chunk<4, true>(a.n, a.npad, a.phi, a.phi, a.ld, a.wv, chunk, a.work, a.blocks, ck);
      }
      continue;
    }
    quadrature_block(sm, a.n, a.npad, a.phi, a.phi, a.ld, a.wv, a.plan, a.work, a.blocks, it.y);
  }
}

// F of every molecule from its chunk partials (blockIdx.y = molecule)
__global__ void __launch_bounds__(NT)
quadrature_reduce_batch_kernel(const QuadBatchArg *__restrict__ args) {
  __shared__ ReduceSmem sm;
  const QuadBatchArg a = args[blockIdx.y];
  const long nb = quad_entry_groups(a.n);
  for (long b = blockIdx.x; b < nb; b += gridDim.x)
    quadrature_reduce_block(sm, a.n, a.plan, a.work, a.F, b);
}

// wv of every molecule (blockIdx.y), zero padded to its npad points
__global__ void combine_weights_batch_kernel(const WeightBatchArg *__restrict__ args, double q) {
  const WeightBatchArg a = args[blockIdx.y];
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < a.npad; p += gridDim.x * blockDim.x)
    a.wv[p] = p < a.npoint ? a.wb[p] * a.w[p] * (q * a.v[p]) : 0.0;
}

}  // namespace

cudaError_t launch_density_batch(const DensBatchArg *args, int nfold, const BatchQueue &q,
                                 int grid, cudaStream_t s) {
  if (q.nitems == 0) return cudaSuccess;
  if (nfold > 0) density_fold_batch_kernel<<<dim3(64, nfold), NT, 0, s>>>(args);
  cudaError_t e = cudaFuncSetAttribute(density_batch_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kDensSmem);
  if (e != cudaSuccess) return e;
  density_batch_kernel<<<grid, NT, kDensSmem, s>>>(args, q);
  return cudaGetLastError();
}

cudaError_t launch_quadrature_batch(const QuadBatchArg *args, const BatchQueue &q, int grid,
                                    cudaStream_t s) {
  if (q.nitems == 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(quadrature_batch_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kQuadSmem);
  if (e != cudaSuccess) return e;
  quadrature_batch_kernel<<<grid, NT, kQuadSmem, s>>>(args, q);
  return cudaGetLastError();
}

cudaError_t launch_quadrature_reduce_batch(const QuadBatchArg *args, int nmol, cudaStream_t s) {
  if (nmol == 0) return cudaSuccess;
  quadrature_reduce_batch_kernel<<<dim3(148 * 4, nmol), NT, 0, s>>>(args);
  return cudaGetLastError();
}

cudaError_t launch_combine_weights_batch(const WeightBatchArg *args, int nmol, double q,
                                         cudaStream_t s) {
  if (nmol == 0) return cudaSuccess;
  combine_weights_batch_kernel<<<dim3(148, nmol), 256, 0, s>>>(args, q);
  return cudaGetLastError();
}

// ------------------------------------------------------ FP64 point screening
namespace {

// keep[p] = 1 when |wb w| max_mu phi_mu(p)^2 >= tol (the test of the int8
// plans: a dropped point changes an element of F by at most tol |v(p)|).
__global__ void screen_points_kernel(const double *__restrict__ phi, long ld, int n, int npoint,
                                     const double *__restrict__ wb, const double *__restrict__ w,
                                     double tol, int *__restrict__ keep) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npoint) return;
  double mx = 0.0;
  for (int mu = 0; mu < n; ++mu) mx = fmax(mx, fabs(__ldg(phi + (long)mu * ld + p)));
  const double t = fabs(wb[p] * w[p]);
  keep[p] = (t * mx) * mx >= tol ? 1 : 0;
}

// flags[b] = 1 when block b of `span` points holds a kept point
__global__ void screen_blocks_kernel(const int *__restrict__ keep, int npoint, int span,
                                     int nb, int *__restrict__ flags) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  int any = 0;
  for (int i = b * span; i < min((b + 1) * span, npoint); ++i) any |= keep[i];
  flags[b] = any;
}

}  // namespace

cudaError_t launch_fp64_screening(int n, int npoint, const double *phi, long ld, const double *wb,
                                  const double *w, double tol, int *keep, int *block_flags,
                                  int *group_flags, cudaStream_t s) {
  if (npoint <= 0) return cudaSuccess;
  screen_points_kernel<<<(npoint + 255) / 256, 256, 0, s>>>(phi, ld, n, npoint, wb, w, tol,
                                                           keep);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int nb = (npoint + BK - 1) / BK, ng = (npoint + BN - 1) / BN;
  screen_blocks_kernel<<<(nb + 255) / 256, 256, 0, s>>>(keep, npoint, BK, nb, block_flags);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  screen_blocks_kernel<<<(ng + 255) / 256, 256, 0, s>>>(keep, npoint, BN, ng, group_flags);
  return cudaGetLastError();
}

cudaError_t launch_combine_weights(int npoint, const double *wb, const double *w,
                                   double q, const double *v, const double *vext,
                                   double *wv, cudaStream_t s) {
  if (npoint <= 0) return cudaSuccess;
  combine_weights_kernel<<<(npoint + 255) / 256, 256, 0, s>>>(npoint, wb, w, q, v,
                                                             vext, wv);
  return cudaGetLastError();
}

}  // namespace napmo

// ===========================================================================
// Allocation-free quadrature: napmo_gpu_quadrature_noalloc.
//
// Some callers of this library cannot allocate device memory while they call
// it: host applications that reserve and budget the whole memory of a GPU at
// start-up and hand plugins no allocator (a cudaMalloc from the plugin would
// take memory the host has already promised elsewhere, or fail), and callers
// that must not let an allocation stall or synchronise the device in the
// middle of their own work.  For them this entry point runs the same split-K
// quadrature kernels as napmo_gpu_quadrature, with the per-chunk partial tiles
// kept in `g_quad_scratch`, a fixed 16 MiB array compiled into the library:
// every GPU that loads libnapmo holds it until the process exits.
//
// Limit: the partial tiles of one chunk must fit, so n <= 1920 basis
// functions; larger n is rejected with an error before anything is launched.
// The chunk count is lowered to fit the array (fewer, longer chunks), so the
// result can differ from napmo_gpu_quadrature in the last bits (different
// summation grouping); it is deterministic from call to call.
//
// Address: every call looks up the device address of the array with
// cudaGetSymbolAddress, with the caller's device current, and passes it to the
// kernels (in host code the array's name is only a host-side stand-in).  The
// lookup allocates nothing; doing it per call rather than caching it keeps the
// address right under any context and after a device reset.  The first call
// on a device may load the library's device code there: make it before any
// stream capture.
//
// Inputs: phi, psi and wv are read with 16-byte loads up to npoint rounded up
// to 128, so they must be 16-byte aligned, ld even, and wv zero padded to that
// length (napmo_gpu_combine_weights writes it so).  npoint = 0 gives F = 0.
//
// Sharing: the array is shared by all calls and keeps the previous call's
// contents; nothing in it needs to start at zero (each chunk overwrites its
// own tiles before they are added).  Calls that overlap on the GPU (different
// streams, or different host threads without ordering) race on the array and
// must be serialised by the caller.
// ===========================================================================
namespace napmo {
namespace {

constexpr size_t kNoAllocScratchDoubles = size_t(2) << 20;  // 16 MiB
__device__ __align__(256) double g_quad_scratch[kNoAllocScratchDoubles];

// Device address of g_quad_scratch in the current context.
int scratch_address(double **out) {
  void *p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_quad_scratch);
  if (e != cudaSuccess)
    return set_error(kCudaError, std::string("cudaGetSymbolAddress(quadrature scratch): ") +
                                     cudaGetErrorString(e));
  *out = static_cast<double *>(p);
  return kOk;
}

}  // namespace
}  // namespace napmo

extern "C" {

// F[mu][nu] = sum_p phi[mu][p] wv[p] psi[nu][p] (psi = phi when null), upper
// triangle mirrored, like napmo_gpu_quadrature, without allocating: the
// split-K scratch lives in a fixed 16 MiB device array (n <= 1920).  See the
// block comment above for the address lookup, the input contract and the
// sharing rules.
int napmo_gpu_quadrature_noalloc(int n, int npoint, const double *phi, const double *psi,
                                 long ld, const double *wv, double *F, void *stream) {
  using namespace napmo;
  clear_error();
  if (n <= 0 || npoint < 0) return set_error(kInvalidArgument, "n must be positive, npoint >= 0");
  const int npad = pad_points(npoint);
  if (ld < npad || ld % 2 != 0)
    return set_error(kInvalidArgument, "ld must be even and >= npoint rounded up to 128");
  const long nblk = (n + BM - 1) / BM;
  const size_t per_chunk = (size_t)(nblk * (nblk + 1) / 2) * BM * BN;
  if (per_chunk > kNoAllocScratchDoubles)
    return set_error(kInvalidArgument,
                     "napmo_gpu_quadrature_noalloc: n = " + std::to_string(n) +
                         " exceeds the 16 MiB fixed scratch (at most 1920 basis functions)");
  cudaStream_t s = (cudaStream_t)stream;
  if (npoint == 0) {  // empty grid: F = 0 (a memset allocates nothing)
    const cudaError_t e = cudaMemsetAsync(F, 0, (size_t)n * n * sizeof(double), s);
    if (e != cudaSuccess) return set_error(kCudaError, std::string("memset F: ") + cudaGetErrorString(e));
    return kOk;
  }
  double *scratch = nullptr;
  int st = scratch_address(&scratch);
  if (st != kOk) return st;
  // the launch policy's split, capped by the fixed array
  int slots = quad_default_slots(n);
  if (n > kSmallN) slots = std::min(slots, (int)(kNoAllocScratchDoubles / (BM * BN)));
  static_assert(4 * 148 * 128 * small_frags(kSmallN / 16) <= (int)kNoAllocScratchDoubles,
                "the small molecules' partial sums fit the fixed array");
  const cudaError_t e = quadrature_launch(quad_plan_slots(n, npad, slots), n, npad, phi,
                                          psi ? psi : phi, ld, wv, scratch, F, s);
  if (e != cudaSuccess) return set_error(kCudaError, std::string("quadrature: ") + cudaGetErrorString(e));
  return kOk;
}

}  // extern "C"

// Float64 scaled Gram (X / s)^H (X / s) of a Casorati matrix on the float64
// tensor cores (mma.sync m8n8k4, the only float64 MMA).
//
// The complex rows are read as real rows Y of 2T columns (re, im interleaved),
// so D = Y^T Y holds the complex Gram: G[i][j] = D[2i][2j] + D[2i+1][2j+1] +
// j (D[2i][2j+1] - D[2i+1][2j]).  Both fragments of m8n8k4 have the same layout
// for a symmetric product (lane l: Y[k + l % 4][8 b + l / 4] for column block
// b), so one staged copy of the rows serves both.
//
// Bound: the float64 pipe, T (2T + 1) multiply-adds per row at 64 per clock and
// SM (37 TFLOP/s measured).  A warp owns a 32 x 32 block of D's upper triangle in
// registers; small blocks waste little on the triangle's edge and on the last
// columns (T = 200: 91 blocks, 93 k of 80 k products needed), and eight fragment
// loads feed sixteen MMAs.  A CTA's sixteen warps share each staged group of 8 or
// 16 rows, converted to scaled doubles once; the CTAs of a slice read the same
// rows at the same time (one HBM read, L2 for the rest).
// Measured against gram_simt (one B200): 524288 x 200 complex64 8.71 -> 4.03 ms,
// 200000 x 400 9.10 -> 5.44 ms, 259200 x 75 1.22 -> 0.34 ms, 65536 x 16 118 -> 49 us;
// 524288 x 200 complex128 12.5 -> 3.95 ms.  Errors against float64 matmul are the
// same or smaller.
#pragma once

#include "clutter.cuh"

namespace rcb {
namespace gramf64 {

constexpr int kTile = 32;      // real columns of a warp's output tile (4 x 4 MMA blocks)
constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kMaxFrames = 512;
constexpr int kLoads = 8;      // samples a thread prefetches per stage

struct Params {
  size_t rows;
  int nt;
  int blocks;      // 32-column blocks of Y
  int tiles;       // upper-triangle tiles
  int units;       // CTAs that share a row slice; each takes up to kWarps tiles
  int slices;      // row slices
  int pitch;       // doubles between staged rows
  const double* scale;
  double* upper;
};

// Doubles between staged rows: 4 mod 16, so that the four rows of a fragment
// load lie in distinct groups of eight banks.
__host__ __device__ inline int row_pitch(int blocks) { return blocks * kTile + 4; }
__host__ __device__ inline int stage_rows(int nt) { return nt <= 256 ? 16 : 8; }

template <typename IN, int ROWS>
__global__ void __launch_bounds__(kThreads, 1) gram_dmma(const IN* __restrict__ x, const Params p) {
  extern __shared__ __align__(16) double stage[];  // [2][ROWS][pitch]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int unit = blockIdx.x % p.units, slice = blockIdx.x / p.units;
  const int first = int((long long)unit * p.tiles / p.units), last = int((long long)(unit + 1) * p.tiles / p.units);
  // Few tiles: `parts` warps share one, each taking every parts-th four rows.
  const int parts = max(1, min(ROWS / 4, kWarps / (last - first)));
  const int mine = first + warp / parts, part = warp % parts;
  const bool active = mine < last;
  int ti = 0, tj = 0;
  if (active) {
    int t = mine;
    while (t >= p.blocks - ti) {
      t -= p.blocks - ti;
      ++ti;
    }
    tj = ti + t;
  }
  const size_t per = ((p.rows + p.slices - 1) / p.slices + ROWS - 1) / ROWS * ROWS;
  const size_t r0 = size_t(slice) * per, r1 = min(p.rows, r0 + per);
  const double s = *p.scale > 0.0 ? 1.0 / *p.scale : 1.0;
  // Warp w stages row w % ROWS, columns lane, lane + 32 (kWarps / ROWS), ...
  constexpr int kShare = kWarps / ROWS, kSteps = ROWS / 4;
  const int srow = warp % ROWS, scol = 32 * (warp / ROWS) + lane;
  IN next[kLoads];
  auto fetch = [&](size_t base) {
    const size_t r = base + srow;
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int c = scol + 32 * kShare * i;
      next[i] = r < r1 && c < p.nt ? x[r * size_t(p.nt) + c] : IN{};
    }
  };
  auto store = [&](double* buf, int i) {
    const int c = scol + 32 * kShare * i;
    if (c < p.nt)
      *reinterpret_cast<double2*>(buf + srow * p.pitch + 2 * c) =
          make_double2(double(next[i].x) * s, double(next[i].y) * s);
  };
  for (int i = threadIdx.x; i < 2 * ROWS * p.pitch; i += kThreads) stage[i] = 0.0;
  double acc[4][4][2] = {};
  fetch(r0);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kLoads; ++i) store(stage, i);
  fetch(r0 + ROWS);
  __syncthreads();
  int cur = 0;
  for (size_t base = r0; base < r1; base += ROWS) {
    const double* buf = stage + cur * ROWS * p.pitch;
    double* other = stage + (cur ^ 1) * ROWS * p.pitch;
    const double* pa = buf + q * p.pitch + ti * kTile + g;
    const double* pb = buf + q * p.pitch + tj * kTile + g;
    // The next rows are converted and stored between the MMAs, so that the
    // float64 pipe does not wait for the staging.
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      if (active && k % parts == part) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          a[i] = pa[4 * k * p.pitch + 8 * i];
          b[i] = pb[4 * k * p.pitch + 8 * i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j >= i) clutter::dmma_f64(acc[i][j][0], acc[i][j][1], a[i], b[j], acc[i][j][0], acc[i][j][1]);
        if (ti != tj) {  // below the diagonal: off-diagonal tiles only
#pragma unroll
          for (int i = 1; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < i; ++j)
              clutter::dmma_f64(acc[i][j][0], acc[i][j][1], a[i], b[j], acc[i][j][0], acc[i][j][1]);
        }
      }
#pragma unroll
      for (int i = 0; i < kLoads / kSteps; ++i) store(other, k * (kLoads / kSteps) + i);
    }
    fetch(base + 2 * ROWS);
    __syncthreads();
    cur ^= 1;
  }
  if (!active) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // Rows m = 2 fi (even g) and 2 fi + 1 (odd g) of frames fi sit in partner lanes.
      const double o0 = __shfl_xor_sync(0xffffffffu, acc[i][j][0], 4);
      const double o1 = __shfl_xor_sync(0xffffffffu, acc[i][j][1], 4);
      const int fi = (ti * kTile + 8 * i + g) / 2, fj = (tj * kTile + 8 * j) / 2 + q;
      if ((g & 1) || (ti == tj && j < i) || fi > fj || fj >= p.nt) continue;
      const double re = acc[i][j][0] + o1, im = acc[i][j][1] - o0;
      double* u = p.upper + 2 * (size_t(fi) * p.nt + fj);
      atomicAdd(u, re);
      atomicAdd(u + 1, im);
      // The finish pass averages both triangles inside its diagonal tiles.
      if (fi != fj && fi / clutter::kGramTile == fj / clutter::kGramTile) {
        double* l = p.upper + 2 * (size_t(fj) * p.nt + fi);
        atomicAdd(l, re);
        atomicAdd(l + 1, -im);
      }
    }
  }
}

}  // namespace gramf64
}  // namespace rcb

// tile_types.h -- plain descriptors shared by host code and the tile kernels.
#pragma once

#include <cuda_runtime.h>

#include "sht_internal.h"

namespace sht {

// One matrix dimension of the contraction as a list of tensor modes.
struct ModeMap {
  int n;                 // number of tensor modes forming this matrix dimension
  int x[kMaxOrder];      // mode index in the first operand (A for rows and k, B for cols)
  int y[kMaxOrder];      // mode index in the second (C for rows and cols, B for k)
};

struct TileMaps {
  ModeMap row, kk, col;
  int oA, oB, oC;
};

template <typename T>
struct TileScalars {
  T alpha, beta;
  int beta_zero;   // beta is +0.0: C is not read
  int alpha_zero;  // alpha is +0.0: products skipped
};

// Tile shapes of the FP64 kernel: the most rows and columns of a tile (at most 64 each).
constexpr int kRingShapes = 4;
__host__ __device__ constexpr int ring_tm(int s) { return s & 2 ? 32 : 64; }
__host__ __device__ constexpr int ring_tn(int s) { return s & 1 ? 32 : 64; }
// number of tiles along an extent, and their size (the last tile may be smaller)
__host__ __device__ __forceinline__ int ring_ntiles(int ext, int t) { return (ext + t - 1) / t; }
__host__ __device__ __forceinline__ int ring_step(int ext, int nt) { return (((ext + nt - 1) / nt) + 7) & ~7; }

// Cost of one C block per unit of contracted extent in a tile shape, in products: what the tensor
// pipe runs (the tile's fragments of 8x8, and four times the busiest warp's, averaged: a tile
// waits for its busiest warp, but another CTA fills the gap), the operand copies, and a fixed
// cost per tile.
__host__ __device__ inline float shape_cost(int m, int n, int sh) {
  const int ntr = ring_ntiles(m, ring_tm(sh)), ntc = ring_ntiles(n, ring_tn(sh));
  const int fr = ring_step(m, ntr) / 8, fc = ring_step(n, ntc) / 8;
  const float busiest = 4.0f * (float)(((fr + 1) / 2) * ((fc + 1) / 2));
  return (float)ntr * (float)ntc * (32.0f * ((float)(fr * fc) + busiest) + 64.0f * (float)(fr + fc) + 512.0f);
}
__host__ __device__ inline int model_shape(int m, int n) {
  float best = 3.0e38f;
  int bi = 0;
  for (int s = 0; s < kRingShapes; ++s) {
    const float c = shape_cost(m, n, s);
    if (c < best) { best = c; bi = s; }
  }
  return bi;
}

// Size class of a C block in the autotuner's table: ceil(log2) of its rows, columns and mean contracted
// extent, 32 values each.
__host__ __device__ inline int ilog2_up(long long v) {
  int b = 0;
  while (b < 31 && (1LL << b) < v) ++b;
  return b;
}
__host__ __device__ inline int class_index(int m, int n, long long kavg) {
  return (ilog2_up(m) * 32 + ilog2_up(n)) * 32 + ilog2_up(kavg > 0 ? kavg : 1);
}

// One block pair of a plan as the FP64 kernel reads it: where its blocks start, the contracted extent
// and the strides of linear addressing (tile_ring.cuh).  Built once per pair; every tile of the pair's
// C block reads it.
struct PairRec {
  long long offA, offB;
  int K, rsA, ksA, rsB, ksB, ia, ib, pad;
};
static_assert(sizeof(PairRec) == 48, "read in 16-byte units");

// One tile of a work list: C block, first row and column, rows | columns << 16.
__host__ __device__ __forceinline__ int4 ring_item(int c, int tile, int m, int n, int tm, int tn) {
  const int ntr = ring_ntiles(m, tm), sr = ring_step(m, ntr), sc = ring_step(n, ring_ntiles(n, tn));
  const int r0 = tile % ntr * sr, c0 = tile / ntr * sc;
  const int mt = m - r0 < sr ? m - r0 : sr, nt = n - c0 < sc ? n - c0 : sc;
  return make_int4(c, r0, c0, mt | nt << 16);
}

// Device pointers and scalars of one block-sparse execute (plain and batched forms).
struct SparseArgs {
  TileMaps mp;
  TileScalars<double> sc;
  const double* A; const long long* offA; const int* dimsA;
  const double* B; const long long* offB; const int* dimsB;
  double* C; const long long* offC; const int* dimsC;
  const int* pair_a; const int* pair_b; const int* pstart;
  const PairRec* recs;  // the FP64 forms (null in a split plan)
};

}  // namespace sht

// linear.cu -- operands whose free or contracted modes lie apart, copied block by block into an order
// that the FP64 tile kernel's linear copies read.
//
// The tile kernel reads a block in place when its free modes and its contracted modes each follow one
// another in memory (element (row, k) at row * rs + k * ks with rs or ks 1).  Other blocks it can only
// gather element by element, once for every tile that uses them, mostly a 32-byte sector for 8 bytes.
// Where the blocks are used more than once, the execute writes the whole operand anew first: block b
// stays at its offset, its elements in the order (row + m * k), or (k + K * row) when the contracted
// index's first mode is the block's fastest, so that the reads run along memory too.
// Measured, an execute with the pass against one with gathers: abdc,cdij->abij (268 GFLOP, 486 pairs) 10.1
// and 20.4 ms (13.5 ms for a tile kernel over operands that were all copied into matrix form); ilj,lk->ijk
// over 20 blocks of 5 to 15 per mode (16,349 pairs) 178 and 347 us, of it the pass 17 us (2.7M elements,
// 43 MB: small blocks, bound by a warp's chain of loads rather than by memory).
#include <algorithm>
#include <cmath>

#include "contract.h"
#include "device_common.cuh"

namespace sht {

constexpr int kLinearFast = 128, kLinearSlow = 16;  // a warp's turn: this many fast by slow indices of a block

struct LinearArgs {
  const double* src; double* dst;
  const long long* off; const int* dims;
  long long fturns, sturns;             // turns of the largest block along the fast and the slow index
  int order, nfast, nslow;              // modes of the written order's fast and slow index
  int fast[kMaxOrder], slow[kMaxOrder];
};
struct LinearPair {
  LinearArgs x[2];
  long long turns0, turns;  // of x[0], of both
};

// i / e by the rounded-up reciprocal 2^32 / e: at most one too large for i < 2^31
__device__ __forceinline__ unsigned linear_div(unsigned i, unsigned e, unsigned inv) {
  if (e == 1) return i;
  const unsigned q = __umulhi(i, inv);
  return q * e > i ? q - 1 : q;
}

struct LinearDigit { unsigned e, inv; int stride; };
__device__ __forceinline__ int linear_offset(const LinearDigit* d, int n, unsigned i) {
  int off = 0;
  for (int t = 0; t < n; ++t) {
    const unsigned q = t + 1 < n ? linear_div(i, d[t].e, d[t].inv) : 0;  // the last digit is what is left
    off += (int)(i - q * d[t].e) * d[t].stride;
    i = q;
  }
  return off;
}

// A lane keeps the offsets of its fast indices (four, 32 apart; few of them leave lanes for two or four slow
// indices at once) and walks the slow index two at a time.  (Both offsets worked out for every element took
// 142 instructions per 32 of them and bound the pass: 2.7M elements in 28 us, 17 us so.)
__global__ void __launch_bounds__(256) k_linear(const __grid_constant__ LinearPair g) {
  __shared__ LinearDigit digits[8][kMaxOrder];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long c = blockIdx.x * 8LL + warp; c < g.turns; c += gridDim.x * 8LL) {
    const bool second = c >= g.turns0;
    const LinearArgs& a = g.x[second ? 1 : 0];
    const long long at = second ? c - g.turns0 : c, row = at / a.fturns, b = row / a.sturns;
    const long long o = a.off[b];
    const int ext = lane < a.order ? a.dims[b * a.order + lane] : 1;
    int stride = 1;
    for (int d = 0; d + 1 < a.order; ++d) {
      const int e = __shfl_sync(0xffffffffu, ext, d);
      if (d < lane) stride *= e;
    }
    const int mode = lane < a.nfast ? a.fast[lane] : lane < a.order ? a.slow[lane - a.nfast] : 0;
    const unsigned e = __shfl_sync(0xffffffffu, ext, mode);
    const int st = __shfl_sync(0xffffffffu, stride, mode);
    unsigned nf = 1, ns = 1;
    for (int d = 0; d < a.order; ++d) {
      const unsigned x = __shfl_sync(0xffffffffu, e, d);
      if (d < a.nfast) nf *= x;
      else ns *= x;
    }
    const long long fb = (at - row * a.fturns) * kLinearFast, sb = (row - b * a.sturns) * kLinearSlow;
    if (fb >= nf || sb >= ns) continue;
    const unsigned f0 = (unsigned)fb, s0 = (unsigned)sb;
    __syncwarp();
    if (lane < a.order) digits[warp][lane] = {e, e > 1 ? 0xffffffffu / e + 1u : 0u, st};
    __syncwarp();
    const LinearDigit *df = digits[warp], *ds = digits[warp] + a.nfast;
    const int w = nf <= 8 ? 3 : nf <= 16 ? 4 : 5, step = 32 >> w;
    const unsigned f = f0 + (lane & ((1 << w) - 1)), s1 = min(ns, s0 + kLinearSlow);
    int fo[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) fo[u] = f + 32 * u < nf && (u == 0 || w == 5) ? linear_offset(df, a.nfast, f + 32 * u) : -1;
    const double* __restrict__ src = a.src + o;
    double* __restrict__ dst = a.dst + o;
    for (unsigned s = s0 + (lane >> w); s < s1; s += 2 * step) {
      const bool two = s + step < s1;
      const int oa = linear_offset(ds, a.nslow, s), ob = two ? linear_offset(ds, a.nslow, s + step) : 0;
      double va[4], vb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (fo[u] >= 0) va[u] = src[oa + fo[u]];
        if (two && fo[u] >= 0) vb[u] = src[ob + fo[u]];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (fo[u] >= 0) dst[s * nf + f + 32 * u] = va[u];
        if (two && fo[u] >= 0) dst[(s + step) * nf + f + 32 * u] = vb[u];
      }
    }
  }
}

// The strides of the pairs' operands as written.
__global__ void k_linear_recs(PairRec* __restrict__ recs, long long np, ModeMap row, ModeMap col, const int* __restrict__ dimsA,
                              const int* __restrict__ dimsB, int oA, int oB, int a, int b, int ka, int kb) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < np; i += (long long)gridDim.x * blockDim.x) {
    PairRec r = recs[i];
    if (a) {
      int m = 1;
      for (int t = 0; t < row.n; ++t) m *= dimsA[(long long)r.ia * oA + row.x[t]];
      r.rsA = ka ? r.K : 1;
      r.ksA = ka ? 1 : m;
    }
    if (b) {
      int n = 1;
      for (int t = 0; t < col.n; ++t) n *= dimsB[(long long)r.ib * oB + col.x[t]];
      r.rsB = kb ? r.K : 1;
      r.ksB = kb ? 1 : n;
    }
    recs[i] = r;
  }
}

bool modes_consecutive(const int* x, int n) {
  for (int t = 1; t < n; ++t)
    if (x[t] != x[t - 1] + 1) return false;
  return true;
}

static bool k_fast(const int* k, int nk) { return nk && k[0] == 0; }

// Turns of the largest block of X along modes x of one index (the largest extents of all its modes).
static double linear_turns(const sht_tensor* X, const int* x, int n, int each) {
  double largest = 1;
  for (int t = 0; t < n; ++t) largest *= X->bmax[x[t]];
  return std::ceil(largest / each);
}

// Scratch for the operands that need the pass and are worth it; without memory for it the tile kernel
// gathers them.
void linear_prepare(sht_plan* p, cudaStream_t s) {
  const TileMaps& mp = p->tmaps;
  if (p->npairs == 0) return;
  DevicePool* pool = p->ctx->pool.get();
  auto take = [&](PoolBuf& buf, sht_tensor* X, const int* f, int nf, const int* k) {
    const int nk = mp.kk.n;
    if (modes_consecutive(f, nf) && modes_consecutive(k, nk)) return;
    // a block used once is read once either way
    if (p->npairs < X->nblocks) return;
    // blocks so unequal that most turns would be empty
    const bool kf = k_fast(k, nk);
    const double turns = linear_turns(X, f, nf, kf ? kLinearSlow : kLinearFast) *
                         linear_turns(X, k, nk, kf ? kLinearFast : kLinearSlow) * (double)X->nblocks;
    if (turns > 32.0 * ((double)X->nnz / (kLinearFast * kLinearSlow) + (double)X->nblocks) || turns > 1e12) return;
    const size_t bytes = (size_t)X->nnz * 8;
    // a plain plan needs no other scratch: it leaves most of the pool to its caller
    if (p->mode == SHT_MODE_PLAIN_FP64 && bytes > pool->free_bytes() / 4) return;
    try {
      buf = PoolBuf(pool, bytes, s);
    } catch (const Error& e) {
      if (e.code != SHT_ERR_OOM) throw;
    }
  };
  take(p->lin_a, p->A, mp.row.x, mp.row.n, mp.kk.x);
  take(p->lin_b, p->B, mp.col.x, mp.col.n, mp.kk.y);
  if (!p->lin_a.ptr && !p->lin_b.ptr) return;
  k_linear_recs<<<grid_for(p->npairs, 256), 256, 0, s>>>(
      p->d_recs.as<PairRec>(), p->npairs, mp.row, mp.col, p->A->d_dims.as<int>(), p->B->d_dims.as<int>(), mp.oA, mp.oB,
      p->lin_a.ptr != nullptr, p->lin_b.ptr != nullptr, k_fast(mp.kk.x, mp.kk.n), k_fast(mp.kk.y, mp.kk.n));
  SHT_CUDA(cudaGetLastError());
}

// The pass itself, from the operands' present values.
void linear_execute(sht_plan* p, cudaStream_t s) {
  LinearPair g{};
  int n = 0;
  long long turns[2] = {0, 0};
  auto add = [&](const PoolBuf& buf, const sht_tensor* X, const ModeMap& fm, const int* k) {
    if (!buf.ptr) return;
    if ((size_t)X->nnz * 8 > buf.bytes) fail(SHT_ERR_STATE, "an operand's pattern grew after the plan was made");
    const int nk = p->tmaps.kk.n;
    const bool kf = k_fast(k, nk);
    LinearArgs& a = g.x[n];
    a.src = X->d_data.as<double>();
    a.dst = buf.as<double>();
    a.off = X->d_offsets.as<long long>();
    a.dims = X->d_dims.as<int>();
    a.order = X->order;
    a.nfast = kf ? nk : fm.n;
    a.nslow = kf ? fm.n : nk;
    std::copy(fm.x, fm.x + fm.n, kf ? a.slow : a.fast);
    std::copy(k, k + nk, kf ? a.fast : a.slow);
    a.fturns = (long long)linear_turns(X, a.fast, a.nfast, kLinearFast);
    a.sturns = (long long)linear_turns(X, a.slow, a.nslow, kLinearSlow);
    turns[n++] = X->nblocks * a.fturns * a.sturns;
  };
  add(p->lin_a, p->A, p->tmaps.row, p->tmaps.kk.x);
  add(p->lin_b, p->B, p->tmaps.col, p->tmaps.kk.y);
  if (n == 0) return;
  g.turns0 = turns[0];
  g.turns = turns[0] + turns[1];
  k_linear<<<(unsigned)std::min<long long>((g.turns + 7) / 8, 1 << 20), 256, 0, s>>>(g);
  SHT_CUDA(cudaGetLastError());
  trace("linear operands", s);
}

}  // namespace sht

// batched.cu -- the FP64 forms of the block-sparse contraction: one persistent kernel (tile_ring.cuh)
// over a work list.
//
// Every C block gets a tile shape from its matrix extents (m, n): by a cost model (shape_cost), or, in
// the batched form, by the autotuner's choice for its size class.  The plan builds a single work
// list of items (ring_item: C block, first row and column, extents) ordered by estimated cost, heaviest
// first; a persistent grid (SMs x resident CTAs) claims items from an atomic counter.  Execute is the
// copy of operands whose modes lie apart (linear.cu), a counter reset and one launch, and is what
// sht_plan_execute_graph captures.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <fstream>
#include <numeric>
#include <cstdio>
#include <sstream>

#include <cub/cub.cuh>

#include "contract.h"
#include "device_common.cuh"
#include "tile_pipe.cuh"
#include "tile_ring.cuh"

namespace sht {

// resident CTAs of the persistent grid (the same for all instances: same shared memory, bounds)
static int ring_grid(sht_ctx* ctx) {
  static DeviceOnce once;
  once.run(ctx->device, [] {
    for (auto* k : {k_tiles<kRingPlan, false>, k_tiles<kRingPlan, true>, k_tiles<kRingMulti, false>,
                    k_tiles<kRingMulti, true>, k_tiles<kRingStack, false>, k_tiles<kRingStack, true>}) {
      SHT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RingSmem)));
      int n = 0;
      SHT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kRingThreads, sizeof(RingSmem)));
      if (n < kRingCtas) fail(SHT_ERR_STATE, "FP64 tile kernel: fewer resident CTAs than its design");
    }
  });
  return ctx->num_sms * kRingCtas;
}

// Polls of one wait, up to a microsecond each: above the time of any tile (the schedule warp waits for
// whole tiles), so that only a fault runs it out.  sht_set_wait_limit replaces it.
static long long ring_wait_limit(const sht_ctx* ctx) { return ctx->wait_limit > 0 ? ctx->wait_limit : 1LL << 26; }

// addressing flags of an expression (tile_ring.cuh)
// the contracted index's first mode is the block's fastest
static int k_first_a(const TileMaps& mp) { return mp.kk.n && mp.kk.x[0] == 0 ? kRingKmA : 0; }
static int k_first_b(const TileMaps& mp) { return mp.kk.n && mp.kk.y[0] == 0 ? kRingKmB : 0; }
static int ring_flags(const TileMaps& mp, const double* A, const double* B) {
  const bool al = reinterpret_cast<uintptr_t>(A) % 16 == 0, bl = reinterpret_cast<uintptr_t>(B) % 16 == 0;
  int f = 0;
  if (al && modes_consecutive(mp.row.x, mp.row.n) && modes_consecutive(mp.kk.x, mp.kk.n)) f |= kRingLinA | k_first_a(mp);
  if (bl && modes_consecutive(mp.col.x, mp.col.n) && modes_consecutive(mp.kk.y, mp.kk.n)) f |= kRingLinB | k_first_b(mp);
  if (modes_consecutive(mp.row.y, mp.row.n)) f |= kRingLinR;
  if (modes_consecutive(mp.col.y, mp.col.n)) f |= kRingLinC;
  return f;
}

// Launches the instance that the operands' addressing needs (all: the flags every request has).
template <int Kind>
static void launch_tiles(const RingArgs& g, int all, int grid, cudaStream_t s) {
  constexpr int linear = kRingLinA | kRingLinB;
  if ((all & linear) == linear) k_tiles<Kind, false><<<grid, kRingThreads, sizeof(RingSmem), s>>>(g);
  else k_tiles<Kind, true><<<grid, kRingThreads, sizeof(RingSmem), s>>>(g);
  SHT_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ small blocks
// C blocks of at most 8 x 8 or 16 x 16: a warp each, one or four fragments, operands straight from memory, many
// warps in flight.
// The persistent kernel pays about 1,100 cycles of hand-overs between its roles for every pair, however
// small.  Same order per element: k ascending within a pair, pairs in order, one fma each.  Measured (us, a
// tile kernel without roles / the persistent kernel / so): 100 x 100 cells of 3x3, 1M pairs 1324 / 2114 / 112;
// 64 x 64 cells of 8x8, 262,144 pairs 534 / 610 / 49; of 16x16 and K 4 387 / 571 / 88; 16 x 16 cells of 8x8, 16,384
// pairs of K 64 312 / 112 / 102.  With few C blocks a warp's chain of pairs is too long (16 x 16 cells of 16x16,
// K 64: 314 / 122 / 196; 24 x 24 cells 185 / 95 / 82): those stay with the persistent kernel, as do serving launches,
// whose requests share one kernel.
template <int F, bool Scale>
__global__ void __launch_bounds__(256) k_small(const __grid_constant__ RingArgs g) {
  const int lane = threadIdx.x & 31, fr = lane >> 2, kq = lane & 3;
  // unsigned: nwork is below 2^31, so that the last step does not wrap
  for (unsigned i = blockIdx.x * 8 + (threadIdx.x >> 5); i < (unsigned)g.nwork; i += gridDim.x * 8) {
    const int4 w = g.work[i];
    const int c = w.x, mt = w.w & 0xffff, nt = w.w >> 16;
    const int ps = g.pstart[c], pe = g.sc.alpha_zero ? ps : g.pstart[c + 1];
    const int ext = lane < g.mp.oC ? g.dimsC[(long long)c * g.mp.oC + lane] : 1;
    int stride = 1;
    for (int d = 0; d + 1 < g.mp.oC; ++d) {
      const int e = __shfl_sync(0xffffffffu, ext, d);
      if (d < lane) stride *= e;
    }
    double* cb = g.C + g.offC[c];
    int ro[F], co[F][2];  // offsets in C, negative past the block
    // rows and columns past the block read its first: they only reach elements that are not stored
    int ra[F], rb[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const int r = 8 * f + fr;
      const int off = ring_digits(g.mp.row.y, g.mp.row.n, r, ext, stride);
      ro[f] = r < mt ? off : -1;
      ra[f] = r < mt ? r : 0;
      rb[f] = r < nt ? r : 0;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int s = 8 * f + 2 * kq + e, cs = ring_digits(g.mp.col.y, g.mp.col.n, s, ext, stride);
        co[f][e] = s < nt ? cs : -1;
      }
    }
    double acc[F][F][2] = {};
    if (!g.sc.beta_zero) {
#pragma unroll
      for (int x = 0; x < F; ++x)
#pragma unroll
        for (int y = 0; y < F; ++y)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if ((ro[x] | co[y][e]) >= 0) acc[x][y][e] = mul_rn(g.sc.beta, cb[ro[x] + co[y][e]]);
    }
    PairRec next{};
    if (ps < pe) next = g.recs[ps];
    for (int p = ps; p < pe; ++p) {
      const PairRec r = next;
      if (p + 1 < pe) next = g.recs[p + 1];
      const double *a[F], *b[F];
#pragma unroll
      for (int f = 0; f < F; ++f) {
        a[f] = g.A + r.offA + ra[f] * r.rsA + kq * r.ksA;
        b[f] = g.B + r.offB + rb[f] * r.rsB + kq * r.ksB;
      }
      // four steps of four k: their loads are in flight together
      for (int k0 = 0; k0 < r.K; k0 += 16) {
        double af[4][F], bf[4][F];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + 4 * u;
          const bool live = k + kq < r.K;  // past the contracted extent: fma(-0, +0, c) == c
#pragma unroll
          for (int f = 0; f < F; ++f) {
            af[u][f] = live ? a[f][k * r.ksA] : -0.0;
            bf[u][f] = live ? b[f][k * r.ksB] : 0.0;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (k0 + 4 * u >= r.K) break;
          if (Scale && k0 + 4 * u + kq < r.K) {
#pragma unroll
            for (int f = 0; f < F; ++f) af[u][f] = mul_rn(g.sc.alpha, af[u][f]);
          }
#pragma unroll
          for (int x = 0; x < F; ++x)
#pragma unroll
            for (int y = 0; y < F; ++y) dmma884(acc[x][y], af[u][x], bf[u][y]);
        }
      }
    }
#pragma unroll
    for (int x = 0; x < F; ++x)
#pragma unroll
      for (int y = 0; y < F; ++y)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if ((ro[x] | co[y][e]) >= 0) cb[ro[x] + co[y][e]] = acc[x][y][e];
  }
}

// Fragments along a side of the largest C block, 0: not for k_small.
constexpr int kSmallExtent = 16, kSmallK = 64;
static int small_blocks(const sht_plan* p) {
  auto largest = [](const sht_tensor* X, const std::vector<int>& modes) {
    long long e = 1;
    for (int x : modes) e = std::min(e * X->bmax[x], 1LL << 31);
    return e;
  };
  const long long side = std::max(largest(p->C, p->maps.rowC), largest(p->C, p->maps.colC)), K = largest(p->A, p->maps.colA);
  if (side > kSmallExtent || K > kSmallK || p->ncblk < (side > 8 ? 256 + 4 * K : 256)) return 0;
  return side > 8 ? 2 : 1;
}

static void launch_small(sht_ctx* ctx, const RingArgs& g, int f, cudaStream_t s) {
  if (g.nwork <= 0) return;
  const int grid = (int)std::min((g.nwork + 7LL) / 8, ctx->num_sms * 8LL);
  const bool scale = g.sc.alpha != 1.0;
  if (f == 1) (scale ? k_small<1, true> : k_small<1, false>)<<<grid, 256, 0, s>>>(g);
  else (scale ? k_small<2, true> : k_small<2, false>)<<<grid, 256, 0, s>>>(g);
  SHT_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ size classes
static int ilog2ceil(long long v) {
  int b = 0;
  while ((1LL << b) < v) ++b;
  return b;
}

struct ClassKey {
  int lm, ln, lk;
  std::string str() const { return std::to_string(lm) + "," + std::to_string(ln) + "," + std::to_string(lk); }
};

struct HostPlanView {
  std::vector<long long> m, n, ksum;  // per C block
  std::vector<int> pstart;
  std::vector<ClassKey> key;
};

static HostPlanView host_view(sht_plan* p, cudaStream_t s) {
  HostPlanView v;
  sht_tensor *A = p->A, *B = p->B, *C = p->C;
  (void)B;
  tensor_sync_host(C, s);
  const long long nc = p->ncblk;
  v.pstart.resize(nc + 1);
  SHT_CUDA(cudaMemcpyAsync(v.pstart.data(), p->d_pstart.ptr, (nc + 1) * 4, cudaMemcpyDeviceToHost, s));
  std::vector<int> pa(p->npairs);
  if (p->npairs) SHT_CUDA(cudaMemcpyAsync(pa.data(), p->d_pair_a.ptr, p->npairs * 4, cudaMemcpyDeviceToHost, s));
  SHT_CUDA(cudaStreamSynchronize(s));
  v.m.resize(nc);
  v.n.resize(nc);
  v.ksum.resize(nc);
  v.key.resize(nc);
  for (long long c = 0; c < nc; ++c) {
    const int64_t id = C->ids[c];
    long long m = 1, n = 1;
    for (int ax : p->maps.rowC) m *= C->bs[ax][(id / C->gstride[ax]) % C->nblk[ax]];
    for (int ax : p->maps.colC) n *= C->bs[ax][(id / C->gstride[ax]) % C->nblk[ax]];
    long long ks = 0;
    for (int q = v.pstart[c]; q < v.pstart[c + 1]; ++q) {
      const int64_t ida = A->ids[pa[q]];
      long long k = 1;
      for (int ax : p->maps.colA) k *= A->bs[ax][(ida / A->gstride[ax]) % A->nblk[ax]];
      ks += k;
    }
    v.m[c] = m;
    v.n[c] = n;
    v.ksum[c] = ks;
    const long long kavg = (v.pstart[c + 1] > v.pstart[c]) ? ks / (v.pstart[c + 1] - v.pstart[c]) : 1;
    v.key[c] = {ilog2ceil(m), ilog2ceil(n), ilog2ceil(std::max(1LL, kavg))};
  }
  return v;
}

// The tiles of the sampled C blocks in one shape, the blocks ordered by cost, heaviest first.
static std::vector<int4> sampled_work(const HostPlanView& v, std::vector<long long> blocks, int sh) {
  const int tm = ring_tm(sh), tn = ring_tn(sh);
  std::stable_sort(blocks.begin(), blocks.end(), [&](long long a, long long b) { return v.ksum[a] > v.ksum[b]; });
  std::vector<int4> w;
  for (long long c : blocks) {
    const int m = (int)v.m[c], n = (int)v.n[c], tiles = ring_ntiles(m, tm) * ring_ntiles(n, tn);
    for (int t = 0; t < tiles; ++t) w.push_back(ring_item((int)c, t, m, n, tm, tn));
  }
  return w;
}

static void launch_plan(sht_ctx* ctx, const RingArgs& g, cudaStream_t s) {
  if (g.nwork <= 0) return;
  SHT_CUDA(cudaMemsetAsync(g.counter, 0, sizeof(int), s));
  const int grid = std::min(ring_grid(ctx), g.nwork);
  launch_tiles<kRingPlan>(g, g.flags, grid, s);
}

// ------------------------------------------------------------------ device work list
__global__ void k_block_shapes(const int* __restrict__ cm, const int* __restrict__ cn,
                               const long long* __restrict__ cksum, const int* __restrict__ pstart, long long nc,
                               const unsigned char* __restrict__ table, int fixed_tm, int fixed_tn,
                               int* __restrict__ shape, long long* __restrict__ tiles,
                               long long* __restrict__ touched_tiles, unsigned long long* __restrict__ key,
                               int* __restrict__ idx) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x) {
    const long long m = cm[c], n = cn[c], ks = cksum[c];
    const int np = pstart[c + 1] - pstart[c];
    int sh = 0;
    if (fixed_tm <= 0) {
      const int t = table ? table[class_index((int)m, (int)n, np > 0 ? ks / np : 1)] : 255;
      sh = t != 255 ? t : model_shape((int)m, (int)n);
    }
    const long long tm = fixed_tm > 0 ? fixed_tm : ring_tm(sh), tn = fixed_tm > 0 ? fixed_tn : ring_tn(sh);
    const long long nt = ((m + tm - 1) / tm) * ((n + tn - 1) / tn);
    shape[c] = sh;
    tiles[c] = nt;
    touched_tiles[c] = np > 0 ? nt : 0;
    // cost of one tile, coarsened to 16 bits (the float's exponent and 7 mantissa bits: the
    // order is for load balance only, and the stable sort keeps ties in block order)
    const float cost = np > 0 ? (float)((double)(tm * tn) * (double)ks + 1.0) : 0.0f;
    key[c] = (unsigned long long)(__float_as_uint(cost) >> 16);
    idx[c] = (int)c;
  }
}

__global__ void k_gather_tiles(const int* __restrict__ idx, const long long* __restrict__ tiles, long long nc,
                               long long* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nc; i += (long long)gridDim.x * blockDim.x)
    out[i] = tiles[idx[i]];
}

// One warp per C block of the order: its tiles, as (C block, tile, ., .) for split plans (ring 0).
__global__ void k_emit_items(const int* __restrict__ idx, const long long* __restrict__ tiles_sorted,
                             const long long* __restrict__ off, const int* __restrict__ shape,
                             const int* __restrict__ cm, const int* __restrict__ cn, int ring, long long nc,
                             int4* __restrict__ work) {
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (long long i = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); i < nc; i += (long long)gridDim.x * wpb) {
    const int c = idx[i], sh = shape[c], m = cm[c], n = cn[c];
    const long long w0 = off[i], nt = tiles_sorted[i];
    for (long long t = lane; t < nt; t += 32)
      work[w0 + t] = ring ? ring_item(c, (int)t, m, n, ring_tm(sh), ring_tn(sh)) : make_int4(c, (int)t, 0, 0);
  }
}

// Up to eight device scalars (each a value or the sum of two) gathered into one buffer for a
// single read-back.
struct ScalarSrc {
  DevSum v[8];
  int n;
};
__global__ void k_collect(ScalarSrc src, long long* __restrict__ out) {
  const int i = threadIdx.x;
  if (i < src.n) out[i] = *src.v[i].a + (src.v[i].b ? *src.v[i].b : 0);
}

PoolBuf tuned_table(sht_ctx* ctx, cudaStream_t s) {
  std::vector<unsigned char> h(32 * 32 * 32, 255);
  for (auto& kv : ctx->tuned) {
    int lm, ln, lk;
    if (std::sscanf(kv.first.c_str(), "%d,%d,%d", &lm, &ln, &lk) == 3 && lm < 32 && ln < 32 && lk < 32)
      h[(lm * 32 + ln) * 32 + lk] = (unsigned char)kv.second;
  }
  PoolBuf table(ctx->pool.get(), h.size(), s);
  SHT_CUDA(cudaMemcpyAsync(table.ptr, h.data(), h.size(), cudaMemcpyHostToDevice, s));
  SHT_CUDA(cudaStreamSynchronize(s));  // pageable source
  return table;
}

void device_work_list(sht_plan* p, int fixed_tm, int fixed_tn, bool per_class, cudaStream_t s, const DevSum* extra,
                      long long* extra_out, int nextra, const unsigned long long* order_key, int order_bits) {
  if (nextra > 3) fail(SHT_ERR_INVALID, "work list: at most three extra scalars");
  DevicePool* pool = p->ctx->pool.get();
  const long long nc = p->ncblk;
  p->bwork = p->bwork_touched = 0;
  if (nc == 0) {
    p->d_bwork = PoolBuf(pool, sizeof(int4), s);
    return;
  }
  PoolBuf table;
  if (per_class && !p->ctx->tuned.empty()) table = tuned_table(p->ctx, s);
  PoolBuf shape(pool, nc * 4, s), tiles(pool, nc * 8, s), ttiles(pool, nc * 8, s), key(pool, nc * 8, s),
      idx(pool, nc * 4, s), key2(pool, nc * 8, s), idx2(pool, nc * 4, s), tsorted(pool, nc * 8, s),
      off(pool, nc * 8, s), sums(pool, 16, s);
  k_block_shapes<<<grid_for(nc, 256), 256, 0, s>>>(
      p->d_cm.as<int>(), p->d_cn.as<int>(), p->d_cksum.as<long long>(), p->d_pstart.as<int>(), nc,
      table.as<unsigned char>(), fixed_tm, fixed_tn, shape.as<int>(), tiles.as<long long>(),
      ttiles.as<long long>(), key.as<unsigned long long>(), idx.as<int>());
  SHT_CUDA(cudaGetLastError());
  // a caller's order (ascending keys, untouched blocks keyed last) replaces the cost order
  auto sort_blocks = [&](void* tmp_ptr, size_t& bytes) {
    if (order_key)
      cub::DeviceRadixSort::SortPairs(tmp_ptr, bytes, key.as<unsigned long long>(), key2.as<unsigned long long>(),
                                      idx.as<int>(), idx2.as<int>(), (int)nc, 0, order_bits, s);
    else
      cub::DeviceRadixSort::SortPairsDescending(tmp_ptr, bytes, key.as<unsigned long long>(),
                                                key2.as<unsigned long long>(), idx.as<int>(), idx2.as<int>(), (int)nc, 0,
                                                16, s);
  };
  if (order_key)
    SHT_CUDA(cudaMemcpyAsync(key.ptr, order_key, nc * 8, cudaMemcpyDeviceToDevice, s));
  size_t tb = 0, tb2 = 0, tb3 = 0;
  sort_blocks(nullptr, tb);
  cub::DeviceScan::ExclusiveSum(nullptr, tb2, tsorted.as<long long>(), off.as<long long>(), (int)nc, s);
  cub::DeviceReduce::Sum(nullptr, tb3, ttiles.as<long long>(), sums.as<long long>(), (int)nc, s);
  PoolBuf tmp(pool, std::max(tb, std::max(tb2, tb3)), s);
  sort_blocks(tmp.ptr, tb);
  k_gather_tiles<<<grid_for(nc, 256), 256, 0, s>>>(idx2.as<int>(), tiles.as<long long>(), nc, tsorted.as<long long>());
  cub::DeviceScan::ExclusiveSum(tmp.ptr, tb2, tsorted.as<long long>(), off.as<long long>(), (int)nc, s);
  cub::DeviceReduce::Sum(tmp.ptr, tb3, ttiles.as<long long>(), sums.as<long long>(), (int)nc, s);
  // one read-back: the list's length and touched count, the plan's flop count (while it is
  // still on the device) and the caller's extra scalars
  ScalarSrc src{};
  src.v[src.n++] = {off.as<long long>() + nc - 1, tsorted.as<long long>() + nc - 1};
  src.v[src.n++] = {sums.as<long long>(), nullptr};
  const bool fl = p->flops_pending;
  if (fl) src.v[src.n++] = {p->d_flops.as<long long>(), nullptr};  // the double's bits
  const bool npc = p->d_npairs.ptr != nullptr;
  const int inp = src.n;
  if (npc) src.v[src.n++] = {p->d_npairs.as<long long>(), nullptr};  // the device's pair count
  const bool msc = p->d_missing.ptr != nullptr;
  const int ims = src.n;
  if (msc) src.v[src.n++] = {p->d_missing.as<long long>(), nullptr};  // product blocks not in C
  for (int i = 0; i < nextra; ++i) src.v[src.n++] = extra[i];
  PoolBuf got(pool, 64, s);
  k_collect<<<1, 32, 0, s>>>(src, got.as<long long>());
  SHT_CUDA(cudaGetLastError());
  long long h[8];
  SHT_CUDA(cudaMemcpyAsync(h, got.ptr, src.n * 8, cudaMemcpyDeviceToHost, s));  // pageable: returns when done
  if (fl) {
    std::memcpy(&p->flops, &h[2], 8);
    p->flops_pending = false;
  }
  for (int i = 0; i < nextra; ++i) extra_out[i] = h[src.n - nextra + i];
  if (msc) {
    p->d_missing = PoolBuf();
    if (h[ims] != 0) throw PatternGrew{};  // the build assumed C's pattern: redo it
  }
  if (npc) {
    // the pair list was sized from the host patterns: the device must have found as many
    if (h[inp] != p->npairs) fail(SHT_ERR_STATE, "pair count of the host patterns differs from the device's");
    p->d_npairs = PoolBuf();
  }
  const long long total = h[0];
  if (total > (long long)INT32_MAX) fail(SHT_ERR_UNSUPPORTED, "work list above 2^31 tiles");
  p->bwork = total;
  p->bwork_touched = h[1];
  p->d_bwork = PoolBuf(pool, std::max(total, 1LL) * sizeof(int4), s);
  k_emit_items<<<grid_for(nc * 32, 128), 128, 0, s>>>(idx2.as<int>(), tsorted.as<long long>(), off.as<long long>(),
                                                      shape.as<int>(), p->d_cm.as<int>(), p->d_cn.as<int>(),
                                                      fixed_tm > 0 ? 0 : 1, nc, p->d_bwork.as<int4>());
  SHT_CUDA(cudaGetLastError());
}

void ring_prepare(sht_plan* p, cudaStream_t s) {
  if (!p->work_ready) {  // else it came with the pairs
    p->d_counter = PoolBuf(p->ctx->pool.get(), 256, s);
    device_work_list(p, 0, 0, p->mode == SHT_MODE_BATCHED_FP64, s);
  }
  linear_prepare(p, s);
  p->small_blocks = small_blocks(p);
  trace("work list", s);
}

// The kernel arguments of one plan's execute (also used by the serving loop).
static RingArgs ring_args(sht_plan* p, const SparseArgs& g) {
  RingArgs r{};
  r.mp = g.mp;
  r.sc = g.sc;
  r.flags = ring_flags(g.mp, g.A, g.B);
  r.A = g.A; r.offA = g.offA; r.dimsA = g.dimsA;
  r.B = g.B; r.offB = g.offB; r.dimsB = g.dimsB;
  if (p->lin_a.ptr) {
    r.A = p->lin_a.as<double>();
    r.flags |= kRingLinA | k_first_a(g.mp);
  }
  if (p->lin_b.ptr) {
    r.B = p->lin_b.as<double>();
    r.flags |= kRingLinB | k_first_b(g.mp);
  }
  r.C = g.C; r.offC = g.offC; r.dimsC = g.dimsC;
  r.recs = g.recs; r.pstart = g.pstart;
  r.work = p->d_bwork.as<int4>();
  uint64_t one, bb;
  const double d1 = 1.0;
  std::memcpy(&one, &d1, 8);
  std::memcpy(&bb, &g.sc.beta, 8);
  r.nwork = (int)((bb == one) ? p->bwork_touched : p->bwork);
  r.counter = p->d_counter.as<unsigned>();
  r.err = ctx_error_word(p->ctx);
  r.wait_limit = ring_wait_limit(p->ctx);
  return r;
}

size_t batched_desc_bytes() { return sizeof(RingArgs); }

// resident CTAs per SM of the persistent kernel
int batched_ctas_per_sm(sht_ctx* ctx) { return ring_grid(ctx) / ctx->num_sms; }

// One persistent launch over the work of several batched executes (the serving loop).
// host_descs: pinned host memory
// for plans.size() descriptors that the caller keeps unchanged until the launch completes (the
// upload reads it asynchronously); `descs` and `counter` are allocated on `s` and must be held
// as long.  ctas_per_sm (1..batched_ctas_per_sm) sets the persistent grid: fewer than the
// maximum leaves room on every SM for small planning kernels of requests that arrive meanwhile (not
// for k_match, whose CTAs take an SM's whole register file: it runs where a launch leaves SMs empty).
// Returns the number of launch items.
long long batched_multi_launch(sht_ctx* ctx, const std::vector<sht_plan*>& plans, const std::vector<SparseArgs>& args,
                               void* host_descs, PoolBuf& descs, PoolBuf& counter, int ctas_per_sm, cudaStream_t s) {
  DevicePool* pool = ctx->pool.get();
  RingArgs* h = static_cast<RingArgs*>(host_descs);
  long long total = 0;
  int all = ~0;
  for (size_t i = 0; i < plans.size(); ++i) {
    h[i] = ring_args(plans[i], args[i]);
    h[i].first = (int)total;
    all &= h[i].flags;
    total += h[i].nwork;
    if (total > (long long)INT32_MAX) fail(SHT_ERR_UNSUPPORTED, "batched launch above 2^31 tiles");
  }
  if (total == 0) return 0;
  descs = PoolBuf(pool, plans.size() * sizeof(RingArgs), s);
  counter = PoolBuf(pool, 256, s);
  SHT_CUDA(cudaMemcpyAsync(descs.ptr, h, plans.size() * sizeof(RingArgs), cudaMemcpyHostToDevice, s));
  RingArgs b = h[0];
  b.nwork = (int)total;
  b.counter = counter.as<unsigned>();
  b.multi = descs.as<RingArgs>();
  b.nmulti = (int)plans.size();
  SHT_CUDA(cudaMemsetAsync(b.counter, 0, sizeof(int), s));
  const int per_sm = std::max(1, std::min(ctas_per_sm, batched_ctas_per_sm(ctx)));
  const int grid = (int)std::min<long long>((long long)ctx->num_sms * per_sm, total);
  launch_tiles<kRingMulti>(b, all, grid, s);
  return total;
}

void ring_stack(sht_ctx* ctx, const SparseArgs& a, const PairRec& rec, const int* dA, const int* dB, const int* dC,
                long long size_a, long long size_b, long long size_c, int m, int n, long long nb_ops, cudaStream_t s) {
  RingArgs r{};
  r.mp = a.mp;
  r.sc = a.sc;
  r.flags = ring_flags(a.mp, a.A, a.B);
  // gathers with few rows or columns run along k where that is the block's fastest (FP64 lik,lkj->ij 27x9x17
  // by 27x17x4, 1,793 ops: 154 -> 130 us; with 28 rows 163 -> 177 the other way)
  if (!(r.flags & kRingLinA) && m <= 16) r.flags |= k_first_a(a.mp);
  if (!(r.flags & kRingLinB) && n <= 16) r.flags |= k_first_b(a.mp);
  r.A = a.A; r.B = a.B; r.C = a.C;
  r.stack = rec;
  r.size_a = size_a; r.size_b = size_b; r.size_c = size_c;
  std::copy(dA, dA + kMaxOrder, r.sdA);
  std::copy(dB, dB + kMaxOrder, r.sdB);
  std::copy(dC, dC + kMaxOrder, r.sdC);
  r.m = m;
  r.n = n;
  const long long tiles = (long long)ring_ntiles(m, kRingTile) * ring_ntiles(n, kRingTile);
  if (tiles * nb_ops > 0x7fffffffLL) fail(SHT_ERR_UNSUPPORTED, "stack too large for one launch");
  r.tiles_per_op = (int)tiles;
  r.nwork = (int)(tiles * nb_ops);
  r.err = ctx_error_word(ctx);
  r.wait_limit = ring_wait_limit(ctx);
  const int grid = std::min(ring_grid(ctx), r.nwork);
  launch_tiles<kRingStack>(r, r.flags, grid, s);
}

void ring_launch(sht_plan* p, const SparseArgs& g, cudaStream_t s) {
  if (!g.sc.alpha_zero) linear_execute(p, s);
  const RingArgs r = ring_args(p, g);
  constexpr int linear = kRingLinA | kRingLinB;
  if (p->small_blocks && (r.flags & linear) == linear) launch_small(p->ctx, r, p->small_blocks, s);
  else launch_plan(p->ctx, r, s);
  trace("tile kernel", s);
}

// ------------------------------------------------------------------ autotuner
// For every size class with work, time each tile shape on a sample of the class's C blocks
// (written to a scratch copy, never to C) and keep the fastest.  Choices persist in the
// context and, when a file is given, in a "key shape" text file keyed by GPU name and set of shapes.
void autotune(sht_plan* p, const char* cache_file, cudaStream_t s) {
  sht_ctx* ctx = p->ctx;
  cudaDeviceProp prop;
  SHT_CUDA(cudaGetDeviceProperties(&prop, ctx->device));
  std::string gpu = prop.name;
  std::replace(gpu.begin(), gpu.end(), ' ', '_');
  // a choice is a number in a set of tile shapes: lines under the bare GPU name were written for
  // another set (64x64, 128x32, 32x128, 128x16)
  for (int sh = 0; sh < kRingShapes; ++sh)
    gpu += (sh ? "," : ":") + std::to_string(ring_tm(sh)) + "x" + std::to_string(ring_tn(sh));
  if (cache_file) {
    std::ifstream in(cache_file);
    std::string g, k;
    int sh;
    while (in >> g >> k >> sh)
      if (g == gpu && sh >= 0 && sh < kRingShapes) ctx->tuned[k] = sh;
  }
  const HostPlanView v = host_view(p, s);
  linear_execute(p, s);  // the operands as the timing runs read them
  std::map<std::string, std::vector<long long>> members;
  for (long long c = 0; c < p->ncblk; ++c)
    if (v.pstart[c + 1] > v.pstart[c]) members[v.key[c].str()].push_back(c);
  DevicePool* pool = ctx->pool.get();
  // scratch C: offsets remapped into a compact buffer for the sampled blocks
  std::vector<long long> offs(p->ncblk, 0);
  cudaEvent_t e0, e1;
  SHT_CUDA(cudaEventCreate(&e0));
  SHT_CUDA(cudaEventCreate(&e1));
  bool changed = false;
  for (auto& kv : members) {
    if (ctx->tuned.count(kv.first)) continue;
    std::vector<long long> sampled;
    long long elems = 0;
    size_t taken = 0;
    const size_t stride = std::max<size_t>(1, kv.second.size() / 256);
    for (size_t i = 0; i < kv.second.size() && taken < 256; i += stride, ++taken) {
      const long long c = kv.second[i];
      sampled.push_back(c);
      offs[c] = elems;
      elems += v.m[c] * v.n[c];
    }
    PoolBuf scratch(pool, std::max(elems, 1LL) * 8, s), doffs(pool, p->ncblk * 8, s), work(pool, 1, s);
    SHT_CUDA(cudaMemcpyAsync(doffs.ptr, offs.data(), p->ncblk * 8, cudaMemcpyHostToDevice, s));
    double best = 1e300;
    int best_sh = model_shape((int)v.m[kv.second[0]], (int)v.n[kv.second[0]]);
    for (int sh = 0; sh < kRingShapes; ++sh) {
      const std::vector<int4> items = sampled_work(v, sampled, sh);
      work = PoolBuf(pool, items.size() * sizeof(int4), s);
      SHT_CUDA(cudaMemcpyAsync(work.ptr, items.data(), items.size() * sizeof(int4), cudaMemcpyHostToDevice, s));
      SparseArgs sa = sparse_args(p, 1.0, 0.0);
      sa.C = scratch.as<double>();
      sa.offC = doffs.as<long long>();
      RingArgs b = ring_args(p, sa);
      b.work = work.as<int4>();
      b.nwork = (int)items.size();
      launch_plan(ctx, b, s);  // warm-up
      float ms = 0, tot = 0;
      for (int r = 0; r < 3; ++r) {
        SHT_CUDA(cudaEventRecord(e0, s));
        launch_plan(ctx, b, s);
        SHT_CUDA(cudaEventRecord(e1, s));
        SHT_CUDA(cudaEventSynchronize(e1));
        SHT_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        tot += ms;
      }
      if (tot < best) { best = tot; best_sh = sh; }
    }
    ctx->tuned[kv.first] = best_sh;
    changed = true;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (cache_file && changed) {
    std::ofstream out(cache_file, std::ios::app);
    for (auto& kv : ctx->tuned) out << gpu << " " << kv.first << " " << kv.second << "\n";
  }
  device_work_list(p, 0, 0, true, s);
}

}  // namespace sht

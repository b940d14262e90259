// contract.cu -- block-sparse contraction on one GPU: the device plan.
//
// Plan (all on the device; the reference has no block-sparse contract, src/Tensor/Tensor.cpp
// is empty, so the rules below are this library's canonical ones, restated in the oracle; the
// steps are those of the general path, plans over small block grids reach the same lists without
// sorts, see k_match):
//   1. keys: per A block the rolled block indices of its contracted modes, per B block the
//      same over B's contracted modes; the C id splits into an A part and a B part;
//   2. B is radix-sorted by key (stable, so equal keys keep id order); every A block finds
//      its equal-key range by binary search, counts surviving pairs (norm screening) and
//      emits (idC, a, b) in (a, b) order;
//   3. a stable radix sort by idC gives the canonical pair order (idC, idA, idB);
//   4. the distinct idC merged with C's stored ids is the result pattern; C is re-reserved
//      to it when it grows (old blocks copied, new blocks zero-filled);
//   5. per C block its pair range; the form's work list of tiles follows (batched.cu, split.cu:
//      tiles of C blocks with pairs first, untouched C blocks after; the latter are skipped
//      when beta == 1).
#include <cub/cub.cuh>

#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <cstring>

#include "contract.h"
#include "device_common.cuh"
#include "tile_core.cuh"

namespace sht {

double now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

void trace(const char* what, cudaStream_t s) {
  // SHT_TRACE=1: synchronize at every point (device + host time per phase);
  // SHT_TRACE=2: host time only (what the host spends issuing each phase)
  static const int on = [] {
    const char* e = std::getenv("SHT_TRACE");
    return e && (e[0] == '1' || e[0] == '2') ? e[0] - '0' : 0;
  }();
  if (!on) return;
  static double last = 0;
  if (on == 1) cudaStreamSynchronize(s);
  const double t = now_ms();
  std::fprintf(stderr, "[sht] %-28s %8.3f ms\n", what, last > 0 ? t - last : 0.0);
  last = t;
}

// ---------------------------------------------------------------------------------------
// plan kernels
// ---------------------------------------------------------------------------------------
struct KeySpec {
  int nk;                   // contracted modes
  int kmode[kMaxOrder];     // mode index in this tensor
  long long kstride[kMaxOrder];
  int nf;                   // free modes
  int fmode[kMaxOrder];
  long long fstride[kMaxOrder];  // C block-grid stride of the matching C mode
};

__global__ void k_keys(TensorMeta m, KeySpec ks, const long long* __restrict__ ids, long long n,
                       unsigned long long* __restrict__ key, long long* __restrict__ part) {
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < n; b += (long long)gridDim.x * blockDim.x) {
    int c[kMaxOrder];
    unroll_block(m, ids[b], c);
    unsigned long long k = 0;
    long long p = 0;
    for (int t = 0; t < ks.nk; ++t) k += (unsigned long long)c[ks.kmode[t]] * (unsigned long long)ks.kstride[t];
    for (int t = 0; t < ks.nf; ++t) p += (long long)c[ks.fmode[t]] * ks.fstride[t];
    key[b] = k;
    part[b] = p;
  }
}

__global__ void k_iota(int* v, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) v[i] = (int)i;
}

__device__ __forceinline__ long long lower_bound_u64(const unsigned long long* a, long long n, unsigned long long x) {
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ long long lower_bound_i64(const long long* a, long long n, long long x) {
  long long lo = 0, hi = n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// per A block: equal-key range in sorted B keys and number of surviving pairs
__global__ void k_count(const unsigned long long* __restrict__ keyA, long long nA,
                        const unsigned long long* __restrict__ keyBs, const int* __restrict__ permB, long long nB,
                        const double* __restrict__ normA, const double* __restrict__ normB, double eps,
                        long long* __restrict__ lo_out, long long* __restrict__ cnt) {
  for (long long a = blockIdx.x * (long long)blockDim.x + threadIdx.x; a < nA; a += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = keyA[a];
    const long long lo = lower_bound_u64(keyBs, nB, k);
    long long hi = lo;
    while (hi < nB && keyBs[hi] == k) ++hi;
    long long c = hi - lo;
    if (normA) {
      c = 0;
      const double na = normA[a];
      for (long long j = lo; j < hi; ++j) c += (na * normB[permB[j]] >= eps) ? 1 : 0;
    }
    lo_out[a] = lo;
    cnt[a] = c;
  }
}

__global__ void k_emit(const unsigned long long* __restrict__ keyA, const long long* __restrict__ partA, long long nA,
                       const unsigned long long* __restrict__ keyBs, const int* __restrict__ permB,
                       const long long* __restrict__ partB, long long nB, const double* __restrict__ normA,
                       const double* __restrict__ normB, double eps, const long long* __restrict__ lo_in,
                       const long long* __restrict__ end, const long long* __restrict__ cnt, long long* __restrict__ pc,
                       int* __restrict__ pa, int* __restrict__ pb) {
  for (long long a = blockIdx.x * (long long)blockDim.x + threadIdx.x; a < nA; a += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = keyA[a];
    long long w = end[a] - cnt[a];  // inclusive prefix sum minus own count
    const long long pA = partA[a];
    const double na = normA ? normA[a] : 0.0;
    for (long long j = lo_in[a]; j < nB && keyBs[j] == k; ++j) {
      const int b = permB[j];
      if (normA && !(na * normB[b] >= eps)) continue;
      pc[w] = pA + partB[b];
      pa[w] = (int)a;
      pb[w] = b;
      ++w;
    }
  }
}

// The operand side of the linear addressing of a block of extents d (tile_ring.cuh): strides of its
// first free and first contracted mode, and the contracted extent.
struct RecModes {
  int order, fx, kx;
  unsigned kmask;
};
__device__ __forceinline__ void rec_strides(const int* __restrict__ d, const RecModes& m, int& rs, int& ks, int& K) {
  rs = ks = K = 1;
#pragma unroll
  for (int u = 0; u < kMaxOrder; ++u) {
    const int e = u < m.order ? d[u] : 1;
    if (u < m.fx) rs *= e;
    if (u < m.kx) ks *= e;
    if (m.kmask >> u & 1) K *= e;
  }
}

__device__ __forceinline__ PairRec pair_rec(int ia, int ib, const RecModes& ma, const RecModes& mb,
                                            const long long* __restrict__ offA, const int* __restrict__ dimsA,
                                            const long long* __restrict__ offB, const int* __restrict__ dimsB) {
  PairRec r;
  int kb;
  r.offA = offA[ia];
  r.offB = offB[ib];
  rec_strides(dimsA + (long long)ia * ma.order, ma, r.rsA, r.ksA, r.K);
  rec_strides(dimsB + (long long)ib * mb.order, mb, r.rsB, r.ksB, kb);
  r.ia = ia;
  r.ib = ib;
  r.pad = 0;
  return r;
}

// The pairs in canonical order, with their records when rec is given.
__global__ void k_gather_pairs(const int* __restrict__ order, const int* __restrict__ pa_in, const int* __restrict__ pb_in,
                               long long n, int* __restrict__ pa, int* __restrict__ pb, PairRec* __restrict__ rec,
                               RecModes ma, RecModes mb, const long long* __restrict__ offA,
                               const int* __restrict__ dimsA, const long long* __restrict__ offB,
                               const int* __restrict__ dimsB) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int o = order[i];
    const int ia = pa_in[o], ib = pb_in[o];
    pa[i] = ia;
    pb[i] = ib;
    if (rec) rec[i] = pair_rec(ia, ib, ma, mb, offA, dimsA, offB, dimsB);
  }
}

static RecModes rec_modes(int order, const std::vector<int>& free_modes, const std::vector<int>& k_modes) {
  RecModes m{order, free_modes.empty() ? 0 : free_modes[0], k_modes.empty() ? 0 : k_modes[0], 0u};
  for (int x : k_modes) m.kmask |= 1u << x;
  return m;
}

// pair range of each C block
__global__ void k_pstart(const long long* __restrict__ cids, long long nc, const long long* __restrict__ pcs,
                         long long np, int* __restrict__ pstart) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c <= nc; c += (long long)gridDim.x * blockDim.x)
    pstart[c] = (c == nc) ? (int)np : (int)lower_bound_i64(pcs, np, cids[c]);
}

// copy surviving old C blocks into the re-reserved layout
template <typename T>
__global__ void k_move_blocks(const T* __restrict__ src, const long long* __restrict__ old_ids,
                              const long long* __restrict__ old_off, const int* __restrict__ old_dims, int order,
                              long long n_old, const long long* __restrict__ new_ids, long long n_new,
                              const long long* __restrict__ new_off, T* __restrict__ dst) {
  for (long long b = blockIdx.x; b < n_old; b += gridDim.x) {
    long long s = 1;
    for (int d = 0; d < order; ++d) s *= old_dims[b * order + d];
    const long long pos = lower_bound_i64(new_ids, n_new, old_ids[b]);
    const T* p = src + old_off[b];
    T* q = dst + new_off[pos];
    for (long long e = threadIdx.x; e < s; e += blockDim.x) q[e] = p[e];
  }
}

using Cfg128x32 = TileCfg<128, 32, 16, 8, 2>;

// The FP64 tiles of a split plan's work list, computed only when the device word *flag is set
// (an operand of the execute holds a non-finite value): persistent, one 128 x 32 tile per
// iteration, the same tiles and element order as the plain form.
__global__ void __launch_bounds__(Cfg128x32::kThreads) k_contract_tiles_if(SparseArgs g, const int4* __restrict__ work,
                                                                            int nwork, const int* __restrict__ flag) {
  if (*flag == 0) return;
  __shared__ TileSmem<double, Cfg128x32> sm;
  for (int i = blockIdx.x; i < nwork; i += gridDim.x) {
    const int4 w = work[i];
    const int c = w.x;
    auto getc = [&](double*& p, const int*& d) {
      p = g.C + g.offC[c];
      d = g.dimsC + (long long)c * g.mp.oC;
    };
    auto getpair = [&](int p, const double*& a, const int*& ad, const double*& b, const int*& bd) {
      const int ia = g.pair_a[p], ib = g.pair_b[p];
      a = g.A + g.offA[ia];
      ad = g.dimsA + (long long)ia * g.mp.oA;
      b = g.B + g.offB[ib];
      bd = g.dimsB + (long long)ib * g.mp.oB;
    };
    tile_run<double, Cfg128x32>(g.mp, g.sc, w.y, getc, getpair, g.pstart[c], g.pstart[c + 1], sm);
    __syncthreads();  // the next tile reuses the shared tables
  }
}

void fallback_tiles_if(const SparseArgs& g, const int4* work, long long nwork, const int* flag, int grid,
                       cudaStream_t s) {
  if (nwork <= 0) return;
  k_contract_tiles_if<<<(unsigned)std::min<long long>(grid, nwork), Cfg128x32::kThreads, 0, s>>>(g, work, (int)nwork,
                                                                                               flag);
  SHT_CUDA(cudaGetLastError());
}

// Count the product block ids (sorted, with repeats) that are absent from the stored C ids
// (sorted, unique): zero means the result pattern is C's pattern.
__global__ void k_count_missing(const long long* __restrict__ pc, long long np, const long long* __restrict__ cids,
                                long long nc, unsigned long long* __restrict__ missing) {
  unsigned long long n = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < np; i += (long long)gridDim.x * blockDim.x) {
    if (i > 0 && pc[i] == pc[i - 1]) continue;  // one search per distinct id
    const long long id = pc[i];
    long long lo = 0, hi = nc;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (cids[mid] < id) lo = mid + 1; else hi = mid;
    }
    if (lo == nc || cids[lo] != id) ++n;
  }
  if (n) atomicAdd(missing, n);
}

// ---------------------------------------------------------------------------------------
// plans over small block grids (cluster-built)
// ---------------------------------------------------------------------------------------
// When C's block grid and the contracted block grid are small, the plan needs no sorts: C's cells
// (block grid positions, in id order) are counted directly, and the pairs of one cell, which differ
// in their contracted coordinates and so in their A block, are ranked by A block.  One cluster of
// eight CTAs (k_match: hardware barriers, eight SMs) counts pairs, finds the result pattern and sums
// what the host needs for its allocations; after one read-back, k_match_cells and k_match_pairs
// write the pattern, the pairs and the work list.  The general path below takes about 45 launches
// and reads for the same plan, two to five microseconds each: ijl,lk->ijk over 20 blocks per mode
// (12,872 pairs) planned in 330 us that way and in 85 us this way, host time and read-backs included.
constexpr int kMatchCtas = 8, kMatchThreads = 1024;
constexpr long long kMatchCells = 1 << 18;  // C's block grid
constexpr int kMatchKeys = 512;             // contracted block grid: also the most pairs of one cell
constexpr int kMatchBuckets = 1024;         // classes of work items in list order; last: untouched blocks
constexpr int kMatchCosts = 64;             // cost classes, heaviest first
constexpr int kMatchSums = 9;               // pairs, blocks, elements, tiles touched / untouched, flops, new blocks,
                                            // row and column table entries (split plans)

// Whether counting is the faster path, from the mean pairs of a key.  Its cluster has eight SMs for the pairs
// and the cells, and a warp lists the tiles of its cells one cell after another: about 0.27 ns a cell, 3.5 ns
// a C block, 2.5 ns a block of the operands and 0.4 ns a pair beyond the launches.  The general path costs some 0.4 ms more to start with
// and 0.1 ns a pair; with no C yet it writes the new pattern in steps of its own, 6 ns a block.  Measured, a
// plan (us, general / counted): 8 keys, 512 x 512 cells, 2.1M pairs 905 / 2355; 512 keys, 512 x 512 cells,
// 0.33M pairs 454 / 880; 100 keys, 100 x 100 cells, 1M pairs 493 / 458; 128 keys, 512 x 512 cells, 12,782
// pairs 372 / 293; one key, 200,000 cells, 99,731 pairs 525 / 833.  A contraction into a new C, the same four: 7983 / 6739, 3015 / 2239, 2714 / 2610, 735 / 467.
static bool match_pays(double cells, double pairs, double operand_blocks, bool new_c) {
  const double blocks = std::min(cells, pairs);
  const double counted = 0.27e-3 * cells + 3.5e-3 * blocks + 0.4e-3 * pairs + 2.5e-3 * operand_blocks;
  return counted <= 500 + (new_c ? 150 + 6e-3 * blocks : 0);
}

struct MatchArgs {
  TensorMeta mA, mB, mC;
  KeySpec ka, kb;
  ModeMap row, col;
  const long long *idsA, *idsB, *idsC;
  long long nA, nB, nC;
  const double *normA, *normB;  // null: no screening
  double eps;
  int ncell, kspan;
  int split_m, split_n;          // split plans: the tile (128 x 32); 0: the FP64 forms' shapes
  int many;                      // split plans: this many blocks are listed by row coordinates, fewer by cost
  int row_span;                  // positions of the row modes' block grid
  const unsigned char* table;    // the autotuner's shapes (null: the model's)
  // workspace
  int *kcnt, *blist, *keyA, *cellA, *kA, *keyB, *cellB, *rankB;
  int *ccnt, *cold, *cidx, *pofs, *rofs, *cofs, *nocc;
  long long *cks, *eofs, *csum;
  unsigned long long *bucket, *bcur;
  long long* out;                // kMatchSums totals, host-mapped
};

__device__ __forceinline__ void match_sync() {
  __threadfence();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// extents, tile shape and cost class of one cell
struct MatchCell {
  int m, n, sh, nt, bucket;
  long long elems;
};
__device__ __forceinline__ MatchCell match_cell(const MatchArgs& g, int cell, int np, long long ks, bool by_row) {
  MatchCell c{1, 1, 0, 0, 0, 1};
  int row = 0, mul = 1;
  for (int t = 0; t < g.row.n; ++t) {
    const int y = g.row.y[t], x = cell / (int)g.mC.gstride[y] % g.mC.nblk[y];
    c.m *= g.mC.bsizes[g.mC.bstart[y] + x];
    row += x * mul;
    mul *= g.mC.nblk[y];
  }
  for (int t = 0; t < g.col.n; ++t) {
    const int y = g.col.y[t];
    c.n *= g.mC.bsizes[g.mC.bstart[y] + cell / (int)g.mC.gstride[y] % g.mC.nblk[y]];
  }
  c.elems = (long long)c.m * c.n;
  int ntr, ntc, sr, sc;
  if (g.split_m) {
    ntr = (c.m + g.split_m - 1) / g.split_m;
    ntc = (c.n + g.split_n - 1) / g.split_n;
    sr = g.split_m;
    sc = g.split_n;
  } else {
    int t = 255;
    if (g.table) t = g.table[class_index(c.m, c.n, np > 0 ? ks / np : 1)];
    c.sh = t != 255 ? t : model_shape(c.m, c.n);
    ntr = ring_ntiles(c.m, ring_tm(c.sh));
    ntc = ring_ntiles(c.n, ring_tn(c.sh));
    sr = ring_step(c.m, ntr);
    sc = ring_step(c.n, ntc);
  }
  c.nt = ntr * ntc;
  if (np == 0) {
    c.bucket = kMatchBuckets - 1;
  } else if (by_row) {  // blocks that read the same A slabs run close together in time
    const int span = min(g.row_span, kMatchBuckets - 1);
    c.bucket = (int)((long long)row * span / g.row_span);
  } else {  // cost of a tile in half octaves, heaviest first
    const float cost = (float)sr * (float)sc * (float)ks + 1.0f;
    c.bucket = kMatchCosts - 1 - min(kMatchCosts - 1, (int)(__float_as_uint(cost) >> 22) - 254);
  }
  return c;
}

// inclusive scan over the CTA (1024 threads); scratch: 32 values
template <typename T>
__device__ __forceinline__ T match_scan(T v, T* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = 1; d < 32; d <<= 1) {
    const T o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += o;
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    T w = scratch[lane];
    for (int d = 1; d < 32; d <<= 1) {
      const T o = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += o;
    }
    scratch[lane] = w;
  }
  __syncthreads();
  return warp ? v + scratch[warp - 1] : v;
}

// the surviving pairs of A block a, `width` lanes at a time (lane: this thread's among them): f(b, cell)
template <class F>
__device__ __forceinline__ void match_pairs_of(const MatchArgs& g, const int* kstart, int a, int lane, int width, F f) {
  const int k = g.keyA[a], cell = g.cellA[a];
  const double na = g.normA ? g.normA[a] : 0.0;
  for (int j = kstart[k] + lane; j < kstart[k + 1]; j += width) {
    const int b = g.blist[j];
    if (g.normA && !(na * g.normB[b] >= g.eps)) continue;
    f(b, cell + g.cellB[b]);
  }
}
// lanes per A block: about the mean length of a key's B list
__device__ __forceinline__ int match_width(const MatchArgs& g) {
  const long long mean = g.nB / g.kspan;
  return mean <= 4 ? 4 : mean <= 8 ? 8 : mean <= 16 ? 16 : 32;
}

__device__ __forceinline__ void match_kstart(const MatchArgs& g, int* kstart) {
  // exclusive starts of the contracted keys' B lists, per CTA (warp 0)
  if (threadIdx.x < 32) {
    int base = 0;
    for (int i = 0; i < g.kspan; i += 32) {
      const int l = threadIdx.x, v = i + l < g.kspan ? g.kcnt[i + l] : 0;
      int x = v;
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, x, d);
        if (l >= d) x += o;
      }
      if (i + l < g.kspan) kstart[i + l] = base + x - v;
      base += __shfl_sync(0xffffffffu, x, 31);
    }
    if (threadIdx.x == 0) kstart[g.kspan] = base;
  }
  __syncthreads();
}

__global__ void __cluster_dims__(kMatchCtas, 1, 1) __launch_bounds__(kMatchThreads) k_match(const __grid_constant__ MatchArgs g) {
  __shared__ int kstart[kMatchKeys + 1];
  __shared__ long long scratch[32];
  __shared__ int iscratch[32];
  __shared__ unsigned long long hist[kMatchBuckets];
  __shared__ long long sums[kMatchSums];
  const int cta = blockIdx.x, gt = cta * kMatchThreads + threadIdx.x, nt = kMatchCtas * kMatchThreads;
  const int lane = threadIdx.x & 31;
  for (int i = gt; i < g.kspan; i += nt) g.kcnt[i] = 0;
  for (int i = gt; i < g.ncell; i += nt) {
    g.ccnt[i] = 0;
    g.cold[i] = 0;
    g.cks[i] = 0;
  }
  if (gt < kMatchBuckets) g.bucket[gt] = g.bcur[gt] = 0;
  if (gt == 0) *g.nocc = 0;
  hist[threadIdx.x] = 0;
  if (threadIdx.x < kMatchSums) sums[threadIdx.x] = 0;
  match_sync();
  // keys and C parts of the operands' blocks; C's stored cells
  for (int b = gt; b < g.nB; b += nt) {
    int c[kMaxOrder];
    unroll_block(g.mB, g.idsB[b], c);
    long long k = 0, p = 0;
    for (int t = 0; t < g.kb.nk; ++t) k += c[g.kb.kmode[t]] * g.kb.kstride[t];
    for (int t = 0; t < g.kb.nf; ++t) p += c[g.kb.fmode[t]] * g.kb.fstride[t];
    g.keyB[b] = (int)k;
    g.cellB[b] = (int)p;
    g.rankB[b] = atomicAdd(&g.kcnt[k], 1);
  }
  for (int a = gt; a < g.nA; a += nt) {
    int c[kMaxOrder];
    unroll_block(g.mA, g.idsA[a], c);
    long long k = 0, p = 0;
    int K = 1;
    for (int t = 0; t < g.ka.nk; ++t) {
      const int x = c[g.ka.kmode[t]];
      k += x * g.ka.kstride[t];
      K *= g.mA.bsizes[g.mA.bstart[g.ka.kmode[t]] + x];
    }
    for (int t = 0; t < g.ka.nf; ++t) p += c[g.ka.fmode[t]] * g.ka.fstride[t];
    g.keyA[a] = (int)k;
    g.cellA[a] = (int)p;
    g.kA[a] = K;
  }
  for (int c = gt; c < g.nC; c += nt) g.cold[g.idsC[c]] = 1;
  match_sync();
  match_kstart(g, kstart);
  for (int b = gt; b < g.nB; b += nt) g.blist[kstart[g.keyB[b]] + g.rankB[b]] = b;
  match_sync();
  // pairs per cell and their contracted extents
  const int width = match_width(g);
  for (int a = gt / width; a < g.nA; a += nt / width)
    match_pairs_of(g, kstart, a, lane & (width - 1), width, [&](int, int cell) {
      atomicAdd(&g.ccnt[cell], 1);
      atomicAdd(reinterpret_cast<unsigned long long*>(&g.cks[cell]), (unsigned long long)g.kA[a]);
    });
  match_sync();
  const int per = (g.ncell + kMatchCtas - 1) / kMatchCtas, c0 = min(g.ncell, cta * per), c1 = min(g.ncell, c0 + per);
  bool by_row = false;
  if (g.split_m) {
    int occ = 0;
    for (int cell = c0 + threadIdx.x; cell < c1; cell += kMatchThreads) occ += g.ccnt[cell] || g.cold[cell];
    for (int d = 16; d; d >>= 1) occ += __shfl_xor_sync(0xffffffffu, occ, d);
    if (lane == 0 && occ) atomicAdd(g.nocc, occ);
    match_sync();
    by_row = *static_cast<volatile int*>(g.nocc) >= g.many;
  }
  // totals of this CTA's range of cells, and the classes
  {
    long long v[kMatchSums] = {};
    for (int cell = c0 + threadIdx.x; cell < c1; cell += kMatchThreads) {
      const int np = g.ccnt[cell], old = g.cold[cell];
      if (!np && !old) continue;
      const long long ks = g.cks[cell];
      const MatchCell c = match_cell(g, cell, np, ks, by_row);
      v[0] += np;
      v[1] += 1;
      v[2] += c.elems;
      v[np ? 3 : 4] += c.nt;
      v[5] += 2 * c.elems * ks;
      v[6] += old ? 0 : 1;
      v[7] += (c.m + 3) & ~3;
      v[8] += (c.n + 3) & ~3;
      atomicAdd(&hist[c.bucket], (unsigned long long)c.nt);
    }
#pragma unroll
    for (int i = 0; i < kMatchSums; ++i) {
      for (int d = 16; d; d >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], d);
      if (lane == 0 && v[i]) atomicAdd(reinterpret_cast<unsigned long long*>(&sums[i]), (unsigned long long)v[i]);
    }
    __syncthreads();
    if (threadIdx.x < kMatchSums) g.csum[cta * kMatchSums + threadIdx.x] = sums[threadIdx.x];
    if (hist[threadIdx.x]) atomicAdd(&g.bucket[threadIdx.x], hist[threadIdx.x]);
  }
  match_sync();
  // positions: pairs before each cell, its block number, its first element, its first table entries
  __shared__ long long base[5];
  if (threadIdx.x < 5) {
    const int i = threadIdx.x < 3 ? threadIdx.x : threadIdx.x + 4;
    long long v = 0;
    for (int r = 0; r < cta; ++r) v += g.csum[r * kMatchSums + i];
    base[threadIdx.x] = v;
  }
  __syncthreads();
  for (int lo = c0; lo < c1; lo += kMatchThreads) {
    const int cell = lo + threadIdx.x;
    int np = 0, occ = 0, rm = 0, rn = 0;
    long long el = 0;
    if (cell < c1) {
      np = g.ccnt[cell];
      occ = np || g.cold[cell] ? 1 : 0;
      if (occ) {
        int m = 1, n = 1;
        for (int t = 0; t < g.row.n; ++t) {
          const int y = g.row.y[t];
          m *= g.mC.bsizes[g.mC.bstart[y] + cell / (int)g.mC.gstride[y] % g.mC.nblk[y]];
        }
        for (int t = 0; t < g.col.n; ++t) {
          const int y = g.col.y[t];
          n *= g.mC.bsizes[g.mC.bstart[y] + cell / (int)g.mC.gstride[y] % g.mC.nblk[y]];
        }
        el = (long long)m * n;
        rm = (m + 3) & ~3;
        rn = (n + 3) & ~3;
      }
    }
    const int pi = match_scan(np, iscratch), oi = match_scan(occ, iscratch);
    const long long ei = match_scan(el, scratch);
    int ri = 0, ni = 0;
    if (g.split_m) {
      ri = match_scan(rm, iscratch);
      ni = match_scan(rn, iscratch);
    }
    if (cell < c1) {
      g.pofs[cell] = (int)base[0] + pi - np;
      g.cidx[cell] = occ ? (int)base[1] + oi - 1 : -1;
      g.eofs[cell] = base[2] + ei - el;
      if (g.split_m) {
        g.rofs[cell] = (int)(base[3] + ri - rm);
        g.cofs[cell] = (int)(base[4] + ni - rn);
      }
    }
    __syncthreads();
    if (threadIdx.x == kMatchThreads - 1) {
      base[0] += pi;
      base[1] += oi;
      base[2] += ei;
      base[3] += ri;
      base[4] += ni;
    }
    __syncthreads();
  }
  if (cta == 0 && threadIdx.x < kMatchSums) {
    long long v = 0;
    for (int r = 0; r < kMatchCtas; ++r) v += g.csum[r * kMatchSums + threadIdx.x];
    g.out[threadIdx.x] = v;
    __threadfence_system();
  }
}

// What k_match found, written into the plan's and (when the pattern grew) C's arrays.
struct MatchOut {
  int *pstart, *cm, *cn, *tmp_a, *tmp_b, *tmp_c;
  long long* cksum;
  long long *ids, *offs;  // C's new index (null: the pattern is unchanged)
  int* dims;
  int4* work;
  unsigned* counter;      // the FP64 forms' (null in split plans)
  long long *rowbase, *colbase;  // split plans: first entry of each block in the row / column tables
  long long npairs, nblocks;
};
__global__ void __launch_bounds__(256) k_match_cells(const __grid_constant__ MatchArgs g, MatchOut o) {
  __shared__ int kstart[kMatchKeys + 1];
  __shared__ unsigned long long bstart[kMatchBuckets];
  // even CTAs write the cells, odd CTAs place the pairs: two chains of dependent loads side by side
  const int lane = threadIdx.x & 31, half = gridDim.x / 2, id = blockIdx.x / 2;
  if (blockIdx.x & 1) {
    match_kstart(g, kstart);
    const int width = match_width(g);
    for (int a = (id * 256 + threadIdx.x) / width; a < g.nA; a += half * 256 / width)
      match_pairs_of(g, kstart, a, lane & (width - 1), width, [&](int b, int cell) {
        // the old-block marks are not needed any more: the cells' cursors (from 0 or 1)
        const int slot = g.pofs[cell] + (atomicAdd(&g.cold[cell], 2) >> 1);
        o.tmp_a[slot] = a;
        o.tmp_b[slot] = b;
        o.tmp_c[slot] = g.cidx[cell];
      });
    return;
  }
  {  // starts of the classes: four per thread
    __shared__ unsigned long long wsum[8];
    const int warp = threadIdx.x >> 5;
    unsigned long long v[4], t = 0;
    for (int i = 0; i < 4; ++i) {
      v[i] = t;
      t += g.bucket[4 * threadIdx.x + i];
    }
    unsigned long long x = t;
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned long long before = x - t;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    for (int i = 0; i < 4; ++i) bstart[4 * threadIdx.x + i] = before + v[i];
  }
  static_assert(kMatchBuckets == 4 * 256, "four classes per thread");
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    o.pstart[o.nblocks] = (int)o.npairs;
    if (o.counter) *o.counter = 0;
  }
  const bool by_row = g.split_m && *g.nocc >= g.many;
  __syncthreads();
  const int gw = (id * 256 + threadIdx.x) >> 5, nw = half * 8;
  for (int base = gw * 32; base < g.ncell; base += nw * 32) {
    const int cell = base + lane;
    const int ci = cell < g.ncell ? g.cidx[cell] : -1;
    MatchCell c{};
    unsigned long long w0 = 0;
    if (ci >= 0) {
      const int np = g.ccnt[cell];
      const long long ks = g.cks[cell];
      c = match_cell(g, cell, np, ks, by_row);
      o.pstart[ci] = g.pofs[cell];
      o.cm[ci] = c.m;
      o.cn[ci] = c.n;
      o.cksum[ci] = ks;
      if (o.ids) {
        o.ids[ci] = cell;
        o.offs[ci] = g.eofs[cell];
        for (int d = 0; d < g.mC.order; ++d)
          o.dims[(long long)ci * g.mC.order + d] =
              g.mC.bsizes[g.mC.bstart[d] + cell / (int)g.mC.gstride[d] % g.mC.nblk[d]];
      }
      if (o.rowbase) {
        o.rowbase[ci] = g.rofs[cell];
        o.colbase[ci] = g.cofs[cell];
      }
      w0 = bstart[c.bucket] + atomicAdd(&g.bcur[c.bucket], (unsigned long long)c.nt);
    }
    // the cells' tiles, one cell after another, lanes over tiles
    {
      for (unsigned todo = __ballot_sync(0xffffffffu, ci >= 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const int m = __shfl_sync(0xffffffffu, c.m, l), n = __shfl_sync(0xffffffffu, c.n, l);
        const int sh = __shfl_sync(0xffffffffu, c.sh, l), nt = __shfl_sync(0xffffffffu, c.nt, l);
        const int cc = __shfl_sync(0xffffffffu, ci, l);
        const unsigned long long w = __shfl_sync(0xffffffffu, w0, l);
        for (int t = lane; t < nt; t += 32)
          o.work[w + t] = g.split_m ? make_int4(cc, t, 0, 0) : ring_item(cc, t, m, n, ring_tm(sh), ring_tn(sh));
      }
    }
  }
}

// The pairs of each cell ranked by A block (no two have the same), with their records.
__global__ void __launch_bounds__(256) k_match_pairs(MatchOut o, RecModes ma, RecModes mb, const long long* __restrict__ offA,
                                                     const int* __restrict__ dimsA, const long long* __restrict__ offB,
                                                     const int* __restrict__ dimsB, int* __restrict__ pa,
                                                     int* __restrict__ pb, PairRec* __restrict__ rec) {
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < o.npairs; i += gridDim.x * 256LL) {
    const int a = o.tmp_a[i], b = o.tmp_b[i], c = o.tmp_c[i];
    const int ps = o.pstart[c], pe = o.pstart[c + 1];
    int rank = ps;
    for (int q = ps; q < pe; ++q) rank += o.tmp_a[q] < a ? 1 : 0;
    pa[rank] = a;
    pb[rank] = b;
    if (rec) rec[rank] = pair_rec(a, b, ma, mb, offA, dimsA, offB, dimsB);
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int bits_for(unsigned long long v) {
  int b = 1;
  while (b < 64 && (v >> b)) ++b;
  return b;
}

template <typename T>
static T d2h_scalar(const void* p, cudaStream_t s) {
  T v{};
  SHT_CUDA(cudaMemcpyAsync(&v, p, sizeof(T), cudaMemcpyDeviceToHost, s));
  SHT_CUDA(cudaStreamSynchronize(s));
  return v;
}

static bool bytes_zero(double v) {
  uint64_t u;
  std::memcpy(&u, &v, 8);
  return u == 0;
}

static void check_block_sizes(const sht_tensor* X, const std::vector<int>& mx, const sht_tensor* Y,
                              const std::vector<int>& my, const char* nx, const char* ny) {
  for (size_t t = 0; t < mx.size(); ++t)
    if (X->bs[mx[t]] != Y->bs[my[t]])
      fail(SHT_ERR_SIZE, std::string("Block sizes of mode ") + std::to_string(mx[t]) + " of " + nx + " and mode " +
                             std::to_string(my[t]) + " of " + ny + " do not match");
}

static ModeMap make_modemap(const std::vector<int>& x, const std::vector<int>& y) {
  ModeMap m{};
  m.n = (int)x.size();
  for (size_t i = 0; i < x.size(); ++i) { m.x[i] = x[i]; m.y[i] = y[i]; }
  return m;
}

// per C block: matrix extents m, n, the sum over its pairs of the contracted extent, flops
__global__ void k_cstats(const int* __restrict__ dimsC, int oC, ModeMap row, ModeMap col,
                         const int* __restrict__ pstart, const int* __restrict__ pair_a,
                         const int* __restrict__ dimsA, int oA, ModeMap kk, long long nc, int* __restrict__ m_out,
                         int* __restrict__ n_out, long long* __restrict__ ksum_out, double* __restrict__ flops_out) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x) {
    long long m = 1, n = 1, ks = 0;
    for (int t = 0; t < row.n; ++t) m *= dimsC[c * oC + row.y[t]];
    for (int t = 0; t < col.n; ++t) n *= dimsC[c * oC + col.y[t]];
    for (int p = pstart[c]; p < pstart[c + 1]; ++p) {
      const int* ad = dimsA + (long long)pair_a[p] * oA;
      long long k = 1;
      for (int t = 0; t < kk.n; ++t) k *= ad[kk.x[t]];
      ks += k;
    }
    m_out[c] = (int)m;
    n_out[c] = (int)n;
    ksum_out[c] = ks;
    flops_out[c] = 2.0 * (double)m * (double)n * (double)ks;
  }
}

void cblock_stats(sht_plan* p, cudaStream_t s) {
  DevicePool* pool = p->ctx->pool.get();
  const long long nc = p->ncblk;
  p->d_cm = PoolBuf(pool, std::max(nc, 1LL) * 4, s);
  p->d_cn = PoolBuf(pool, std::max(nc, 1LL) * 4, s);
  p->d_cksum = PoolBuf(pool, std::max(nc, 1LL) * 8, s);
  p->flops = 0.0;
  p->flops_pending = false;
  if (nc == 0) return;
  PoolBuf fl(pool, nc * 8, s);
  p->d_flops = PoolBuf(pool, 8, s);
  k_cstats<<<grid_for(nc, 256), 256, 0, s>>>(p->C->d_dims.as<int>(), p->C->order, p->tmaps.row, p->tmaps.col,
                                              p->d_pstart.as<int>(), p->d_pair_a.as<int>(), p->A->d_dims.as<int>(),
                                              p->A->order, p->tmaps.kk, nc, p->d_cm.as<int>(), p->d_cn.as<int>(),
                                              p->d_cksum.as<long long>(), fl.as<double>());
  SHT_CUDA(cudaGetLastError());
  size_t tb = 0;
  cub::DeviceReduce::Sum(nullptr, tb, fl.as<double>(), p->d_flops.as<double>(), (int)nc, s);
  PoolBuf tmp(pool, tb, s);
  cub::DeviceReduce::Sum(tmp.ptr, tb, fl.as<double>(), p->d_flops.as<double>(), (int)nc, s);
  p->flops_pending = true;  // read with the next synchronization (plan_flops)
  if (!p->flops_event) SHT_CUDA(cudaEventCreateWithFlags(&p->flops_event, cudaEventDisableTiming));
  SHT_CUDA(cudaEventRecord(p->flops_event, s));
}

double plan_flops(sht_plan* p, cudaStream_t s) {
  if (p->flops_pending) {
    // s need not be the stream that computed the count: order the read after it
    if (p->flops_event) SHT_CUDA(cudaStreamWaitEvent(s, p->flops_event, 0));
    p->flops = d2h_scalar<double>(p->d_flops.ptr, s);
    p->flops_pending = false;
  }
  return p->flops;
}

// ------------------------------------------------------------------ plans over small block grids
// A slot of host-mapped memory borrowed from the context for one plan's read-back.
struct PinLease {
  sht_ctx* ctx;
  long long* host;
  explicit PinLease(sht_ctx* c) : ctx(c) {
    std::lock_guard<std::mutex> lk(ctx->lanes_mu);
    if (ctx->pins.empty()) {
      void* h = nullptr;
      SHT_CUDA(cudaHostAlloc(&h, 4096, cudaHostAllocMapped));
      ctx->pin_pages.push_back(h);
      for (int i = 0; i < 32; ++i) ctx->pins.push_back(static_cast<long long*>(h) + 16 * i);
    }
    host = ctx->pins.back();
    ctx->pins.pop_back();
  }
  ~PinLease() {
    std::lock_guard<std::mutex> lk(ctx->lanes_mu);
    ctx->pins.push_back(host);
  }
  PinLease(const PinLease&) = delete;
  PinLease& operator=(const PinLease&) = delete;
};

struct MatchState {
  MatchArgs g{};
  PoolBuf ws, normA, normB, table;
  PinLease pin;
  cudaStream_t stream;
  bool done = false;
  explicit MatchState(sht_ctx* ctx, cudaStream_t s) : pin(ctx), stream(s) {}
  // the kernel writes the pinned slot: it must have finished before the slot is lent again
  ~MatchState() {
    if (!done) cudaStreamSynchronize(stream);
  }
};

}  // namespace sht

sht_plan::~sht_plan() {
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  if (graph) cudaGraphDestroy(graph);
  if (flops_event) cudaEventDestroy(flops_event);
}
sht_plan::sht_plan() = default;

namespace sht {

static void key_specs(const sht_plan* p, KeySpec& ka, KeySpec& kb, unsigned long long& kspan, long double& cgrid) {
  const ShtMaps& mp = p->maps;
  const sht_tensor *A = p->A, *C = p->C;
  kspan = 1;
  ka = KeySpec{};
  kb = KeySpec{};
  ka.nk = kb.nk = (int)mp.colA.size();
  for (size_t t = 0; t < mp.colA.size(); ++t) {
    ka.kmode[t] = mp.colA[t];
    kb.kmode[t] = mp.rowB[t];
    ka.kstride[t] = kb.kstride[t] = (long long)kspan;
    const unsigned long long nb = (unsigned long long)A->nblk[mp.colA[t]];
    if (kspan > (1ULL << 62) / nb) fail(SHT_ERR_UNSUPPORTED, "contracted block grid too large");
    kspan *= nb;
  }
  ka.nf = (int)mp.rowA.size();
  for (size_t t = 0; t < mp.rowA.size(); ++t) { ka.fmode[t] = mp.rowA[t]; ka.fstride[t] = C->gstride[mp.rowC[t]]; }
  kb.nf = (int)mp.colB.size();
  for (size_t t = 0; t < mp.colB.size(); ++t) { kb.fmode[t] = mp.colB[t]; kb.fstride[t] = C->gstride[mp.colC[t]]; }
  cgrid = 1;
  for (int d = 0; d < C->order; ++d) cgrid *= C->nblk[d];
  if (cgrid > 9.0e18L) fail(SHT_ERR_UNSUPPORTED, "C block grid too large");
}

// Launches k_match on s when the grids are small enough (and the pool has room for its workspace);
// plan_build finishes the plan from it.  Called early by callers that have other work to queue.
void plan_match_begin(sht_plan* p, cudaStream_t s) {
  sht_tensor *A = p->A, *B = p->B, *C = p->C;
  const long long nA = A->nblocks, nB = B->nblocks, nC = C->nblocks;
  KeySpec ka, kb;
  unsigned long long kspan;
  long double cgrid;
  key_specs(p, ka, kb, kspan, cgrid);
  if (nA == 0 || nB == 0 || kspan > (unsigned long long)kMatchKeys || cgrid > (long double)kMatchCells) return;
  if (nA > (1 << 20) || nB > (1 << 20)) return;
  if (!match_pays((double)cgrid, (double)nA * (double)nB / (double)kspan, (double)(nA + nB), nC == 0)) return;
  DevicePool* pool = p->ctx->pool.get();
  for (sht_tensor* t : {A, B, C}) tensor_touch(t, s);
  auto st = std::make_shared<MatchState>(p->ctx, s);
  MatchArgs& g = st->g;
  const long long nc = (long long)cgrid;
  try {
    size_t at = 0;
    auto part = [&](size_t bytes) {
      const size_t o = at;
      at += (bytes + 15) & ~(size_t)15;
      return o;
    };
    const size_t o_cks = part(nc * 8), o_eofs = part(nc * 8), o_csum = part(kMatchCtas * kMatchSums * 8),
                 o_bucket = part(kMatchBuckets * 8), o_bcur = part(kMatchBuckets * 8), o_ccnt = part(nc * 4),
                 o_cold = part(nc * 4), o_cidx = part(nc * 4), o_pofs = part(nc * 4), o_rofs = part(nc * 4),
                 o_cofs = part(nc * 4), o_nocc = part(4), o_kcnt = part(kspan * 4),
                 o_blist = part(nB * 4), o_keyA = part(nA * 4), o_cellA = part(nA * 4), o_kA = part(nA * 4),
                 o_keyB = part(nB * 4), o_cellB = part(nB * 4), o_rankB = part(nB * 4);
    st->ws = PoolBuf(pool, at, s);
    char* w = st->ws.as<char>();
    auto ll = [&](size_t o) { return reinterpret_cast<long long*>(w + o); };
    auto in = [&](size_t o) { return reinterpret_cast<int*>(w + o); };
    g.cks = ll(o_cks); g.eofs = ll(o_eofs); g.csum = ll(o_csum);
    g.bucket = reinterpret_cast<unsigned long long*>(w + o_bucket);
    g.bcur = reinterpret_cast<unsigned long long*>(w + o_bcur);
    g.ccnt = in(o_ccnt); g.cold = in(o_cold); g.cidx = in(o_cidx); g.pofs = in(o_pofs); g.rofs = in(o_rofs); g.cofs = in(o_cofs); g.nocc = in(o_nocc); g.kcnt = in(o_kcnt);
    g.blist = in(o_blist); g.keyA = in(o_keyA); g.cellA = in(o_cellA); g.kA = in(o_kA);
    g.keyB = in(o_keyB); g.cellB = in(o_cellB); g.rankB = in(o_rankB);
    if (p->eps > 0.0) {
      st->normA = PoolBuf(pool, nA * 8, s);
      st->normB = PoolBuf(pool, nB * 8, s);
      tensor_norms_device(A, p->norm, st->normA.as<double>(), s);
      tensor_norms_device(B, p->norm, st->normB.as<double>(), s);
      g.normA = st->normA.as<double>();
      g.normB = st->normB.as<double>();
    }
  } catch (const Error& e) {
    st->done = true;
    if (e.code == SHT_ERR_OOM) return;  // the general path needs less at a time, and reports it
    throw;
  }
  g.mA = make_meta(A); g.mB = make_meta(B); g.mC = make_meta(C);
  g.ka = ka; g.kb = kb;
  g.row = make_modemap(p->maps.rowA, p->maps.rowC);
  g.col = make_modemap(p->maps.colB, p->maps.colC);
  g.idsA = A->d_ids.as<long long>(); g.idsB = B->d_ids.as<long long>(); g.idsC = C->d_ids.as<long long>();
  g.nA = nA; g.nB = nB; g.nC = nC;
  g.eps = p->eps;
  g.ncell = (int)nc;
  g.kspan = (int)kspan;
  if (p->mode == SHT_MODE_SPLIT) {
    split_tile(g.split_m, g.split_n);
    g.many = 16 * p->ctx->num_sms;
    g.row_span = 1;
    for (int t = 0; t < g.row.n; ++t) g.row_span *= C->nblk[g.row.y[t]];
  }
  if (p->mode == SHT_MODE_BATCHED_FP64 && !p->ctx->tuned.empty()) st->table = tuned_table(p->ctx, s);
  g.table = st->table.as<unsigned char>();
  void* dev = nullptr;
  SHT_CUDA(cudaHostGetDevicePointer(&dev, st->pin.host, 0));
  g.out = static_cast<long long*>(dev);
  k_match<<<kMatchCtas, kMatchThreads, 0, s>>>(g);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    st->done = true;
    fail(SHT_ERR_CUDA, std::string("k_match: ") + cudaGetErrorString(e));
  }
  p->match = std::move(st);
}

// The plan from k_match's totals: allocations, C's grown pattern, pairs, work list.  False when the
// pool has no room (nothing is changed then).
static bool match_finish(sht_plan* p, cudaStream_t s) {
  const std::shared_ptr<MatchState> st = std::move(p->match);
  p->match.reset();
  DevicePool* pool = p->ctx->pool.get();
  sht_tensor *A = p->A, *B = p->B, *C = p->C;
  SHT_CUDA(cudaStreamSynchronize(s));
  st->done = true;
  long long tot[kMatchSums];
  for (int i = 0; i < kMatchSums; ++i) tot[i] = static_cast<volatile long long*>(st->pin.host)[i];
  const long long np = tot[0], nc = tot[1], nwork = tot[3] + tot[4], nC_old = C->nblocks;
  const bool grow = tot[6] > 0, fp64 = p->mode != SHT_MODE_SPLIT;
  if (np > (long long)INT32_MAX) fail(SHT_ERR_UNSUPPORTED, "more than 2^31 block pairs");
  if (nwork > (long long)INT32_MAX) fail(SHT_ERR_UNSUPPORTED, "work list above 2^31 tiles");
  if (!fp64 && (tot[7] >= (1LL << 31) || tot[8] >= (1LL << 31)))
    fail(SHT_ERR_UNSUPPORTED, "split mode: C row / column tables above 2^31");
  PoolBuf pa, pb, recs, pstart, cm, cn, ck, tmp, work, counter, rowb, colb, ids, offs, dims, data;
  try {
    if (np > 0) {
      pa = PoolBuf(pool, np * 4, s);
      pb = PoolBuf(pool, np * 4, s);
      if (fp64) recs = PoolBuf(pool, np * sizeof(PairRec), s);
      tmp = PoolBuf(pool, np * 12, s);
    }
    pstart = PoolBuf(pool, (nc + 1) * 4, s);
    cm = PoolBuf(pool, std::max(nc, 1LL) * 4, s);
    cn = PoolBuf(pool, std::max(nc, 1LL) * 4, s);
    ck = PoolBuf(pool, std::max(nc, 1LL) * 8, s);
    work = PoolBuf(pool, std::max(nwork, 1LL) * sizeof(int4), s);
    if (fp64) {
      counter = PoolBuf(pool, 256, s);
    } else {
      rowb = PoolBuf(pool, std::max(nc, 1LL) * 8, s);
      colb = PoolBuf(pool, std::max(nc, 1LL) * 8, s);
    }
    if (grow) {
      ids = PoolBuf(pool, nc * 8, s);
      offs = PoolBuf(pool, nc * 8, s);
      dims = PoolBuf(pool, nc * C->order * 4, s);
      data = PoolBuf(pool, std::max(tot[2], 1LL) * 8, s);
    }
  } catch (const Error& e) {
    if (e.code == SHT_ERR_OOM) return false;
    throw;
  }
  MatchOut o{};
  o.pstart = pstart.as<int>();
  o.cm = cm.as<int>();
  o.cn = cn.as<int>();
  o.cksum = ck.as<long long>();
  o.tmp_a = tmp.as<int>();
  o.tmp_b = o.tmp_a + np;
  o.tmp_c = o.tmp_b + np;
  o.ids = ids.as<long long>();
  o.offs = offs.as<long long>();
  o.dims = dims.as<int>();
  o.work = work.as<int4>();
  o.counter = counter.as<unsigned>();
  o.rowbase = rowb.as<long long>();
  o.colbase = colb.as<long long>();
  o.npairs = np;
  o.nblocks = nc;
  const long long warps = std::max<long long>((st->g.ncell + 31) / 32, st->g.nA);
  k_match_cells<<<2 * (unsigned)std::min<long long>((warps + 7) / 8, p->ctx->num_sms * 1LL), 256, 0, s>>>(st->g, o);
  if (np > 0)
    k_match_pairs<<<grid_for(np, 256), 256, 0, s>>>(
        o, rec_modes(A->order, p->maps.rowA, p->maps.colA), rec_modes(B->order, p->maps.colB, p->maps.rowB),
        A->d_offsets.as<long long>(), A->d_dims.as<int>(), B->d_offsets.as<long long>(), B->d_dims.as<int>(),
        pa.as<int>(), pb.as<int>(), recs.as<PairRec>());
  SHT_CUDA(cudaGetLastError());
  if (grow) {
    // C's old blocks may still be in use by earlier work on the caller's stream
    if (nC_old > 0 && p->caller_event) SHT_CUDA(cudaStreamWaitEvent(s, p->caller_event, 0));
    // new blocks start zero-filled, unless the caller writes every element next with nothing left
    // that could fail for want of memory (the FP64 forms: their work list and counter are here)
    if (!(p->c_overwritten && fp64)) {
      SHT_CUDA(cudaMemsetAsync(data.ptr, 0, std::max(tot[2], 1LL) * 8, s));
      if (nC_old > 0) {
        const int grid = (int)std::min<long long>(nC_old, (long long)p->ctx->num_sms * 8);
        k_move_blocks<double><<<grid, 256, 0, s>>>(C->d_data.as<double>(), C->d_ids.as<long long>(),
                                                   C->d_offsets.as<long long>(), C->d_dims.as<int>(), C->order, nC_old,
                                                   ids.as<long long>(), nc, offs.as<long long>(), data.as<double>());
        SHT_CUDA(cudaGetLastError());
      }
    }
    C->d_ids = std::move(ids);
    C->d_offsets = std::move(offs);
    C->d_dims = std::move(dims);
    C->d_data = std::move(data);
    C->nblocks = nc;
    C->nnz = tot[2];
    // the host mirror is read back when a host-side step needs it (no block of it is marked)
    C->host_stale = C->stale_unmarked = true;
    p->index_pending = true;
  }
  p->d_pair_a = std::move(pa);
  p->d_pair_b = std::move(pb);
  p->d_recs = std::move(recs);
  p->d_pstart = std::move(pstart);
  p->d_cm = std::move(cm);
  p->d_cn = std::move(cn);
  p->d_cksum = std::move(ck);
  p->npairs = np;
  p->ncblk = nc;
  p->flops = (double)tot[5];
  p->flops_pending = false;
  p->d_bwork = std::move(work);
  p->d_counter = std::move(counter);
  p->bwork = nwork;
  p->bwork_touched = tot[3];
  p->work_ready = true;
  p->sp_rowbase = std::move(rowb);
  p->sp_colbase = std::move(colb);
  p->sp_rtot = tot[7];
  p->sp_ctot = tot[8];
  return true;
}

void plan_settle(sht_plan* p, cudaStream_t s) {
  if (!p->index_pending) return;
  SHT_CUDA(cudaStreamSynchronize(s));
  p->index_pending = false;
}

sht_plan* plan_create(sht_ctx* ctx, const std::string& expr, sht_tensor* A, sht_tensor* B, sht_tensor* C,
                      double eps, sht_norm norm, sht_mode mode, cudaStream_t s) {
  std::unique_ptr<sht_plan> p(plan_init(ctx, expr, A, B, C, eps, norm, mode, s));
  plan_build(p.get(), s);
  // C's index is complete for any later call; callers order what they queue next on s themselves
  SHT_CUDA(cudaStreamSynchronize(s));
  p->index_pending = false;
  return p.release();
}

sht_plan* plan_init(sht_ctx* ctx, const std::string& expr, sht_tensor* A, sht_tensor* B, sht_tensor* C,
                    double eps, sht_norm norm, sht_mode mode, cudaStream_t s) {
  const double t0 = now_ms();
  trace("plan: start", s);
  if (!A || !B || !C) fail(SHT_ERR_INVALID, "null tensor");
  if (A->ctx != ctx || B->ctx != ctx || C->ctx != ctx) fail(SHT_ERR_INVALID, "tensors from another context");
  if (A->dtype != SHT_F64 || B->dtype != SHT_F64 || C->dtype != SHT_F64)
    fail(SHT_ERR_UNSUPPORTED, "block-sparse contraction runs on FP64 tensors");
  if (A == C || B == C) fail(SHT_ERR_INVALID, "C must not alias A or B");
  for (sht_tensor* t : {A, B, C}) {
    tensor_touch(t, s);
    // a pattern grown by a contraction is known to be unmarked: C's host mirror can stay behind
    if (t != C || !t->stale_unmarked) tensor_sync_host(t, s);
    if (t->has_marked) fail(SHT_ERR_STATE, "tensor has filtered blocks that were not compressed");
  }
  auto p = std::make_unique<sht_plan>();
  p->keep = ctx->pool;
  p->ctx = ctx;
  p->mode = mode;
  p->A = A; p->B = B; p->C = C;
  parse_einsum(expr, A->order, nullptr, B->order, nullptr, C->order, nullptr, p->maps);
  const ShtMaps& mp = p->maps;
  check_block_sizes(A, mp.rowA, C, mp.rowC, "tensor A", "tensor C");
  check_block_sizes(B, mp.colB, C, mp.colC, "tensor B", "tensor C");
  check_block_sizes(A, mp.colA, B, mp.rowB, "tensor A", "tensor B");
  p->eps = eps;
  p->norm = norm;
  p->plan_ms = now_ms() - t0;
  return p.release();
}

void plan_build(sht_plan* p, cudaStream_t s, bool speculate) {
  const double t0 = now_ms();
  sht_ctx* ctx = p->ctx;
  sht_tensor *A = p->A, *B = p->B, *C = p->C;
  // buffers the build reads or replaces are released against this stream
  for (sht_tensor* t : {A, B, C}) tensor_touch(t, s);
  const double eps = p->eps;
  const sht_norm norm = p->norm;
  const ShtMaps& mp = p->maps;
  DevicePool* pool = ctx->pool.get();
  const long long nA = A->nblocks, nB = B->nblocks;

  p->tmaps.row = make_modemap(mp.rowA, mp.rowC);
  p->tmaps.kk = make_modemap(mp.colA, mp.rowB);
  p->tmaps.col = make_modemap(mp.colB, mp.colC);
  p->tmaps.oA = A->order;
  p->tmaps.oB = B->order;
  p->tmaps.oC = C->order;
  if (!p->match) plan_match_begin(p, s);
  if (p->match && match_finish(p, s)) {
    trace("plan: matched", s);
    p->plan_ms += now_ms() - t0;
    return;
  }

  // contracted key radices
  KeySpec ka, kb;
  unsigned long long kspan;
  long double cgrid;
  key_specs(p, ka, kb, kspan, cgrid);

  // Without screening the pair count follows from the host patterns (per contracted key the
  // number of B blocks, summed over A's blocks), so the device count need not be read back.
  long long np_host = -1;
  if (!(eps > 0.0) && kspan <= (1ULL << 16) && nA > 0 && nB > 0) {
    const int* xa = tensor_host_coords(A);
    const int* xb = tensor_host_coords(B);
    std::vector<long long> nbk(kspan, 0);
    for (long long b = 0; b < nB; ++b) {
      long long k = 0;
      for (int t = 0; t < kb.nk; ++t) k += xb[b * B->order + kb.kmode[t]] * kb.kstride[t];
      nbk[k]++;
    }
    np_host = 0;
    for (long long a = 0; a < nA; ++a) {
      long long k = 0;
      for (int t = 0; t < ka.nk; ++t) k += xa[a * A->order + ka.kmode[t]] * ka.kstride[t];
      np_host += nbk[k];
    }
  }
  long long np = 0;
  PoolBuf pc_sorted;
  if (nA > 0 && nB > 0) {
    PoolBuf keyA(pool, nA * 8, s), partA(pool, nA * 8, s), keyB(pool, nB * 8, s), partB(pool, nB * 8, s);
    k_keys<<<grid_for(nA, 256), 256, 0, s>>>(make_meta(A), ka, A->d_ids.as<long long>(), nA,
                                              keyA.as<unsigned long long>(), partA.as<long long>());
    k_keys<<<grid_for(nB, 256), 256, 0, s>>>(make_meta(B), kb, B->d_ids.as<long long>(), nB,
                                              keyB.as<unsigned long long>(), partB.as<long long>());
    SHT_CUDA(cudaGetLastError());
    PoolBuf keyBs, iota(pool, nB * 4, s), permB;
    k_iota<<<grid_for(nB, 256), 256, 0, s>>>(iota.as<int>(), nB);
    // B's blocks are stored by id (column-major over the block grid): when the contracted
    // modes are B's last modes, in order, the keys already ascend in storage order
    bool b_sorted = true;
    for (size_t t = 0; t < mp.rowB.size(); ++t)
      b_sorted = b_sorted && mp.rowB[t] == B->order - (int)mp.rowB.size() + (int)t;
    const int kbits = bits_for(kspan);
    size_t tb = 0;
    if (b_sorted) {
      keyBs = std::move(keyB);
      permB = std::move(iota);
    } else {
      keyBs = PoolBuf(pool, nB * 8, s);
      permB = PoolBuf(pool, nB * 4, s);
      cub::DeviceRadixSort::SortPairs(nullptr, tb, keyB.as<unsigned long long>(), keyBs.as<unsigned long long>(),
                                      iota.as<int>(), permB.as<int>(), (int)nB, 0, kbits, s);
      PoolBuf tmp(pool, tb, s);
      cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, keyB.as<unsigned long long>(), keyBs.as<unsigned long long>(),
                                      iota.as<int>(), permB.as<int>(), (int)nB, 0, kbits, s);
    }
    PoolBuf normA, normB;
    if (eps > 0.0) {
      normA = PoolBuf(pool, nA * 8, s);
      normB = PoolBuf(pool, nB * 8, s);
      tensor_norms_device(A, norm, normA.as<double>(), s);
      tensor_norms_device(B, norm, normB.as<double>(), s);
    }
    PoolBuf lo(pool, nA * 8, s), cnt(pool, nA * 8, s), off(pool, nA * 8, s);
    k_count<<<grid_for(nA, 128), 128, 0, s>>>(keyA.as<unsigned long long>(), nA, keyBs.as<unsigned long long>(),
                                              permB.as<int>(), nB, normA.as<double>(), normB.as<double>(), eps,
                                              lo.as<long long>(), cnt.as<long long>());
    SHT_CUDA(cudaGetLastError());
    cub::DeviceScan::InclusiveSum(nullptr, tb, cnt.as<long long>(), off.as<long long>(), (int)nA, s);
    {
      PoolBuf tmp(pool, tb, s);
      cub::DeviceScan::InclusiveSum(tmp.ptr, tb, cnt.as<long long>(), off.as<long long>(), (int)nA, s);
    }
    if (np_host >= 0) {
      // checked against the device's count at the next read-back (work list)
      np = np_host;
      p->d_npairs = PoolBuf(pool, 8, s);
      SHT_CUDA(cudaMemcpyAsync(p->d_npairs.ptr, off.as<long long>() + nA - 1, 8, cudaMemcpyDeviceToDevice, s));
    } else {
      np = d2h_scalar<long long>(off.as<long long>() + nA - 1, s);
    }
    if (np > (long long)INT32_MAX) fail(SHT_ERR_UNSUPPORTED, "more than 2^31 block pairs");
    if (np > 0) {
      PoolBuf pc(pool, np * 8, s), pa(pool, np * 4, s), pb(pool, np * 4, s);
      k_emit<<<grid_for(nA, 128), 128, 0, s>>>(keyA.as<unsigned long long>(), partA.as<long long>(), nA,
                                               keyBs.as<unsigned long long>(), permB.as<int>(), partB.as<long long>(),
                                               nB, normA.as<double>(), normB.as<double>(), eps, lo.as<long long>(),
                                               off.as<long long>(), cnt.as<long long>(), pc.as<long long>(),
                                               pa.as<int>(), pb.as<int>());
      SHT_CUDA(cudaGetLastError());
      PoolBuf pidx(pool, np * 4, s), porder(pool, np * 4, s);
      pc_sorted = PoolBuf(pool, np * 8, s);
      k_iota<<<grid_for(np, 256), 256, 0, s>>>(pidx.as<int>(), np);
      const int cbits = bits_for((unsigned long long)(cgrid > 1 ? (long long)cgrid - 1 : 1));
      cub::DeviceRadixSort::SortPairs(nullptr, tb, pc.as<long long>(), pc_sorted.as<long long>(), pidx.as<int>(),
                                      porder.as<int>(), (int)np, 0, cbits, s);
      {
        PoolBuf tmp(pool, tb, s);
        cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, pc.as<long long>(), pc_sorted.as<long long>(), pidx.as<int>(),
                                        porder.as<int>(), (int)np, 0, cbits, s);
      }
      p->d_pair_a = PoolBuf(pool, np * 4, s);
      p->d_pair_b = PoolBuf(pool, np * 4, s);
      if (p->mode != SHT_MODE_SPLIT) p->d_recs = PoolBuf(pool, np * sizeof(PairRec), s);
      k_gather_pairs<<<grid_for(np, 256), 256, 0, s>>>(
          porder.as<int>(), pa.as<int>(), pb.as<int>(), np, p->d_pair_a.as<int>(), p->d_pair_b.as<int>(),
          p->d_recs.as<PairRec>(), rec_modes(A->order, mp.rowA, mp.colA), rec_modes(B->order, mp.colB, mp.rowB),
          A->d_offsets.as<long long>(), A->d_dims.as<int>(), B->d_offsets.as<long long>(), B->d_dims.as<int>());
      SHT_CUDA(cudaGetLastError());
    }
  }
  p->npairs = np;
  trace("plan: match+sort pairs", s);

  // result pattern: unique idC ∪ stored C ids
  long long nu = 0;
  PoolBuf uids;
  bool grow = np > 0;
  if (np > 0 && C->nblocks > 0) {
    // the repeated case: every product block is stored already (one count, no sorts)
    PoolBuf miss(pool, 8, s);
    SHT_CUDA(cudaMemsetAsync(miss.ptr, 0, 8, s));
    k_count_missing<<<grid_for(np, 256), 256, 0, s>>>(pc_sorted.as<long long>(), np, C->d_ids.as<long long>(),
                                                       C->nblocks, miss.as<unsigned long long>());
    SHT_CUDA(cudaGetLastError());
    if (speculate) {
      p->d_missing = std::move(miss);
      grow = false;
    } else {
      grow = d2h_scalar<unsigned long long>(miss.ptr, s) > 0;
    }
  }
  if (grow) {
    uids = PoolBuf(pool, np * 8, s);
    PoolBuf counts(pool, np * 4, s), nruns(pool, 8, s);
    size_t tb = 0;
    cub::DeviceRunLengthEncode::Encode(nullptr, tb, pc_sorted.as<long long>(), uids.as<long long>(),
                                       counts.as<int>(), nruns.as<long long>(), (int)np, s);
    PoolBuf tmp(pool, tb, s);
    cub::DeviceRunLengthEncode::Encode(tmp.ptr, tb, pc_sorted.as<long long>(), uids.as<long long>(),
                                       counts.as<int>(), nruns.as<long long>(), (int)np, s);
    nu = d2h_scalar<long long>(nruns.ptr, s);
  }
  const long long nC_old = C->nblocks;
  PoolBuf union_ids;
  long long nunion = nC_old;
  if (nu > 0) {
    if (nC_old == 0) {
      union_ids = std::move(uids);
      nunion = nu;
    } else {
      PoolBuf cat(pool, (nu + nC_old) * 8, s), cats(pool, (nu + nC_old) * 8, s), nsel(pool, 8, s);
      SHT_CUDA(cudaMemcpyAsync(cat.ptr, uids.ptr, nu * 8, cudaMemcpyDeviceToDevice, s));
      SHT_CUDA(cudaMemcpyAsync(cat.as<long long>() + nu, C->d_ids.ptr, nC_old * 8, cudaMemcpyDeviceToDevice, s));
      size_t tb = 0;
      cub::DeviceRadixSort::SortKeys(nullptr, tb, cat.as<long long>(), cats.as<long long>(), (int)(nu + nC_old), 0, 63, s);
      {
        PoolBuf tmp(pool, tb, s);
        cub::DeviceRadixSort::SortKeys(tmp.ptr, tb, cat.as<long long>(), cats.as<long long>(), (int)(nu + nC_old), 0, 63, s);
      }
      union_ids = PoolBuf(pool, (nu + nC_old) * 8, s);
      cub::DeviceSelect::Unique(nullptr, tb, cats.as<long long>(), union_ids.as<long long>(), nsel.as<long long>(),
                                (int)(nu + nC_old), s);
      {
        PoolBuf tmp(pool, tb, s);
        cub::DeviceSelect::Unique(tmp.ptr, tb, cats.as<long long>(), union_ids.as<long long>(), nsel.as<long long>(),
                                  (int)(nu + nC_old), s);
      }
      nunion = d2h_scalar<long long>(nsel.ptr, s);
    }
  }
  if (nunion != nC_old) {
    // re-reserve C to the union pattern
    PoolBuf ndims(pool, std::max(nunion, 1LL) * C->order * 4, s), nsizes(pool, nunion * 8, s),
        noff(pool, nunion * 8, s);
    block_dims_sizes(C, union_ids.as<long long>(), nunion, ndims.as<int>(), nsizes.as<long long>(), s);
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, nsizes.as<long long>(), noff.as<long long>(), (int)nunion, s);
    {
      PoolBuf tmp(pool, tb, s);
      cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, nsizes.as<long long>(), noff.as<long long>(), (int)nunion, s);
    }
    const long long nnz = d2h_scalar<long long>(noff.as<long long>() + nunion - 1, s) +
                          d2h_scalar<long long>(nsizes.as<long long>() + nunion - 1, s);
    PoolBuf ndata(pool, std::max(nnz, 1LL) * 8, s);
    SHT_CUDA(cudaMemsetAsync(ndata.ptr, 0, std::max(nnz, 1LL) * 8, s));
    if (nC_old > 0) {
      const int grid = (int)std::min<long long>(nC_old, (long long)ctx->num_sms * 8);
      k_move_blocks<double><<<grid, 256, 0, s>>>(C->d_data.as<double>(), C->d_ids.as<long long>(),
                                                 C->d_offsets.as<long long>(), C->d_dims.as<int>(), C->order, nC_old,
                                                 union_ids.as<long long>(), nunion, noff.as<long long>(),
                                                 ndata.as<double>());
      SHT_CUDA(cudaGetLastError());
    }
    C->d_ids = std::move(union_ids);
    C->d_offsets = std::move(noff);
    C->d_dims = std::move(ndims);
    C->d_data = std::move(ndata);
    C->nblocks = nunion;
    C->nnz = nnz;
    C->host_stale = true;
    tensor_sync_host(C, s);
  }
  const long long nc = C->nblocks;
  p->ncblk = nc;
  trace("plan: result pattern", s);

  // pair ranges and work list
  p->d_pstart = PoolBuf(pool, (nc + 1) * 4, s);
  k_pstart<<<grid_for(nc + 1, 256), 256, 0, s>>>(C->d_ids.as<long long>(), nc, pc_sorted.as<long long>(), np,
                                                  p->d_pstart.as<int>());
  SHT_CUDA(cudaGetLastError());
  // per C block m, n, sum of the pairs' k and flops; the total flop count
  cblock_stats(p, s);
  trace("plan: pstart+flops", s);
  p->plan_ms += now_ms() - t0;
}

SparseArgs sparse_args(sht_plan* p, double alpha, double beta) {
  const sht_tensor *A = p->A, *B = p->B, *C = p->C;
  SparseArgs g{};
  g.mp = p->tmaps;
  g.sc.alpha = alpha;
  g.sc.beta = beta;
  g.sc.beta_zero = bytes_zero(beta);
  g.sc.alpha_zero = bytes_zero(alpha);
  g.A = A->d_data.as<double>(); g.offA = A->d_offsets.as<long long>(); g.dimsA = A->d_dims.as<int>();
  g.B = B->d_data.as<double>(); g.offB = B->d_offsets.as<long long>(); g.dimsB = B->d_dims.as<int>();
  g.C = C->d_data.as<double>(); g.offC = C->d_offsets.as<long long>(); g.dimsC = C->d_dims.as<int>();
  g.pair_a = p->d_pair_a.as<int>(); g.pair_b = p->d_pair_b.as<int>(); g.pstart = p->d_pstart.as<int>();
  g.recs = p->d_recs.as<PairRec>();
  return g;
}

void plan_touch(sht_plan* p, cudaStream_t s) {
  for (sht_tensor* t : {p->A, p->B, p->C}) tensor_touch(t, s);
  for (PoolBuf* b : {&p->d_pair_a, &p->d_pair_b, &p->d_recs, &p->d_pstart, &p->d_bwork, &p->d_counter, &p->lin_a,
                     &p->lin_b})
    b->use_on(s);
  for (PoolBuf* b : {&p->sp_a, &p->sp_b, &p->sp_ae, &p->sp_be, &p->sp_bsc, &p->sp_meta, &p->sp_items, &p->sp_pairs,
                     &p->sp_rowtab, &p->sp_coltab, &p->sp_rowbase, &p->sp_colbase})
    b->use_on(s);
}

void plan_execute(sht_plan* p, double alpha, double beta, cudaStream_t s) {
  plan_touch(p, s);
  const SparseArgs g = sparse_args(p, alpha, beta);
  if (p->mode == SHT_MODE_SPLIT) split_execute(p, g, s);
  else ring_launch(p, g, s);
}

}  // namespace sht

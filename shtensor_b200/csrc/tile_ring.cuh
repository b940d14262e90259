// tile_ring.cuh -- output-stationary FP64 tiles on the FP64 tensor cores, warp-specialized.
//
// Arithmetic per output element is the reference XMM kernel's (src/Kernel/KernelImpl.cpp:
// 594-619, 661-683): c = beta*c (0 when beta is +0.0), then for every pair in order and every
// contracted index k ascending, c = fma(alpha*a_ik, b_kj, c).  The products run on
// mma.sync.m8n8k4.f64: on sm_100a one m8n8k4 step accumulates its four k in ascending order
// with one rounding each (measured bit-identical to the fma chain over 1.28M outputs), so
// feeding k ascending keeps the results bit-identical to the CPU restatement.  A contracted
// extent that is not a multiple of 4 is padded in registers with a = -0.0, b = +0.0:
// fma(-0, +0, c) == c for every c, signed zeros included.
//
// A CTA of twelve warps (one idle) walks tiles of C blocks:
//   warps 0-7  multiply: a 2x4 grid of warps over a tile of up to 64 x 64; every warp owns up to 4x2
//              fragments of 8x8, interleaved (fragment f of grid row w covers rows (2f + w)*8 ..),
//              so a tile whose extents are not multiples of 32 is shared out evenly and
//              fragments outside it are skipped;
//   warps 8-9  load, one operand each: copy the operands straight from the blocks' own column-major
//              layouts with cp.async into a three-stage ring of 32-deep k-chunks.  Blocks and
//              their rows start at any element; a row that starts at an odd one is copied with
//              its stage row shifted by one, so that 16-byte copies serve every row;
//   warp 10    schedule: claims tiles, resolves their C offset tables and block pairs ahead of
//              the loaders, so that the dependent global loads of a tile's start (work item ->
//              pair range -> pair -> block) are off the multiply warps' path.
// A C block of m rows is cut into ceil(m / 64) row tiles of equal size rounded up to 8 (columns
// likewise): 65 rows are 40 + 25, not 64 + 1.
//
// Bound: the FP64 tensor pipe (one m8n8k4 per 16 cycles and SM sub-partition; 37.1 TFLOP/s), then the
// hand-over between the roles on small tiles.  Two CTAs per SM give every sub-partition four multiply
// warps, so one tile's epilogue and start overlap the other's products.  Measured, whole contraction
// of iaP,jbP->ijab (111.7 GFLOP, 250,514 tiles, mean 45 x 45 x 75): 5.05 ms, against 15.6 ms for a
// DFMA tile with per-element gathers and 6.3 ms for a DMMA tile over operands copied into matrix form
// first (k_tiles itself 4.85 ms: 66% of the pipe with the padding to 8); abcd,cdij->abij (154.8
// GFLOP, 36 C blocks): 6.38 ms against 7.28 ms.
#pragma once

#include "mbar.cuh"
#include "tile_core.cuh"

namespace sht {

constexpr int kRingK = 32;        // k-depth of one stage
constexpr int kRingStages = 3;
constexpr int kRingTile = 64;     // rows and columns of a tile, at most
// Stage layouts, pitches chosen so that both the copies and the fragment loads (8 rows x 4 k per
// warp) spread over the shared-memory banks: rows fastest, k-row pitch 68; or, for an operand whose
// blocks have the contracted index fastest, k fastest, row pitch 36.
constexpr int kRingPitchR = kRingTile + 4, kRingPitchK = kRingK + 4;
constexpr int kRingOperandD = kRingTile * kRingPitchK;  // doubles of one operand's part (the larger layout)
static_assert(kRingOperandD >= kRingK * kRingPitchR, "both layouts fit");
constexpr int kRingTileSlots = 4, kRingPairSlots = 8;
constexpr int kRingMmaWarps = 8, kRingLoadWarps = 2;
constexpr int kRingThreads = 32 * (kRingMmaWarps + 4);  // and the load, schedule and one idle warp
constexpr int kRingCtas = 2;      // per SM

// How the operands and C are addressed (from the expression, the same for every block):
constexpr int kRingLinA = 1, kRingLinB = 2;  // element (row, k) at row * rs + k * ks, rs or ks 1; data 16-byte aligned
constexpr int kRingKmA = 4, kRingKmB = 8;    // stage layout with k fastest (linear: ks == 1, else rs == 1)
constexpr int kRingLinR = 16, kRingLinC = 32;  // C rows / columns at index * stride

struct RingArgs {
  TileMaps mp;
  TileScalars<double> sc;
  int flags;
  const double* A; const long long* offA; const int* dimsA;
  const double* B; const long long* offB; const int* dimsB;
  double* C; const long long* offC; const int* dimsC;
  const PairRec* recs;     // pairs in canonical order
  const int* pstart;       // pair range of every C block
  const int4* work;        // ring_item
  int nwork;
  unsigned* counter;       // next item (stacks: items are strided over the grid)
  // several requests in one launch: request r owns items [multi[r].first, +multi[r].nwork)
  const RingArgs* multi;
  int nmulti, first;
  // stacks: equal blocks, one pair per C block (its extents and strides in `stack`)
  PairRec stack;
  long long size_a, size_b, size_c;
  int sdA[kMaxOrder], sdB[kMaxOrder], sdC[kMaxOrder];
  int tiles_per_op, m, n;
  volatile int* err;       // the context's error word: SHT_ERR_TIMEOUT
  long long wait_limit;    // polls of one wait before the launch gives up
};
constexpr int kRingPlan = 0, kRingMulti = 1, kRingStack = 2;

struct RingTile {
  double* c;
  const RingArgs* g;
  double alpha, beta;
  int np, mt, nt, r0, c0, flags, beta_zero;
  int rowoff[kRingTile], coloff[kRingTile];
};
struct RingPair {
  const double *a, *b;      // linear: element (first row of the tile, k = 0); else the block
  const int *da, *db;       // block extents (for the gathers that are not linear)
  int K, rsA, ksA, rsB, ksB;
  int parA, parB;           // bit 0: parity of a (b) in elements, bit 1: of its shift's stride
};

struct RingSmem {
  double stage[kRingStages][2][kRingOperandD];  // A, B
  RingTile tile[kRingTileSlots];
  RingPair pair[kRingPairSlots];
  unsigned long long full[kRingStages], empty[kRingStages];
  unsigned long long tfull[kRingTileSlots], tempty[kRingTileSlots];
  unsigned long long pfull[kRingPairSlots], pempty[kRingPairSlots];
  int abort;
};

struct RingWait {
  volatile int* abort;
  volatile int* err;
  long long limit;
  // true once the phase is complete; the first try is the usual case, later ones suspend the warp
  // for up to a microsecond each
  __device__ __forceinline__ bool operator()(unsigned long long* bar, unsigned parity) const {
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait_suspended(bar, parity, abort, limit, err));
  }
};

// ------------------------------------------------------------------ schedule warp
// The work entry and block header of one item, loaded ahead of its use.
struct RingHead {
  const RingArgs* g;
  double* c;
  int r0, c0, mt, nt, ps, pe, cblk;
  int dim;  // lane d: extent of the block's mode d
};

template <int Kind>
__device__ __forceinline__ int4 ring_work(const RingArgs& g, unsigned item, const RingArgs*& r, int lane) {
  r = &g;
  if (item >= (unsigned)g.nwork) return make_int4(0, 0, 0, 0);
  if constexpr (Kind == kRingStack) {
    return ring_item((int)(item / g.tiles_per_op), (int)(item % g.tiles_per_op), g.m, g.n, kRingTile, kRingTile);
  } else if constexpr (Kind == kRingMulti) {
    int lo = 0, n = g.nmulti;  // the last request whose first item is <= item, 32 ways at a time
    while (n > 1) {
      const int step = (n + 31) >> 5, off = lane * step;
      const bool le = off < n && (unsigned)g.multi[lo + off].first <= item;
      const int last = 31 - __clz(__ballot_sync(0xffffffffu, le));
      lo += last * step;
      n = min(step, n - last * step);
    }
    r = g.multi + lo;
    return r->work[item - r->first];
  } else {
    return g.work[item];
  }
}

template <int Kind>
__device__ __forceinline__ RingHead ring_head(const RingArgs* r, int4 w, int lane) {
  RingHead h;
  h.g = r;
  h.cblk = w.x;
  h.r0 = w.y;
  h.c0 = w.z;
  h.mt = w.w & 0xffff;
  h.nt = w.w >> 16;
  if constexpr (Kind == kRingStack) {
    h.c = r->C + (long long)w.x * r->size_c;
    h.ps = 0;
    h.pe = 1;
    h.dim = lane < r->mp.oC ? r->sdC[lane] : 1;
  } else {
    h.c = r->C + r->offC[w.x];
    h.ps = r->pstart[w.x];
    h.pe = r->pstart[w.x + 1];
    h.dim = lane < r->mp.oC ? r->dimsC[(long long)w.x * r->mp.oC + lane] : 1;
  }
  return h;
}

// Offsets of `cnt` consecutive indices (from i0) of one C dimension into out.
__device__ __forceinline__ void ring_offsets(const ModeMap& mm, bool linear, int dim, int stride, int i0, int cnt,
                                             int* out, int lane) {
  if (linear) {
    const int s = mm.n ? __shfl_sync(0xffffffffu, stride, mm.y[0]) : 1;
    for (int i = lane; i < cnt; i += 32) out[i] = (i0 + i) * s;
    return;
  }
  int idx[2], off[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    idx[j] = i0 + lane + 32 * j;
    off[j] = 0;
  }
  for (int t = 0; t < mm.n; ++t) {
    const int e = __shfl_sync(0xffffffffu, dim, mm.y[t]), s = __shfl_sync(0xffffffffu, stride, mm.y[t]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int q = t + 1 < mm.n ? idx[j] / e : 0;  // the last digit is what is left
      off[j] += (idx[j] - q * e) * s;
      idx[j] = q;
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (lane + 32 * j < cnt) out[lane + 32 * j] = off[j];
}

// position of an element within its 16-byte unit
__device__ __forceinline__ int ring_parity(const double* p) { return (int)(reinterpret_cast<size_t>(p) >> 3) & 1; }

template <int Kind>
__device__ __forceinline__ void ring_schedule(const RingArgs& g, RingSmem& sm, int lane, const RingWait& wait) {
  // an item is claimed one tile ahead of its use; raw: the claim as issued (lane 0 holds it)
  unsigned last = blockIdx.x;
  auto claim = [&]() -> unsigned {
    if constexpr (Kind == kRingStack) {
      const unsigned it = last;
      last = it > 0x7fffffffu ? it : it + gridDim.x;
      return it;
    }
    return lane == 0 ? atomicAdd(g.counter, 1u) : 0u;
  };
  auto resolve = [&](unsigned raw) { return __shfl_sync(0xffffffffu, raw, 0); };
  const RingArgs* r;
  unsigned it0 = resolve(claim()), raw1 = claim();
  int4 w = ring_work<Kind>(g, it0, r, lane);
  RingHead h{};
  if (it0 < (unsigned)g.nwork) h = ring_head<Kind>(r, w, lane);
  unsigned nt = 0, q = 0;
  bool ok = true;
  while (ok && it0 < (unsigned)g.nwork) {
    const int ts = (int)(nt % kRingTileSlots);
    if (!wait(&sm.tempty[ts], (unsigned)(((nt / kRingTileSlots) & 1) ^ 1))) { ok = false; break; }
    ++nt;
    const unsigned it1 = resolve(raw1);
    raw1 = claim();
    const RingArgs& a = *h.g;
    const int np = a.sc.alpha_zero ? 0 : h.pe - h.ps;
    PairRec rec{};
    if (Kind != kRingStack && lane < np) rec = a.recs[h.ps + lane];
    // the next item's work entry, in flight meanwhile
    const int4 w1 = ring_work<Kind>(g, it1, r, lane);
    // C offset tables
    int stride = 1;
    for (int d = 0; d + 1 < a.mp.oC; ++d) {
      const int e = __shfl_sync(0xffffffffu, h.dim, d);
      if (d < lane) stride *= e;
    }
    const int r0 = h.r0, c0 = h.c0, mt = h.mt, nc = h.nt;
    RingTile& t = sm.tile[ts];
    ring_offsets(a.mp.row, (a.flags & kRingLinR) != 0, h.dim, stride, r0, mt, t.rowoff, lane);
    ring_offsets(a.mp.col, (a.flags & kRingLinC) != 0, h.dim, stride, c0, nc, t.coloff, lane);
    if (lane == 0) {
      t.c = h.c;
      t.g = h.g;
      t.alpha = a.sc.alpha;
      t.beta = a.sc.beta;
      t.beta_zero = a.sc.beta_zero;
      t.np = np;
      t.mt = mt;
      t.nt = nc;
      t.r0 = r0;
      t.c0 = c0;
      t.flags = a.flags;
    }
    mbar_arrive(&sm.tfull[ts]);  // release: this lane's stores come first
    const int ps = h.ps, op = h.cblk;
    RingHead h1{};
    if (it1 < (unsigned)g.nwork) h1 = ring_head<Kind>(r, w1, lane);
    // the pairs, 32 at a time
    for (int base = 0; ok && base < np; base += 32) {
      const int cnt = min(32, np - base);
      RingPair p{};
      if (lane < cnt) {
        if constexpr (Kind == kRingStack) {
          p.a = a.A + (long long)op * a.size_a;
          p.b = a.B + (long long)op * a.size_b;
          p.da = a.sdA;
          p.db = a.sdB;
          rec = a.stack;
        } else {
          if (base > 0) rec = a.recs[ps + base + lane];
          p.a = a.A + rec.offA;
          p.b = a.B + rec.offB;
          p.da = a.dimsA + (long long)rec.ia * a.mp.oA;
          p.db = a.dimsB + (long long)rec.ib * a.mp.oB;
        }
        p.K = rec.K;
        p.rsA = rec.rsA;
        p.ksA = rec.ksA;
        p.rsB = rec.rsB;
        p.ksB = rec.ksB;
        if (a.flags & kRingLinA) {
          p.a += (long long)r0 * p.rsA;
          p.parA = ring_parity(p.a) | ((a.flags & kRingKmA ? p.rsA : p.ksA) & 1) << 1;
        }
        if (a.flags & kRingLinB) {
          p.b += (long long)c0 * p.rsB;
          p.parB = ring_parity(p.b) | ((a.flags & kRingKmB ? p.rsB : p.ksB) & 1) << 1;
        }
      }
      for (int j = 0; ok && j < cnt; ++j, ++q) {
        const int qs = (int)(q % kRingPairSlots);
        ok = wait(&sm.pempty[qs], (unsigned)(((q / kRingPairSlots) & 1) ^ 1));
        if (ok && lane == j) {
          sm.pair[qs] = p;
          mbar_arrive(&sm.pfull[qs]);  // release: the record's stores come first
        }
      }
    }
    h = h1;
    it0 = it1;
  }
  if (ok) {
    const int ts = (int)(nt % kRingTileSlots);
    if (wait(&sm.tempty[ts], (unsigned)(((nt / kRingTileSlots) & 1) ^ 1))) {
      if (lane == 0) sm.tile[ts].np = -1;
      mbar_arrive(&sm.tfull[ts]);
    }
  }
}

// ------------------------------------------------------------------ load warps
__device__ __forceinline__ void ring_cp8(double* smem, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
// 16 bytes, of which only the first `bytes` are read (the rest is zero-filled)
__device__ __forceinline__ void ring_cp16(double* smem, const double* gmem, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes)
               : "memory");
}

// A chunk of an operand whose rows are contiguous: k-row k is copied as 16-byte pairs into the
// stage row shifted by the parity of its first element, so that source and destination have the
// same alignment.  A pair may start one element before the row (the other half of a 16-byte unit
// of the tensor) and never reads past its end.  par: bit 0 the parity of src, bit 1 that of ks.
__device__ __forceinline__ void ring_copy_rows(double* dst, const double* src, int ks, int rows, int kc, int par,
                                               int lane) {
  const bool narrow = rows < 32;  // 16 pairs and two k per instruction
  const int j = narrow ? lane & 15 : lane;
  const long long step = 2LL * ks;
  for (int h = 0; h < 2; ++h) {
    const int kh = narrow ? lane >> 4 : h;  // this lane's k: kh, kh + 2, ..
    const int sh = (par ^ (kh & (par >> 1))) & 1;
    const int odd = sh && (rows & 63) == 0 ? 1 : 0;  // whole rounds of 32 pairs end one element short
    for (int e = 2 * j - sh; e < rows - odd; e += 64) {
      const int bytes = e + 1 < rows ? 16 : 8;
      const double* s = src + e + (long long)kh * ks;
      double* d = dst + e + sh + kh * kRingPitchR;
      int i = 0;
      for (; kh + 2 * i + 14 < kc; i += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) ring_cp16(d + 2 * (i + u) * kRingPitchR, s + (i + u) * step, bytes);
      }
      for (; kh + 2 * i < kc; ++i) ring_cp16(d + 2 * i * kRingPitchR, s + i * step, bytes);
      if (odd && j == 31 && e + 64 >= rows)
        for (int i = 0; kh + 2 * i < kc; ++i) ring_cp8(d + 2 + 2 * i * kRingPitchR, s + 2 + i * step);
    }
    if (narrow) break;
  }
}

// The same for an operand with the contracted index contiguous: k pairs over the lanes, several rows per
// instruction; a shifted row of a whole chunk needs its last element on its own.  par: bit 0 the
// parity of src, bit 1 that of the row stride rs.
__device__ __forceinline__ void ring_copy_k(double* dst, const double* src, int rs, int rows, int kc, int par,
                                            int lane) {
  constexpr int kPairs = kRingK / 2, kRows = 32 / kPairs;
  const int r = lane / kPairs, j = lane % kPairs;
  const int sh = (par ^ (r & (par >> 1))) & 1;  // kRows is even: a lane's rows have one parity
  const int e = 2 * j - sh;
  const int bytes = e >= kc ? 0 : e + 1 < kc ? 16 : 8;
  const bool last = sh && j == kPairs - 1 && kc == kRingK;
  if (bytes == 0) return;
  const double* s = src + (long long)r * rs;
  double* d = dst + r * kRingPitchK;
  const long long step = (long long)kRows * rs;
  const int n = (rows - r + kRows - 1) / kRows;
  int i = 0;
  for (; i + 4 <= n; i += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      ring_cp16(d + kRows * u * kRingPitchK + 2 * j, s + u * step + e, bytes);
      if (last) ring_cp8(d + kRows * u * kRingPitchK + kRingK, s + u * step + kRingK - 1);
    }
    s += 4 * step;
    d += 4 * kRows * kRingPitchK;
  }
  for (; i < n; ++i) {
    ring_cp16(d + 2 * j, s + e, bytes);
    if (last) ring_cp8(d + kRingK, s + kRingK - 1);
    s += step;
    d += kRows * kRingPitchK;
  }
}

// Any order of modes, or data that is not 16-byte aligned: a pair's elements copied one by one through
// offsets (rows-fastest stage layout, no shift).  Lane d holds extent and stride of the block's mode d.
//
// Offset of combined index idx of the modes xs[0 .. n); all lanes take part.
__device__ __forceinline__ int ring_digits(const int* xs, int n, int idx, int ext, int stride) {
  int off = 0;
  for (int t = 0; t < n; ++t) {
    const int x = xs[t];
    const int e = __shfl_sync(0xffffffffu, ext, x), s = __shfl_sync(0xffffffffu, stride, x);
    const int q = t + 1 < n ? idx / e : 0;  // the last digit is what is left
    off += (idx - q * e) * s;
    idx = q;
  }
  return off;
}

// All chunks of one pair from stage st on; false when a wait ran out.  The extents are loaded and the row
// offsets worked out once per pair (with that done per chunk, the extents loaded again for every mode, a
// chunk took up to 9,000 cycles: abcd,cidj->abij, 281 GFLOP, 16.9 ms, now 13.1).  Lanes run along the rows
// of one k, or (kfast: the contracted index's first mode is the block's fastest) along the k of one row,
// two or four of them at a time when they are few.
static __device__ __noinline__ bool ring_gather(RingSmem& sm, bool isb, bool kfast, const RingArgs* g, const double* src,
                                                const int* dims, int r0, int rows, int K, int st, unsigned ph, int lane) {
  const RingWait wait{&sm.abort, g->err, g->wait_limit};
  const int order = isb ? g->mp.oB : g->mp.oA;
  const ModeMap& fm = isb ? g->mp.col : g->mp.row;
  const int* kx = isb ? g->mp.kk.y : g->mp.kk.x;
  const int nk = g->mp.kk.n;
  const int ext = lane < order ? dims[lane] : 1;
  int stride = 1;
  for (int d = 0; d + 1 < order; ++d) {
    const int e = __shfl_sync(0xffffffffu, ext, d);
    if (d < lane) stride *= e;
  }
  // lane i: offsets of rows i and 32 + i
  const int ra = ring_digits(fm.x, fm.n, r0 + lane, ext, stride);
  const int rb = rows > 32 ? ring_digits(fm.x, fm.n, r0 + 32 + lane, ext, stride) : 0;
  for (int k0 = 0; k0 < K; k0 += kRingK) {
    const int kc = min(kRingK, K - k0);
    const int ko = ring_digits(kx, nk, k0 + lane, ext, stride);  // lane k: offset of k0 + k
    if (!wait(&sm.empty[st], ph ^ 1u)) return false;
    // `inner` indices over 2^w lanes, 32 >> w outer ones at once
    const int inner = kfast ? kc : min(rows, 32), outer = kfast ? rows : kc;
    const int w = inner <= 8 ? 3 : inner <= 16 ? 4 : 5, step = 32 >> w;
    const int i = lane & ((1 << w) - 1), o0 = lane >> w;
    const int pitch = kfast ? kRingPitchK : kRingPitchR;
    double* d = sm.stage[st][isb ? 1 : 0] + i + o0 * pitch;
    const int mine = __shfl_sync(0xffffffffu, kfast ? ko : ra, i);
    const double *s0 = src + mine, *s1 = src + rb;
    const bool in0 = i < inner, in1 = !kfast && 32 + lane < rows;
#pragma unroll 4
    for (int o = 0; o < outer; o += step) {
      const int at = o + o0;
      int off = __shfl_sync(0xffffffffu, kfast ? ra : ko, at & 31);
      if (kfast && o >= 32) off = __shfl_sync(0xffffffffu, rb, at & 31);
      if (at < outer) {
        if (in0) ring_cp8(d + o * pitch, s0 + off);
        if (in1) ring_cp8(d + o * pitch + 32, s1 + off);
      }
    }
    mbar_arrive_cp_async(&sm.full[st]);
    if (++st == kRingStages) {
      st = 0;
      ph ^= 1u;
    }
  }
  return true;
}

// One load warp per operand; both run this code.  Gather: some operand needs ring_gather (an instance of
// its own: its code beside the linear copies' costs those 2 to 8%).
template <bool Gather>
__device__ __forceinline__ void ring_load(RingSmem& sm, bool isb, int lane, const RingWait& wait) {
  int st = 0;
  unsigned ph = 0, q = 0;
  bool ok = true;
  for (unsigned nt = 0; ok; ++nt) {
    const int ts = (int)(nt % kRingTileSlots);
    if (!wait(&sm.tfull[ts], (nt / kRingTileSlots) & 1)) break;
    const RingTile& t = sm.tile[ts];
    const RingArgs* g = t.g;
    const int np = t.np, rows = isb ? t.nt : t.mt, r0 = isb ? t.c0 : t.r0;
    const bool km = t.flags & (isb ? kRingKmB : kRingKmA), lin = t.flags & (isb ? kRingLinB : kRingLinA);
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tempty[ts]);
    if (np < 0) break;
    for (int p = 0; ok && p < np; ++p, ++q) {
      const int qs = (int)(q % kRingPairSlots);
      if (!wait(&sm.pfull[qs], (q / kRingPairSlots) & 1)) { ok = false; break; }
      const RingPair& v = sm.pair[qs];
      const double* src = isb ? v.b : v.a;
      const int* dims = isb ? v.db : v.da;
      const int rs = isb ? v.rsB : v.rsA, ks = isb ? v.ksB : v.ksA, par = isb ? v.parB : v.parA, K = v.K;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.pempty[qs]);
      if (Gather && !lin) {
        ok = ring_gather(sm, isb, km, g, src, dims, r0, rows, K, st, ph, lane);
        for (int k0 = 0; k0 < K; k0 += kRingK)
          if (++st == kRingStages) {
            st = 0;
            ph ^= 1u;
          }
        continue;
      }
      for (int k0 = 0; k0 < K; k0 += kRingK) {
        const int kc = min(kRingK, K - k0);
        if (!wait(&sm.empty[st], ph ^ 1u)) { ok = false; break; }
        double* d = sm.stage[st][isb ? 1 : 0];
        if (km) ring_copy_k(d, src + k0, rs, rows, kc, par, lane);
        else ring_copy_rows(d, src + (long long)k0 * ks, ks, rows, kc, par, lane);
        mbar_arrive_cp_async(&sm.full[st]);
        if (++st == kRingStages) {
          st = 0;
          ph ^= 1u;
        }
      }
    }
  }
  // copies still in flight (after a wait that ran out) write into this CTA's shared memory
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// ------------------------------------------------------------------ multiply warps
struct RingCursor {
  int st;
  unsigned ph, q;
};

// Up to 4x2 fragments of one k-step of four.  Rows past ml and a second column are skipped by uniform
// branches inside the instruction block.  (A predicated-off m8n8k4 or FP64 multiplication takes its
// 16 or 2 cycles of the pipe all the same; one unrolled body per size measured up to 2x slower on
// tiles of mixed sizes, the warps of an SM then run different loops and wait for instructions; and
// branches written outside the block cost 1.4x, each becomes a point of reconvergence.)
#define SHT_MMA(c0, c1, a, b) \
  "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%" #c0 ",%" #c1 "}, {%" #a "}, {%" #b "}, {%" #c0 ",%" #c1 "};\n\t"
__device__ __forceinline__ void dmma_4x2(double (&d)[4][2][2], const double (&a)[4], const double (&b)[2], int ml,
                                         int nl) {
  asm volatile(
      "{\n\t.reg .pred q1, q2, q3, q;\n\t"
      "setp.lt.s32 q, %23, 2;\n\t"
      "setp.lt.s32 q1, %22, 2;\n\t"
      "setp.lt.s32 q2, %22, 3;\n\t"
      "setp.lt.s32 q3, %22, 4;\n\t"
      "@q bra.uni SHT_ONE;\n\t"
      SHT_MMA(0, 1, 16, 20) SHT_MMA(2, 3, 16, 21)
      "@q1 bra.uni SHT_END;\n\t"
      SHT_MMA(4, 5, 17, 20) SHT_MMA(6, 7, 17, 21)
      "@q2 bra.uni SHT_END;\n\t"
      SHT_MMA(8, 9, 18, 20) SHT_MMA(10, 11, 18, 21)
      "@q3 bra.uni SHT_END;\n\t"
      SHT_MMA(12, 13, 19, 20) SHT_MMA(14, 15, 19, 21)
      "bra.uni SHT_END;\n\t"
      "SHT_ONE:\n\t"
      SHT_MMA(0, 1, 16, 20)
      "@q1 bra.uni SHT_END;\n\t"
      SHT_MMA(4, 5, 17, 20)
      "@q2 bra.uni SHT_END;\n\t"
      SHT_MMA(8, 9, 18, 20)
      "@q3 bra.uni SHT_END;\n\t"
      SHT_MMA(12, 13, 19, 20)
      "SHT_END:\n\t}\n"
      : "+d"(d[0][0][0]), "+d"(d[0][0][1]), "+d"(d[0][1][0]), "+d"(d[0][1][1]), "+d"(d[1][0][0]), "+d"(d[1][0][1]),
        "+d"(d[1][1][0]), "+d"(d[1][1][1]), "+d"(d[2][0][0]), "+d"(d[2][0][1]), "+d"(d[2][1][0]), "+d"(d[2][1][1]),
        "+d"(d[3][0][0]), "+d"(d[3][0][1]), "+d"(d[3][1][0]), "+d"(d[3][1][1])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]), "r"(ml), "r"(nl));
}
#undef SHT_MMA

// One k-step of four.  AF / BF: distance of two fragments of the warp in a stage.
template <int AF, int BF, bool Scale, bool Tail>
__device__ __forceinline__ void ring_step4(const double* sa, const double* sb, double alpha, int ml, int nl, bool dead,
                                           double (&acc)[4][2][2]) {
  double af[4], bf[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) af[i] = sa[i * AF];
#pragma unroll
  for (int i = 0; i < 2; ++i) bf[i] = sb[i * BF];
  if (Scale) {
#pragma unroll
    for (int i = 0; i < 4; ++i) af[i] = mul_rn(alpha, af[i]);
  }
  if (Tail) {  // past the contracted extent
#pragma unroll
    for (int i = 0; i < 4; ++i) af[i] = dead ? -0.0 : af[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) bf[i] = dead ? 0.0 : bf[i];
  }
  dmma_4x2(acc, af, bf, ml, nl);
}

// All pairs of one tile into the warp's ml x nl fragments (a warp without fragments in this tile only
// passes the stages on).  Ka / Kb: operand stages with k fastest; Scale: alpha is not 1 (an instance of
// its own: four multiplications per step, even predicated off, cost 12% of the pipe).
template <bool Ka, bool Kb, bool Scale>
__device__ __forceinline__ bool ring_products(RingSmem& sm, int np, RingCursor& cu, double alpha, int ml, int nl,
                                              int wi, int wj, int lane, double (&acc)[4][2][2], const RingWait& wait) {
  constexpr int AR = Ka ? kRingPitchK : 1, AK = Ka ? 1 : kRingPitchR;  // distance of two rows, two k
  constexpr int BR = Kb ? kRingPitchK : 1, BK = Kb ? 1 : kRingPitchR;
  const int fr = lane >> 2, kq = lane & 3;
  const int aoff = (wi * 8 + fr) * AR + kq * AK, boff = (wj * 8 + fr) * BR + kq * BK;
  // which parity bit of the lane its stage row has: of its k, or (k fastest) of its row
  const int abit = Ka ? fr & 1 : kq & 1, bbit = Kb ? fr & 1 : kq & 1;
  for (int p = 0; p < np; ++p, ++cu.q) {
    const unsigned qs = cu.q % kRingPairSlots;
    if (!wait(&sm.pfull[qs], (cu.q / kRingPairSlots) & 1)) return false;
    const int K = sm.pair[qs].K, pra = sm.pair[qs].parA, prb = sm.pair[qs].parB;
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.pempty[qs]);
    // the shift of this lane's stage rows
    const int ao = aoff + ((pra ^ (abit & (pra >> 1))) & 1), bo = boff + ((prb ^ (bbit & (prb >> 1))) & 1);
    for (int k0 = 0; k0 < K; k0 += kRingK) {
      if (!wait(&sm.full[cu.st], cu.ph)) return false;
      if (ml > 0 && nl > 0) {
        const int kc = min(kRingK, K - k0);
        const double* sa = sm.stage[cu.st][0] + ao;
        const double* sb = sm.stage[cu.st][1] + bo;
#pragma unroll 1
        for (int k = 4; k <= kc; k += 4) {
          ring_step4<16 * AR, 32 * BR, Scale, false>(sa, sb, alpha, ml, nl, false, acc);
          sa += 4 * AK;
          sb += 4 * BK;
        }
        if (kc & 3) ring_step4<16 * AR, 32 * BR, Scale, true>(sa, sb, alpha, ml, nl, kq >= (kc & 3), acc);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.empty[cu.st]);
      if (++cu.st == kRingStages) {
        cu.st = 0;
        cu.ph ^= 1u;
      }
    }
  }
  return true;
}

__device__ __forceinline__ void ring_multiply(RingSmem& sm, int warp, int lane, const RingWait& wait) {
  RingCursor cu{0, 0u, 0u};
  const int fr = lane >> 2, fq = lane & 3;  // fragment row, k (operands) / column pair (C)
  for (unsigned nt = 0;; ++nt) {
    const int ts = (int)(nt % kRingTileSlots);
    if (!wait(&sm.tfull[ts], (unsigned)((nt / kRingTileSlots) & 1))) return;
    const RingTile& t = sm.tile[ts];
    const int np = t.np, mt = t.mt, nc = t.nt, flags = t.flags;
    if (np < 0) return;
    // the warp with the most fragments moves over the sub-partitions from tile to tile
    // (in reverse order in the grid's second half, whose CTAs share SMs with the first half's)
    const int v = (warp + (int)nt) & (kRingMmaWarps - 1), w = blockIdx.x * 2 >= gridDim.x ? kRingMmaWarps - 1 - v : v;
    const int wi = w & 1, wj = w >> 1;
    const int ml = ((mt + 7) / 8 - wi + 1) >> 1, nl = ((nc + 7) / 8 - wj + 3) >> 2;
    const int row0 = wi * 8 + fr, col0 = wj * 8;
    const double beta = t.beta, alpha = t.alpha;
    double* c = t.c;
    double acc[4][2][2];
    if (t.beta_zero) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = row0 + i * 16, s = col0 + j * 32 + 2 * fq + e;
            acc[i][j][e] = r < mt && s < nc ? mul_rn(beta, c[t.rowoff[r] + t.coloff[s]]) : 0.0;
          }
    }
    bool ok;
    switch ((flags & (kRingKmA | kRingKmB)) | (alpha != 1.0 ? 1 : 0)) {
#define SHT_RING_CASE(KA, KB)                                                                                         \
  case (KA ? kRingKmA : 0) | (KB ? kRingKmB : 0):                                                                     \
    ok = ring_products<KA, KB, false>(sm, np, cu, alpha, ml, nl, wi, wj, lane, acc, wait);                            \
    break;                                                                                                            \
  case (KA ? kRingKmA : 0) | (KB ? kRingKmB : 0) | 1:                                                                 \
    ok = ring_products<KA, KB, true>(sm, np, cu, alpha, ml, nl, wi, wj, lane, acc, wait);                             \
    break;
      SHT_RING_CASE(false, false)
      SHT_RING_CASE(true, false)
      SHT_RING_CASE(false, true)
      SHT_RING_CASE(true, true)
#undef SHT_RING_CASE
      default: return;
    }
    if (!ok) return;
    // each store covers 8 rows x 4 columns; streaming, so that C does not evict the operands
    int co[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int s = col0 + j * 32 + 2 * fq + e;
        co[j][e] = s < nc ? t.coloff[s] : -1;
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = row0 + i * 16;
      if (r < mt) {
        double* cr = c + t.rowoff[r];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (co[j][e] >= 0) __stcs(cr + co[j][e], acc[i][j][e]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tempty[ts]);
  }
}

template <int Kind, bool Gather>
__global__ void __launch_bounds__(kRingThreads, kRingCtas) k_tiles(const __grid_constant__ RingArgs g) {
  extern __shared__ __align__(16) unsigned char ring_smem[];
  RingSmem& sm = *reinterpret_cast<RingSmem*>(ring_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRingStages; ++i) {
      mbar_init(&sm.full[i], 32 * kRingLoadWarps);
      mbar_init(&sm.empty[i], kRingMmaWarps);
    }
    for (int i = 0; i < kRingTileSlots; ++i) {
      mbar_init(&sm.tfull[i], 32);
      mbar_init(&sm.tempty[i], kRingMmaWarps + kRingLoadWarps);
    }
    for (int i = 0; i < kRingPairSlots; ++i) {
      mbar_init(&sm.pfull[i], 1);
      mbar_init(&sm.pempty[i], kRingMmaWarps + kRingLoadWarps);
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const RingWait wait{&sm.abort, g.err, g.wait_limit};
  if (warp < kRingMmaWarps) {
    ring_multiply(sm, warp, lane, wait);
  } else {
    if (warp < kRingMmaWarps + kRingLoadWarps) ring_load<Gather>(sm, warp > kRingMmaWarps, lane, wait);
    else if (warp == kRingMmaWarps + kRingLoadWarps) ring_schedule<Kind>(g, sm, lane, wait);
  }
}

}  // namespace sht

// stack.cu -- Kernel<T>::call on the device: nb_ops same-shape (A, B, C) block triples.
//
// Replaces the two CPU back ends of src/Kernel/KernelImpl.cpp (LAPACK reshape+gemm, :75-208,
// and the asmjit AVX2 gather/FMA/scatter microkernel, :210-770).  The permutes are fused into the
// operand reads and the per-element arithmetic is the XMM kernel's (k ascending, one fma each), so
// results are bit-identical to the CPU restatement.  Three kernels:
//   * blocks whose A and B fit in shared memory (staged_fits): a CTA takes one op after
//     another, copies the next op's two blocks whole -- contiguous, whatever the index order --
//     while it multiplies the current one from shared memory through offset tables built once
//     (with few ops several CTAs share one);
//     FP64 on the tensor cores (k_stack_dmma), FP32 with FFMA register tiles (k_stack_fma);
//   * larger FP64 blocks: the ring tile kernel (tile_ring.cuh), one pair per C block;
//   * larger FP32 blocks: the gathering tile (tile_core.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <tuple>

#include "contract.h"
#include "device_common.cuh"
#include "tile_core.cuh"
#include "tile_pipe.cuh"
#include "tile_ring.cuh"

namespace sht {

template <typename T>
struct StackArgs {
  TileMaps mp;
  TileScalars<T> sc;
  const T* A; const T* B; T* C;
  long long size_a, size_b, size_c;
  int dimsA[kMaxOrder], dimsB[kMaxOrder], dimsC[kMaxOrder];
  int tiles_per_op;
};

template <typename T, class Cfg>
__global__ void __launch_bounds__(Cfg::kThreads) k_stack(StackArgs<T> g) {
  __shared__ TileSmem<T, Cfg> sm;
  const long long op = blockIdx.x / g.tiles_per_op;
  const int tile = (int)(blockIdx.x % g.tiles_per_op);
  auto getc = [&](T*& p, const int*& d) {
    p = g.C + op * g.size_c;
    d = g.dimsC;
  };
  auto getpair = [&](int, const T*& a, const int*& ad, const T*& b, const int*& bd) {
    a = g.A + op * g.size_a;
    ad = g.dimsA;
    b = g.B + op * g.size_b;
    bd = g.dimsB;
  };
  tile_run<T, Cfg>(g.mp, g.sc, tile, getc, getpair, 0, 1, sm);
}

// ------------------------------------------------------------------ staged blocks
// Offset tables of one shape: for every row its offset in A and in C, for every column in B and C,
// for every contracted index in A and B; padded with zeros to whole tiles.  Offsets into A and B are
// in bytes.
struct StagedModes {      // one matrix dimension in one tensor: extents, strides, 2^32 / extent rounded up
  int n;
  int ext[kMaxOrder], str[kMaxOrder];
  unsigned inv[kMaxOrder];
};
template <typename T>
struct StagedArgs {
  StagedModes rA, rC, cB, cC, kA, kB;
  TileScalars<T> sc;
  const T* A; const T* B; T* C;
  long long size_a, size_b, size_c, nb_ops;
  int m, n, K;
  int mp, np, kp;          // padded table lengths
  int abytes, bbytes;      // one buffer of A, of B (128-byte multiples with room for the alignment)
  int lr;                  // FP32: lanes along rows (8, 16 or 32)
};

// idx < 2048 (staged_fits): the multiplication by the rounded-up reciprocal divides exactly
__device__ __forceinline__ int staged_offset(const StagedModes& m, int idx) {
  int off = 0;
  for (int t = 0; t < m.n; ++t) {
    const int q = m.ext[t] == 1 ? idx : t + 1 < m.n ? (int)__umulhi((unsigned)idx, m.inv[t]) : 0;
    off += (idx - q * m.ext[t]) * m.str[t];
    idx = q;
  }
  return off;
}

struct StagedTables {
  int *rowA, *rowC, *colB, *colC, *kA, *kB;
};

template <typename T>
__device__ __forceinline__ StagedTables staged_tables(const StagedArgs<T>& g, unsigned char*& smem) {
  StagedTables t;
  int* p = reinterpret_cast<int*>(smem);
  t.rowA = p; p += g.mp;
  t.rowC = p; p += g.mp;
  t.colB = p; p += g.np;
  t.colC = p; p += g.np;
  t.kA = p; p += g.kp;
  t.kB = p;
  smem += ((2 * (g.mp + g.np + g.kp) * 4) + 127) & ~127;
  for (int i = threadIdx.x; i < g.mp; i += blockDim.x) {
    t.rowA[i] = i < g.m ? staged_offset(g.rA, i) * (int)sizeof(T) : 0;
    t.rowC[i] = i < g.m ? staged_offset(g.rC, i) : 0;
  }
  for (int i = threadIdx.x; i < g.np; i += blockDim.x) {
    t.colB[i] = i < g.n ? staged_offset(g.cB, i) * (int)sizeof(T) : 0;
    t.colC[i] = i < g.n ? staged_offset(g.cC, i) : 0;
  }
  for (int i = threadIdx.x; i < g.kp; i += blockDim.x) {
    t.kA[i] = i < g.K ? staged_offset(g.kA, i) * (int)sizeof(T) : 0;
    t.kB[i] = i < g.K ? staged_offset(g.kB, i) * (int)sizeof(T) : 0;
  }
  return t;
}

// Where byte o of a block lies in its buffer: in place, or (Swz) with the 16-byte units of every 128
// bytes permuted by the next three address bits, which spreads operand reads with power-of-two
// strides over the banks (8x8x8 blocks, contracted modes apart: 16 wavefronts per fragment become 4).
template <bool Swz>
__host__ __device__ __forceinline__ unsigned staged_at(unsigned o) {
  return Swz ? o ^ ((o >> 3) & 0x70u) : o;
}
// Asynchronous copy of n elements into the buffer at shared address buf (128-byte aligned); the data
// keeps its position within its 16-byte units, so whole units are copied at once and only the two
// ends by element.
__device__ __forceinline__ unsigned staged_shift(const void* src) {
  return (unsigned)(reinterpret_cast<size_t>(src) & 15);
}
template <typename T, bool Swz>
__device__ __forceinline__ void staged_copy(unsigned buf, const T* src, int n) {
  const int mis = (int)staged_shift(src), end = mis + n * (int)sizeof(T);
  const unsigned char* s = reinterpret_cast<const unsigned char*>(src) - mis;
  for (int lo = 16 * threadIdx.x; lo < end; lo += 16 * blockDim.x) {
    if (lo >= mis && lo + 16 <= end) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(buf + staged_at<Swz>(lo)), "l"(s + lo)
                   : "memory");
    } else {
      for (int o = max(lo, mis); o < min(lo + 16, end); o += (int)sizeof(T))
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(buf + staged_at<Swz>(o)), "l"(s + o),
                     "n"(sizeof(T))
                     : "memory");
    }
  }
}
// byte o of the block whose buffer starts at byte `buf` of shared memory
template <bool Swz, typename T>
__device__ __forceinline__ T staged_read(const unsigned char* smem, unsigned buf, unsigned o) {
  return *reinterpret_cast<const T*>(smem + (buf + staged_at<Swz>(o)));
}

// The op loop shared by both kernels: two buffers, the next op's copies in flight while body works.
// body(where A's buffer starts in smem, where B's, byte shift of A's data in it, of B's, C).
// Single: no room for two buffers, the next op's copies wait for the current op.
template <typename T, bool Swz, bool Single, class Body>
__device__ __forceinline__ void staged_ops(const StagedArgs<T>& g, unsigned char* smem, Body body) {
  const unsigned bufs = smem_u32(smem), both = (unsigned)(g.abytes + g.bbytes);
  auto fetch = [&](long long op, unsigned at) {
    if (op < g.nb_ops && !g.sc.alpha_zero) {
      staged_copy<T, Swz>(at, g.A + op * g.size_a, (int)g.size_a);
      staged_copy<T, Swz>(at + g.abytes, g.B + op * g.size_b, (int)g.size_b);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  fetch(blockIdx.x, bufs);
  unsigned cur = 0;
  for (long long op = blockIdx.x; op < g.nb_ops; op += gridDim.x, cur = Single ? 0 : both - cur) {
    if (!Single) fetch(op + gridDim.x, bufs + both - cur);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(Single ? 0 : 1) : "memory");
    __syncthreads();  // every thread's copies of this op (and, the first time, the tables)
    body(cur, cur + g.abytes, staged_shift(g.A + op * g.size_a), staged_shift(g.B + op * g.size_b),
         g.C + op * g.size_c);
    __syncthreads();  // the buffer is refilled from here on
    if (Single) fetch(op + gridDim.x, bufs);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Both staged kernels are bound by instruction issue and shared-memory reads, then DRAM.  Measured,
// against a tile per CTA with per-element gathers and tables rebuilt per op:
//   FP64 ikl,ljk->ij, 8x8x8, 10000 ops (87 MB): 79.4 -> 20.5 us (4.2 TB/s); of that 34 us with reads in
//   place (16-way bank conflicts on B) and one tile size for all shapes, 20.5 us with the swizzle and
//   the tile fitted to the block; FP32 ijl,lk->ijk, 13x9x11 by 11x15, 5000 ops (64 MB): 86 -> 28.5 us.
// FP64: warps take groups of 8*ML x 8*NL of the C block (ML x NL fragments of m8n8k4; fragments past
// the block multiply padding: the tensor pipe is not what bounds blocks of this size).
constexpr int kStagedWarpsMax = 8;
// Instances: one CTA an op, the next op's copies in flight (kStagedWhole); several CTAs share an op's groups
// (kStagedSliced); the same with one buffer (kStagedSingle).  What the last two need at run time costs the first
// up to 18% of small ops.
constexpr int kStagedWhole = 0, kStagedSliced = 1, kStagedSingle = 2;
template <int ML, int NL, bool Scale, bool Swz, int Kind>
__global__ void __launch_bounds__(32 * kStagedWarpsMax) k_stack_dmma(const __grid_constant__ StagedArgs<double> g) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw;
  const StagedTables t = staged_tables(g, smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int fr = lane >> 2, kq = lane & 3;
  const int gr = g.mp / (8 * ML), groups = gr * (g.np / (8 * NL));
  const int g0 = Kind ? warp + nw * blockIdx.y : warp, gstep = Kind ? nw * gridDim.y : nw;
  staged_ops<double, Swz, Kind == kStagedSingle>(g, smem, [&](unsigned sa, unsigned sb, unsigned ea, unsigned eb, double* c) {
    for (int grp = g0; grp < groups; grp += gstep) {
      const int r0 = grp % gr * (8 * ML) + fr, c0 = grp / gr * (8 * NL);
      unsigned pa[ML], pb[NL];
#pragma unroll
      for (int i = 0; i < ML; ++i) pa[i] = (Swz ? 0 : sa) + ea + t.rowA[r0 + 8 * i];
#pragma unroll
      for (int j = 0; j < NL; ++j) pb[j] = (Swz ? 0 : sb) + eb + t.colB[c0 + 8 * j + fr];
      int ro[ML], co[NL][2];  // offsets in C, negative past the block
#pragma unroll
      for (int i = 0; i < ML; ++i) ro[i] = r0 + 8 * i < g.m ? t.rowC[r0 + 8 * i] : -1;
#pragma unroll
      for (int j = 0; j < NL; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int s = c0 + 8 * j + 2 * kq + e;
          co[j][e] = s < g.n ? t.colC[s] : -1;
        }
      double acc[ML][NL][2] = {};
      if (!g.sc.beta_zero) {
#pragma unroll
        for (int i = 0; i < ML; ++i)
#pragma unroll
          for (int j = 0; j < NL; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if ((ro[i] | co[j][e]) >= 0) acc[i][j][e] = mul_rn(g.sc.beta, c[ro[i] + co[j][e]]);
      }
      auto step = [&](int k, bool dead) {
        const unsigned ka = t.kA[k + kq], kb = t.kB[k + kq];
        double af[ML], bf[NL];
#pragma unroll
        for (int i = 0; i < ML; ++i) {
          af[i] = staged_read<Swz, double>(smem, Swz ? sa : 0, pa[i] + ka);
          if (Scale) af[i] = mul_rn(g.sc.alpha, af[i]);
          if (dead) af[i] = -0.0;  // past the contracted extent: fma(-0, +0, c) == c
        }
#pragma unroll
        for (int j = 0; j < NL; ++j) {
          bf[j] = staged_read<Swz, double>(smem, Swz ? sb : 0, pb[j] + kb);
          if (dead) bf[j] = 0.0;
        }
#pragma unroll
        for (int i = 0; i < ML; ++i)
#pragma unroll
          for (int j = 0; j < NL; ++j) dmma884(acc[i][j], af[i], bf[j]);
      };
      const int K = g.sc.alpha_zero ? 0 : g.K;
#pragma unroll 4
      for (int k = 0; k < (K & ~3); k += 4) step(k, false);
      if (K & 3) step(K & ~3, kq >= (K & 3));
#pragma unroll
      for (int i = 0; i < ML; ++i)
        if (ro[i] >= 0) {
          double* cr = c + ro[i];
#pragma unroll
          for (int j = 0; j < NL; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (co[j][e] >= 0) cr[co[j][e]] = acc[i][j][e];
        }
      __syncwarp();
    }
  });
}

// FP32: warps take groups of RM*lr rows x CN*(32/lr) columns; a lane has RM rows lr apart and CN
// columns 32/lr apart, so that its stores run along the rows.
template <int RM, int CN, bool Scale, bool Swz, int Kind>
__global__ void __launch_bounds__(32 * kStagedWarpsMax) k_stack_fma(const __grid_constant__ StagedArgs<float> g) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw;
  const StagedTables t = staged_tables(g, smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int lr = g.lr, lc = 32 / lr, r1 = lane & (lr - 1), c1 = lane / lr;
  const int gr = g.mp / (RM * lr), groups = gr * (g.np / (CN * lc));
  const int g0 = Kind ? warp + nw * blockIdx.y : warp, gstep = Kind ? nw * gridDim.y : nw;
  staged_ops<float, Swz, false>(g, smem, [&](unsigned sa, unsigned sb, unsigned ea, unsigned eb, float* c) {
    for (int grp = g0; grp < groups; grp += gstep) {
      const int r0 = grp % gr * (RM * lr) + r1, c0 = grp / gr * (CN * lc) + c1;
      unsigned pa[RM], pb[CN];
#pragma unroll
      for (int i = 0; i < RM; ++i) pa[i] = (Swz ? 0 : sa) + ea + t.rowA[r0 + i * lr];
#pragma unroll
      for (int j = 0; j < CN; ++j) pb[j] = (Swz ? 0 : sb) + eb + t.colB[c0 + j * lc];
      int ro[RM];  // offsets in C, negative past the block
#pragma unroll
      for (int i = 0; i < RM; ++i) ro[i] = r0 + i * lr < g.m ? t.rowC[r0 + i * lr] : -1;
      float acc[RM][CN] = {};
      if (!g.sc.beta_zero) {
#pragma unroll
        for (int j = 0; j < CN; ++j)
#pragma unroll
          for (int i = 0; i < RM; ++i)
            if (ro[i] >= 0 && c0 + j * lc < g.n) acc[i][j] = mul_rn(g.sc.beta, c[ro[i] + t.colC[c0 + j * lc]]);
      }
      const int K = g.sc.alpha_zero ? 0 : g.K;
#pragma unroll 2
      for (int k = 0; k < K; ++k) {
        const unsigned ka = t.kA[k], kb = t.kB[k];
        float a[RM], b[CN];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          a[i] = staged_read<Swz, float>(smem, Swz ? sa : 0, pa[i] + ka);
          if (Scale) a[i] = mul_rn(g.sc.alpha, a[i]);
        }
#pragma unroll
        for (int j = 0; j < CN; ++j) b[j] = staged_read<Swz, float>(smem, Swz ? sb : 0, pb[j] + kb);
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < CN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
#pragma unroll
      for (int j = 0; j < CN; ++j) {
        if (c0 + j * lc < g.n) {
          float* cs = c + t.colC[c0 + j * lc];
#pragma unroll
          for (int i = 0; i < RM; ++i)
            if (ro[i] >= 0) cs[ro[i]] = acc[i][j];
        }
      }
    }
  });
}

// Both blocks of an op at most this many bytes: two ops' buffers are then 48 KB, so that several CTAs share
// an SM, which hides the copies' latency (four and more by shared memory; registers keep the eight-warp
// instances at two or three).
constexpr long long kStagedBytes = 24 * 1024, kStagedTables = 4096;
// FP64 blocks whose free or contracted modes lie apart: as many as fit an SM, two ops' buffers up to
// kStagedTwo.  The ring kernel can only gather such blocks element by element.  Measured, kil,ljk->ji,
// 14x23x18 by 18x20x14 (86 KB), 2,258 ops: 183 us with a gathering tile, 223 us with the ring, 78 us staged;
// abcd,dcij->abij 8x5x12x6 by 6x12x8x10, 2,761 ops: 310, 199, 133; one buffer, kil,ljk->ji 19x21x25 by
// 25x23x19 (167 KB), 1,913 ops: 300, 425, 144.
// Rows and columns that both lie across C's order: the ring's stores are all apart, here they run along it.
// Pia,Pjb->abij 14x7x21 by 14x20x17 (55 KB), 2,129 ops: 596 us with
// a gathering tile, 1,279 with the ring, 315 staged.
constexpr long long kStagedTwo = 100 * 1024, kStagedApart = 200 * 1024;
static long long staged_bytes(const sht_kernel* k, size_t es) { return (k->size_a + k->size_b) * (long long)es; }
static bool staged_single(const sht_kernel* k, size_t es) { return staged_bytes(k, es) > kStagedTwo; }
static bool modes_apart(const sht_kernel* k) {
  auto apart = [](const std::vector<int>& v) { return !modes_consecutive(v.data(), (int)v.size()); };
  return apart(k->maps.rowA) || apart(k->maps.colA) || apart(k->maps.colB) || apart(k->maps.rowB);
}
static bool staged_fits(const sht_kernel* k, size_t es) {
  const long long most = es == 8 && (k->apart || k->scattered) ? kStagedApart : kStagedBytes;
  return staged_bytes(k, es) <= most && k->m + k->n + k->k <= kStagedTables / 2;
}
// With fewer ops than SMs the ring kernel spreads an op's tiles over the chip, which from four tiles on is
// the faster (iPa,jPb->ijab 21x14x27 by 8x14x24, one op, 27 tiles: 41.6 us staged, 10.5 with the ring;
// acbd,cidj->abij 7x9x10x3 by 9x9x3x12, 2 ops, 4 tiles: 10.5 and 10.4; 10x12x6x10 by 12x9x10x2, one op, 2
// tiles: 8.4 and 16.6).
static bool use_staged(const sht_kernel* k, size_t es, long long nb_ops) {
  if (!staged_fits(k, es)) return false;
  if (staged_bytes(k, es) <= kStagedBytes || nb_ops >= k->ctx->num_sms) return true;
  return ring_ntiles((int)k->m, kRingTile) * ring_ntiles((int)k->n, kRingTile) < 4;
}

static StagedModes staged_modes(const std::vector<int>& modes, const std::vector<int>& dims) {
  StagedModes m{};
  m.n = (int)modes.size();
  for (int t = 0; t < m.n; ++t) {
    m.ext[t] = dims[modes[t]];
    m.str[t] = 1;
    for (int u = 0; u < modes[t]; ++u) m.str[t] *= dims[u];
    m.inv[t] = (unsigned)((1ull << 32) / (unsigned)m.ext[t] + 1);
  }
  return m;
}
static int host_offset(const StagedModes& m, int idx) {
  int off = 0;
  for (int t = 0; t < m.n; ++t) {
    off += idx % m.ext[t] * m.str[t];
    idx /= m.ext[t];
  }
  return off;
}

template <typename T>
static StagedArgs<T> staged_args(const sht_kernel* k, const StackArgs<T>& g, long long nb_ops, int row_tile, int col_tile) {
  StagedArgs<T> s{};
  s.rA = staged_modes(k->staged.rowA, k->sa);
  s.rC = staged_modes(k->staged.rowC, k->sc);
  s.cB = staged_modes(k->staged.colB, k->sb);
  s.cC = staged_modes(k->staged.colC, k->sc);
  s.kA = staged_modes(k->staged.colA, k->sa);
  s.kB = staged_modes(k->staged.rowB, k->sb);
  s.sc = g.sc;
  s.A = g.A; s.B = g.B; s.C = g.C;
  s.size_a = g.size_a; s.size_b = g.size_b; s.size_c = g.size_c;
  s.nb_ops = nb_ops;
  s.m = (int)k->m; s.n = (int)k->n; s.K = (int)k->k;
  s.mp = (s.m + row_tile - 1) / row_tile * row_tile;
  s.np = (s.n + col_tile - 1) / col_tile * col_tile;
  s.kp = (s.K + 3) & ~3;
  s.abytes = (int)((g.size_a * sizeof(T) + 16 + 127) & ~127ull);
  s.bbytes = (int)((g.size_b * sizeof(T) + 16 + 127) & ~127ull);
  s.lr = 32;
  return s;
}

// Shared-memory wavefronts of one operand's reads in the first k-steps, in place (0) and swizzled (1),
// data at the start of its 16-byte unit.  FP64: 8 rows x 4 k per read; FP32: lr rows, one k.
static void staged_wavefronts(const StagedModes& rows, const StagedModes& ks, int nrows, int K, bool f64, int lr,
                              int (&total)[2]) {
  const int es = f64 ? 8 : 4, kw = f64 ? 4 : 1, steps = std::min(2, (K + kw - 1) / kw);
  int ro[32], ko[8];
  for (int r = 0; r < lr; ++r) ro[r] = r < nrows ? host_offset(rows, r) : 0;
  for (int k = 0; k < steps * kw; ++k) ko[k] = k < K ? host_offset(ks, k) : 0;
  for (int s = 0; s < steps; ++s)
    for (int swz = 0; swz < 2; ++swz) {
      unsigned seen[32][32];  // distinct words per bank (of es bytes)
      int count[32] = {0}, most = 0;
      for (int r = 0; r < lr; ++r)
        for (int k = 0; k < kw; ++k) {
          unsigned o = (unsigned)(es * (ro[r] + ko[s * kw + k]));
          if (swz) o = staged_at<true>(o);
          const int bank = o / es % (128 / es);
          int i = 0;
          while (i < count[bank] && seen[bank][i] != o) ++i;
          if (i == count[bank]) seen[bank][count[bank]++] = o;
          most = std::max(most, count[bank]);
        }
      total[swz] += most;
    }
}

// FP32 register tile and lanes along rows: the least issue slots over the op's groups (products, operand and
// table reads per k).  With few ops (up to three for each SM) the op's own time counts too: its groups run at
// once on up to kStagedWarpsMax warps, each k waiting about 40 cycles for its reads, and an SM has registers
// for kStagedResident warps of the largest instances.  Measured, ik,kj->ij 30x60
// by 60x30 (us, by issue slots alone / so): 149 ops 14.3 / 8.2, 300 ops 14.4 / 8.2.
struct FmaShape { int rm, cn, lr; };
constexpr double kFewPerSm = 3, kManyOps = 1e9;
constexpr int kStagedResident = 16;
static FmaShape pick_fma_shape(int m, int n, double ops_per_sm) {
  static const int tiles[][2] = {{1, 2}, {2, 4}, {4, 4}, {4, 8}};
  FmaShape best{4, 8, 32};
  double bc = 1e300;
  for (const auto& t : tiles)
    for (int lr = 32; lr >= 8; lr /= 2) {
      const int rt = t[0] * lr, ct = t[1] * (32 / lr);
      const double groups = (double)((m + rt - 1) / rt) * (double)((n + ct - 1) / ct);
      const double k = t[0] * t[1] + 1.5 * (t[0] + t[1]) + 6;
      const double rounds = std::ceil(ops_per_sm / std::floor(kStagedResident / std::min(groups, (double)kStagedWarpsMax)));
      const double latency = rounds * std::ceil(groups / kStagedWarpsMax) * (k + 40), issue = groups * k;
      // an SM issues for four warps at once
      const double c = ops_per_sm <= 1 ? latency : ops_per_sm <= kFewPerSm ? std::max(latency, ops_per_sm * issue / 4) : issue;
      if (c < bc) { bc = c; best = {t[0], t[1], lr}; }
    }
  return best;
}

// Host decisions of a kernel's calls that depend on its shape only.
void stack_prepare(sht_kernel* k) {
  const bool f64 = k->dtype == SHT_F64;
  k->swizzle = false;
  k->apart = modes_apart(k);
  auto leads = [](const std::vector<int>& v) { return !v.empty() && v[0] == 0; };
  k->scattered = !leads(k->maps.rowC) && !leads(k->maps.colC);
  // The staged kernels address every row and column through tables: in C's order their stores run along it
  // (Pai,Pbj->ijab 7x22x8 by 7x24x8, 2,295 ops: 854 us in the operands' order, 133 so)
  k->staged = k->maps;
  auto by_c = [](std::vector<int>& op, std::vector<int>& c) {
    std::vector<std::pair<int, int>> v;
    for (size_t i = 0; i < c.size(); ++i) v.emplace_back(c[i], op[i]);
    std::sort(v.begin(), v.end());
    for (size_t i = 0; i < c.size(); ++i) std::tie(c[i], op[i]) = v[i];
  };
  by_c(k->staged.rowA, k->staged.rowC);
  by_c(k->staged.colB, k->staged.colC);
  if (!staged_fits(k, f64 ? 8 : 4)) return;
  const StagedModes ra = staged_modes(k->staged.rowA, k->sa), ka = staged_modes(k->staged.colA, k->sa);
  const StagedModes cb = staged_modes(k->staged.colB, k->sb), kb = staged_modes(k->staged.rowB, k->sb);
  const int m = (int)k->m, n = (int)k->n, K = (int)k->k;
  // FP32 columns are the same for whole rows of lanes: only A's reads spread over the banks
  const int lr = f64 ? 8 : pick_fma_shape(m, n, kManyOps).lr;
  int w[2] = {0, 0};
  staged_wavefronts(ra, ka, m, K, f64, lr, w);
  if (f64) staged_wavefronts(cb, kb, n, K, f64, 8, w);
  k->swizzle = 4 * w[1] < 3 * w[0];  // it costs two integer instructions a read
}

// kernels: [kind][Scale * 2 + Swz] of the tile; groups: of an op
template <typename T, class Kernel>
static void launch_staged(sht_kernel* k, const StagedArgs<T>& s, int groups, bool few, const Kernel* kernels,
                          cudaStream_t st) {
  // a warp per group of the block; more where the copies would take a thread many turns
  const int warps = std::min(std::max(groups, few ? (s.abytes + s.bbytes) / 1024 : 0), kStagedWarpsMax);
  const bool single = staged_single(k, sizeof(T));
  const size_t smem = (((size_t)2 * (s.mp + s.np + s.kp) * 4 + 127) & ~(size_t)127) +
                      (single ? 1 : 2) * (size_t)(s.abytes + s.bbytes);
  // CTAs by shared memory and by threads; ops are strided over them (registers may keep some of the grid for
  // a second wave)
  const long long per_sm = std::max<long long>(1, std::min<long long>({32, 227 * 1024 / (long long)(smem + 1024), 32 / warps}));
  const long long grid = std::min(s.nb_ops, per_sm * k->ctx->num_sms);
  // Few ops of many groups: several CTAs share an op, each with its two blocks staged.  Measured (us, a tile for
  // each CTA / one CTA an op / so): FP64 ik,kj->ij 143x5 by 5x288, 22 ops 9.4 / 17.2 / 8.5; FP32
  // Pia,Pjb->abij 4x29x26 by 4x28x20, 5 ops 18.8 / 96.6 / 10.5.
  const long long slices = std::min<long long>((groups + warps - 1) / warps, per_sm * k->ctx->num_sms / s.nb_ops);
  const int kind = single ? kStagedSingle : slices > 1 ? kStagedSliced : kStagedWhole;
  kernels[4 * kind + (s.sc.alpha != 1.0 ? 2 : 0) + (k->swizzle ? 1 : 0)]<<<
      dim3((unsigned)grid, (unsigned)std::max<long long>(slices, 1)), 32 * warps, smem, st>>>(s);
  SHT_CUDA(cudaGetLastError());
}

// [tile][kind * 4 + Scale * 2 + Swz]; FP64 tiles: 1, 2 or 4 fragment rows x 1 or 2 columns
#define SHT_KIND(K, X, Y, KIND) \
  K<X, Y, false, false, KIND>, K<X, Y, false, true, KIND>, K<X, Y, true, false, KIND>, K<X, Y, true, true, KIND>
#define SHT_DMMA(ML, NL)                                                                                           \
  {SHT_KIND(k_stack_dmma, ML, NL, kStagedWhole), SHT_KIND(k_stack_dmma, ML, NL, kStagedSliced),                     \
   SHT_KIND(k_stack_dmma, ML, NL, kStagedSingle)}
static void (*const kStackDmma[6][12])(StagedArgs<double>) = {SHT_DMMA(1, 1), SHT_DMMA(1, 2), SHT_DMMA(2, 1),
                                                              SHT_DMMA(2, 2), SHT_DMMA(4, 1), SHT_DMMA(4, 2)};
#define SHT_FMA(RM, CN) {SHT_KIND(k_stack_fma, RM, CN, kStagedWhole), SHT_KIND(k_stack_fma, RM, CN, kStagedSliced)}
static void (*const kStackFma[4][8])(StagedArgs<float>) = {SHT_FMA(1, 2), SHT_FMA(2, 4), SHT_FMA(4, 4), SHT_FMA(4, 8)};
#undef SHT_KIND
#undef SHT_DMMA
#undef SHT_FMA

static void stack_setup(int device) {
  static DeviceOnce once;
  once.run(device, [] {
    const int big = 222 * 1024;  // buffers and tables of the largest staged shape
    for (const auto& r : kStackDmma)
      for (auto* f : r) SHT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    for (const auto& r : kStackFma)
      for (auto* f : r) SHT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  });
}

// An SM for each op: a call then takes the latency of one op, not its share of issue slots.  Measured
// with the event overhead of a lone call (11.6 us): FP32 ik,kj->ij 63x51 by 51x10, 13 ops: 20.5 us
// with the issue-bound shape, 13.9 us so; FP64 ikl,ljk->ij 5x16x9, 117 ops: 17.3 and 11.9.
static bool few_ops(const sht_kernel* k, long long nb_ops) { return nb_ops <= k->ctx->num_sms; }
static void launch_staged_op(sht_kernel* k, const StackArgs<double>& g, long long nb_ops, cudaStream_t st) {
  // the smallest tile that takes the block's rows and columns at once, up to 32 x 16; with few ops the
  // smallest whose groups a CTA's warps take at once
  const bool few = few_ops(k, nb_ops) || staged_bytes(k, 8) > kStagedBytes;
  int ri = k->m <= 8 ? 0 : k->m <= 16 ? 1 : 2, ci = k->n <= 8 ? 0 : 1;
  for (int t = 0, end = few ? 2 * ri + ci : 0; t < end; ++t)
    if (((k->m - 1) / (8 << t / 2) + 1) * ((k->n - 1) / (8 << t % 2) + 1) <= kStagedWarpsMax) {
      ri = t / 2;
      ci = t % 2;
      break;
    }
  const int rt = 8 << ri, ct = 8 << ci;
  const StagedArgs<double> s = staged_args(k, g, nb_ops, rt, ct);
  launch_staged(k, s, (s.mp / rt) * (s.np / ct), few, kStackDmma[2 * ri + ci], st);
}
static void launch_staged_op(sht_kernel* k, const StackArgs<float>& g, long long nb_ops, cudaStream_t st) {
  const double ops_per_sm = (double)nb_ops / k->ctx->num_sms;
  const FmaShape f = pick_fma_shape((int)k->m, (int)k->n, ops_per_sm);
  const int rt = f.rm * f.lr, ct = f.cn * (32 / f.lr);
  StagedArgs<float> s = staged_args(k, g, nb_ops, rt, ct);
  s.lr = f.lr;
  // more warps for the copies where every op stays resident
  const int copy_warps = std::min(std::max((s.mp / rt) * (s.np / ct), (s.abytes + s.bbytes) / 1024), kStagedWarpsMax);
  const bool few = ops_per_sm <= kFewPerSm && ops_per_sm <= kStagedResident / copy_warps;
  const int tile = f.rm == 1 ? 0 : f.rm == 2 ? 1 : f.cn == 4 ? 2 : 3;
  launch_staged(k, s, (s.mp / rt) * (s.np / ct), few, kStackFma[tile], st);
}

// ------------------------------------------------------------------ larger blocks
// FP64: the ring tile kernel.
static void launch_large(sht_kernel* k, const StackArgs<double>& g, long long nb_ops, cudaStream_t st) {
  SparseArgs a{};
  a.mp = g.mp;
  a.sc = g.sc;
  a.A = g.A; a.B = g.B; a.C = g.C;
  auto strides = [](const int* d, int order, const std::vector<int>& f, const std::vector<int>& kk, int& rs, int& ks) {
    rs = ks = 1;
    for (int u = 0; u < order; ++u) {
      if (!f.empty() && u < f[0]) rs *= d[u];
      if (!kk.empty() && u < kk[0]) ks *= d[u];
    }
  };
  PairRec rec{};
  rec.K = (int)k->k;
  strides(g.dimsA, g.mp.oA, k->maps.rowA, k->maps.colA, rec.rsA, rec.ksA);
  strides(g.dimsB, g.mp.oB, k->maps.colB, k->maps.rowB, rec.rsB, rec.ksB);
  ring_stack(k->ctx, a, rec, g.dimsA, g.dimsB, g.dimsC, g.size_a, g.size_b, g.size_c, (int)k->m, (int)k->n, nb_ops, st);
}

// FP32: one gathering tile per CTA.
using S64x64 = TileCfg<64, 64, 16, 4, 4>;
using S128x32 = TileCfg<128, 32, 16, 8, 2>;
using S32x128 = TileCfg<32, 128, 16, 2, 8>;
using S32x32 = TileCfg<32, 32, 16, 2, 2>;
using S16x16 = TileCfg<16, 16, 16, 2, 2>;

struct StackShape { int tm, tn; };
static const StackShape kStackShapes[] = {{64, 64}, {128, 32}, {32, 128}, {32, 32}, {16, 16}};

static int pick_stack_shape(long long m, long long n) {
  double best = 1e300;
  int bi = 0;
  for (int i = 0; i < 5; ++i) {
    const long long tm = kStackShapes[i].tm, tn = kStackShapes[i].tn;
    const long long tiles = ((m + tm - 1) / tm) * ((n + tn - 1) / tn);
    const double cost = (double)tiles * (double)(tm * tn + 1024);
    if (cost < best) { best = cost; bi = i; }
  }
  return bi;
}

static void launch_large(sht_kernel* k, StackArgs<float>& g, long long nb_ops, cudaStream_t s) {
  const int sh = pick_stack_shape(k->m, k->n);
  const long long tm = kStackShapes[sh].tm, tn = kStackShapes[sh].tn;
  g.tiles_per_op = (int)(((k->m + tm - 1) / tm) * ((k->n + tn - 1) / tn));
  const long long blocks = nb_ops * g.tiles_per_op;
  if (blocks > 0x7fffffffLL) fail(SHT_ERR_UNSUPPORTED, "stack too large for one launch");
  const unsigned grid = (unsigned)blocks;
  switch (sh) {
    case 0: k_stack<float, S64x64><<<grid, S64x64::kThreads, 0, s>>>(g); break;
    case 1: k_stack<float, S128x32><<<grid, S128x32::kThreads, 0, s>>>(g); break;
    case 2: k_stack<float, S32x128><<<grid, S32x128::kThreads, 0, s>>>(g); break;
    case 3: k_stack<float, S32x32><<<grid, S32x32::kThreads, 0, s>>>(g); break;
    default: k_stack<float, S16x16><<<grid, S16x16::kThreads, 0, s>>>(g); break;
  }
  SHT_CUDA(cudaGetLastError());
}

static bool is_device_pointer(const void* p) {
  cudaPointerAttributes at{};
  cudaError_t e = cudaPointerGetAttributes(&at, p);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

template <typename T>
static void launch_stack(sht_kernel* k, const T* a, const T* b, T* c, long long nb_ops, cudaStream_t s) {
  StackArgs<T> g{};
  g.mp.row.n = (int)k->maps.rowA.size();
  for (size_t i = 0; i < k->maps.rowA.size(); ++i) { g.mp.row.x[i] = k->maps.rowA[i]; g.mp.row.y[i] = k->maps.rowC[i]; }
  g.mp.kk.n = (int)k->maps.colA.size();
  for (size_t i = 0; i < k->maps.colA.size(); ++i) { g.mp.kk.x[i] = k->maps.colA[i]; g.mp.kk.y[i] = k->maps.rowB[i]; }
  g.mp.col.n = (int)k->maps.colB.size();
  for (size_t i = 0; i < k->maps.colB.size(); ++i) { g.mp.col.x[i] = k->maps.colB[i]; g.mp.col.y[i] = k->maps.colC[i]; }
  g.mp.oA = (int)k->sa.size();
  g.mp.oB = (int)k->sb.size();
  g.mp.oC = (int)k->sc.size();
  for (size_t i = 0; i < k->sa.size(); ++i) g.dimsA[i] = k->sa[i];
  for (size_t i = 0; i < k->sb.size(); ++i) g.dimsB[i] = k->sb[i];
  for (size_t i = 0; i < k->sc.size(); ++i) g.dimsC[i] = k->sc[i];
  g.sc.alpha = (T)k->alpha;
  g.sc.beta = (T)k->beta;
  const T al = (T)k->alpha, be = (T)k->beta;
  unsigned char zb[sizeof(T)] = {0};
  g.sc.alpha_zero = std::memcmp(&al, zb, sizeof(T)) == 0;
  g.sc.beta_zero = std::memcmp(&be, zb, sizeof(T)) == 0;
  g.A = a; g.B = b; g.C = c;
  g.size_a = k->size_a; g.size_b = k->size_b; g.size_c = k->size_c;
  stack_setup(k->ctx->device);
  if (use_staged(k, sizeof(T), nb_ops)) launch_staged_op(k, g, nb_ops, s);
  else launch_large(k, g, nb_ops, s);
}

void stack_call(sht_kernel* k, const void* a, const void* b, void* c, int64_t nb_ops, cudaStream_t s) {
  if (nb_ops < 0) fail(SHT_ERR_INVALID, "nb_ops < 0");
  if (nb_ops == 0) return;
  if (!a || !b || !c) fail(SHT_ERR_INVALID, "null operand");
  const size_t es = k->dtype == SHT_F64 ? 8 : 4;
  const bool dev = is_device_pointer(a) && is_device_pointer(b) && is_device_pointer(c);
  if (dev) {
    if (k->dtype == SHT_F64)
      launch_stack<double>(k, (const double*)a, (const double*)b, (double*)c, nb_ops, s);
    else
      launch_stack<float>(k, (const float*)a, (const float*)b, (float*)c, nb_ops, s);
    return;
  }
  // host operands: stage through the pool
  DevicePool* pool = k->ctx->pool.get();
  const size_t ba = (size_t)nb_ops * k->size_a * es, bb = (size_t)nb_ops * k->size_b * es,
               bc = (size_t)nb_ops * k->size_c * es;
  PoolBuf da(pool, ba, s), db(pool, bb, s), dc(pool, bc, s);
  SHT_CUDA(cudaMemcpyAsync(da.ptr, a, ba, cudaMemcpyHostToDevice, s));
  SHT_CUDA(cudaMemcpyAsync(db.ptr, b, bb, cudaMemcpyHostToDevice, s));
  SHT_CUDA(cudaMemcpyAsync(dc.ptr, c, bc, cudaMemcpyHostToDevice, s));
  if (k->dtype == SHT_F64)
    launch_stack<double>(k, da.as<double>(), db.as<double>(), dc.as<double>(), nb_ops, s);
  else
    launch_stack<float>(k, da.as<float>(), db.as<float>(), dc.as<float>(), nb_ops, s);
  SHT_CUDA(cudaMemcpyAsync(c, dc.ptr, bc, cudaMemcpyDeviceToHost, s));
  SHT_CUDA(cudaStreamSynchronize(s));
}

}  // namespace sht

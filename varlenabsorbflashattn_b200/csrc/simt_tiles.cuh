// Tiled fp32-arithmetic attention kernels for the shapes the tcgen05 kernels do not take (fp32 I/O, head dims
// other than 64/128), head dim up to 256.
//
// Bound: the FMA pipe (128 multiply-adds per clock and SM; packed pairs halve the issue slots).  A CTA of eight
// warps owns 64 outer rows of one segment (query rows for the forward and dQ, key rows for dK/dV) and walks the
// segment's inner rows in blocks of C; a warp owns eight of the outer rows in every step, so scores, row
// statistics and accumulators of a row never leave its warp and only the block loads need a CTA barrier.
//   scores : lane (rg, cg) = (lane / 16, lane % 16) computes outer rows 4 rg .. 4 rg + 3 against inner rows cg + 16 j;
//            16-byte shared-memory reads along the head dim, pairs of products per instruction, partial sums of
//            32 products (a single chain over the head dim would round worse than the sum of lanes it replaces)
//   second product: the block's weights (P or dS) go through shared memory within the warp; a lane owns four
//            (head dim 256: eight) columns of 2-8 rows
// The rows of all heads that share K/V (the absorb operator: H heads over the raw X rows) are stacked into one
// outer tile, so that a block of X is loaded once for all of them.
// A cluster of 1-8 CTAs shares one outer tile, rank i taking blocks i, i + N, ...; the partial results are
// merged through distributed shared memory in rank order (no atomics, no workspace, run-to-run identical).
// Outer tiles are found without a list (seg_search.cuh).
//
// Measured on a B200, 64 users of 1-16 targets over 8-2048 keys, 8 heads, d_kv = 256, fp32 (forward / dQ / dX): 160 /
// 211 / 185 us, against 1746 / 2251 / 1155 us with one warp per output row (simt_kernels.cu), which spends five
// shuffles per (row, key) and reads every key once per row.  (Before the rows were copied asynchronously, see load_tile: 189 / 232 /
// 229 us, with at most four CTAs per tile 195 / 261 / 232.)
#pragma once
#include <cooperative_groups.h>
#include <type_traits>

#include "profile.cuh"
#include "seg_search.cuh"
#include "simt_kernels.cuh"
#include "sm100_ptx.cuh"

namespace vafa {
namespace tiles {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;  // eight warps of eight outer rows
constexpr int kMaxSplits = 8;  // portable cluster size

struct TileParams {
  const void *q, *k, *v, *d_o;
  void *o, *dq, *dk, *dv;
  float* lse;
  const float* delta;
  const int32_t *cu_q, *cu_k;
  int n_seg, D, H;
  int heads;    // outer heads that are walked separately: H, or 1 when all heads are stacked
  int stack;    // heads stacked into a tile: 1, or H
  int splits;   // cluster size
  long long slots;
  int64_t q_row, k_row, v_row, do_row;      // elements between consecutive (stacked) rows
  int64_t q_head, k_head, v_head, do_head;  // elements between separately walked heads
  int vec_q, vec_k, vec_v, vec_do, vec_o;   // rows can be read / written four elements at a time
  int causal;
  float scale;
  int total_q, total_k, guard;  // guard: see SimtAttnParams
};

template <int DP> struct Dim {
  static constexpr int kStride = DP + 4;                  // floats between rows in shared memory: 16-byte reads of
                                                          // eight consecutive rows touch all banks once
  static constexpr int kLanes = DP / 4 < 32 ? DP / 4 : 32;  // lanes across the columns in the second product
  static constexpr int kGroups = 32 / kLanes;             // row groups of a warp there
  static constexpr int kRpl = 8 / kGroups;                // rows per lane
  static constexpr int kVec = DP / (4 * kLanes);          // four-column pieces per lane
};

template <typename T> __device__ __forceinline__ float4 load4(const T* p) {
  float4 f;
  if constexpr (sizeof(T) == 4) {
    f = *reinterpret_cast<const float4*>(p);
  } else {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    T e[4];
    memcpy(e, &w, 8);
    f = make_float4(to_float(e[0]), to_float(e[1]), to_float(e[2]), to_float(e[3]));
  }
  return f;
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 f) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = f;
  } else {
    uint2 w;
    w.x = pack2_out<T>(f.x, f.y);
    w.y = pack2_out<T>(f.z, f.w);
    *reinterpret_cast<uint2*>(p) = w;
  }
}

// 16 bytes from global to shared memory without a register on the way; `bytes` = 0 writes zeros and reads nothing.
__device__ __forceinline__ void copy16_async(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
// The thread's copies so far have arrived (load_tile: before the barrier that publishes the tile).
__device__ __forceinline__ void tile_arrived() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// kN rows of DP columns into shared memory; rows past n_valid, rows `keep` refuses and columns past D become zeros.
// fp32 rows that can be read four elements at a time are all on their way at once, several tiles together; through registers,
// eight loads at a time, a CTA waited four times for its first two tiles.  Forward | dQ | dK/dV, registers -> now: 64 users of
// 1-16 targets, widths 256, 217 -> 160 | 238 -> 211 | 211 -> 185 us; 148 users x 2048 keys 1114 -> 766 | 1431 -> 1084 | 1796 -> 1426.
// (A second set of tiles, filled while the first is multiplied: 156 | 213 | 183 and 736 | 1084 | 1408.)
template <int DP, int kN, typename T, typename Keep>
__device__ __forceinline__ void load_tile(float* dst, const T* src, int64_t row_stride, int n_valid, int D, int vec, Keep keep) {
  constexpr int kQuads = DP / 4;
  constexpr int kIters = kN * kQuads / kThreads;
  if constexpr (sizeof(T) == 4) {
    if (vec) {
#pragma unroll 4
      for (int it = 0; it < kIters; ++it) {
        const int i = it * kThreads + threadIdx.x;
        const int r = i / kQuads, c = (i % kQuads) * 4;
        const bool ok = r < n_valid && c < D && keep(r);
        copy16_async(dst + r * Dim<DP>::kStride + c, ok ? src + r * row_stride + c : src, ok ? 16 : 0);
      }
      return;
    }
  }
#pragma unroll 8
  for (int it = 0; it < kIters; ++it) {
    const int i = it * kThreads + threadIdx.x;
    const int r = i / kQuads, c = (i % kQuads) * 4;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n_valid && c < D && keep(r)) {
      const T* p = src + r * row_stride + c;
      if (vec) {
        f = load4(p);
      } else {
        f.x = to_float(p[0]);
        if (c + 1 < D) f.y = to_float(p[1]);
        if (c + 2 < D) f.z = to_float(p[2]);
        if (c + 3 < D) f.w = to_float(p[3]);
      }
    }
    *reinterpret_cast<float4*>(dst + r * Dim<DP>::kStride + c) = f;
  }
}
struct KeepAll {
  __device__ __forceinline__ bool operator()(int) const { return true; }
};

// s[i][j] = a[4 rg + i] . b[cg + 16 j] over DP columns.
template <int DP, int J>
__device__ __forceinline__ void dot_block(const float* a, const float* b, float (&s)[4][J]) {
  constexpr int S = Dim<DP>::kStride;
  const int lane = threadIdx.x & 31;
  const float* ap = a + (lane >> 4) * 4 * S;
  const float* bp = b + (lane & 15) * S;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) s[i][j] = 0.f;
#pragma unroll 1
  for (int k0 = 0; k0 < DP; k0 += 32) {
    uint64_t acc[4][J];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int k = 0; k < 32; k += 4) {
      ulonglong2 av[4], bv[J];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(ap + i * S + k0 + k);
#pragma unroll
      for (int j = 0; j < J; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(bp + j * 16 * S + k0 + k);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j) {
          acc[i][j] = ptx::fma_f2(av[i].x, bv[j].x, acc[i][j]);
          acc[i][j] = ptx::fma_f2(av[i].y, bv[j].y, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < J; ++j) {
        float lo, hi;
        ptx::unpack_f2(acc[i][j], lo, hi);
        s[i][j] += lo + hi;
      }
  }
}

// acc[r][.] += sum over j < n of w[r][j] * v[j][.] for the lane's rows and columns.  kMask: a row takes inner rows
// lo[r] <= j < hi[r] only (weights outside are zero already, but zero times an infinity or NaN of a row that is
// not visible must not reach the sum).
template <int DP, int C, bool kMask>
__device__ __forceinline__ void add_weighted(uint64_t (&acc)[Dim<DP>::kRpl][Dim<DP>::kVec * 2], const float* w, const float* v, int n,
                                             const int* lo, const int* hi) {
  using X = Dim<DP>;
  const int lane = threadIdx.x & 31;
  const float* wp = w + (lane / X::kLanes) * X::kRpl * (C + 4);
  const float* vp = v + (lane % X::kLanes) * 4;
#pragma unroll 2
  for (int j = 0; j < n; j += 4) {
    float4 wv[X::kRpl];
#pragma unroll
    for (int r = 0; r < X::kRpl; ++r) wv[r] = *reinterpret_cast<const float4*>(wp + r * (C + 4) + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      ulonglong2 vv[X::kVec];
#pragma unroll
      for (int u = 0; u < X::kVec; ++u) vv[u] = *reinterpret_cast<const ulonglong2*>(vp + (j + jj) * X::kStride + u * 128);
#pragma unroll
      for (int r = 0; r < X::kRpl; ++r) {
        if (kMask && !(j + jj >= lo[r] && j + jj < hi[r])) continue;
        const float x = jj == 0 ? wv[r].x : jj == 1 ? wv[r].y : jj == 2 ? wv[r].z : wv[r].w;
        const uint64_t x2 = ptx::pack_f2(x, x);
#pragma unroll
        for (int u = 0; u < X::kVec; ++u) {
          acc[r][2 * u] = ptx::fma_f2(x2, vv[u].x, acc[r][2 * u]);
          acc[r][2 * u + 1] = ptx::fma_f2(x2, vv[u].y, acc[r][2 * u + 1]);
        }
      }
    }
  }
}

// Which outer tile this CTA works on.  Row units: stacked rows of `cu` (stack per token).
struct Tile {
  int seg, rank, h;
  long long row0;  // first outer row of the tile within the segment
  bool any;
};
__device__ __forceinline__ Tile find_tile(const TileParams& p, const int32_t* cu, int stack) {
  Tile t;
  t.rank = (int)(blockIdx.x % (unsigned)p.splits);
  const long long unit = blockIdx.x / (unsigned)p.splits;
  t.h = (int)(unit % p.heads);
  const long long slot = unit / p.heads;
  SegSearch find(p.n_seg, kThreads);
  while (!find.done()) find.narrow(__syncthreads_count(find.starts_by(cu, stack, slot, threadIdx.x)), kThreads);
  t.seg = (int)find.lo;
  t.row0 = (slot - first_slot(cu, t.seg, stack)) * kRows;
  t.any = t.row0 >= 0 && t.row0 < ((long long)cu[t.seg + 1] - cu[t.seg]) * stack;
  return t;
}

// Column pieces of one accumulator row to global memory.
template <int DP, typename T>
__device__ __forceinline__ void store_row(T* dst, const float4* f, int D, int vec) {
  using X = Dim<DP>;
  const int lc = (threadIdx.x & 31) % X::kLanes;
#pragma unroll
  for (int u = 0; u < X::kVec; ++u) {
    const int c = lc * 4 + u * 128;
    if (c >= D) continue;
    if (vec) {
      store4(dst + c, f[u]);
    } else {
      dst[c] = from_float<T>(f[u].x);
      if (c + 1 < D) dst[c + 1] = from_float<T>(f[u].y);
      if (c + 2 < D) dst[c + 2] = from_float<T>(f[u].z);
      if (c + 3 < D) dst[c + 3] = from_float<T>(f[u].w);
    }
  }
}

// Accumulator -> out rows, summed over the cluster in rank order.  row_mul(r): factor of the tile's row r before the
// sum; row_fin(r, f): makes the sum the final value; buf: kRows x stride floats of shared memory that nobody
// reads any more.  Row r of the tile goes to out + r * out_row.
// Called by the ranks below n_ranks, which all pass the same n_ranks; the others have returned (a cluster barrier
// waits for the CTAs that have not exited).
template <int DP, typename T, typename Mul, typename Fin>
__device__ __forceinline__ void reduce_store(const TileParams& p, uint64_t (&acc)[Dim<DP>::kRpl][Dim<DP>::kVec * 2], float* buf, int n_ranks,
                                             int rank, int rows, T* out, int64_t out_row, int vec, Mul row_mul, Fin row_fin) {
  using X = Dim<DP>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = warp * 8 + (lane / X::kLanes) * X::kRpl;
  if (n_ranks <= 1) {
#pragma unroll
    for (int r = 0; r < X::kRpl; ++r) {
      if (first + r >= rows) continue;
      const float m = row_mul(first + r);
      float4 f[X::kVec];
#pragma unroll
      for (int u = 0; u < X::kVec; ++u) {
        ptx::unpack_f2(acc[r][2 * u], f[u].x, f[u].y);
        ptx::unpack_f2(acc[r][2 * u + 1], f[u].z, f[u].w);
        f[u].x *= m; f[u].y *= m; f[u].z *= m; f[u].w *= m;
        row_fin(first + r, f[u]);
      }
      store_row<DP>(out + (first + r) * out_row, f, p.D, vec);
    }
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
#pragma unroll
  for (int r = 0; r < X::kRpl; ++r) {
    const float m = row_mul(first + r);
#pragma unroll
    for (int u = 0; u < X::kVec; ++u) {
      float4 f;
      ptx::unpack_f2(acc[r][2 * u], f.x, f.y);
      ptx::unpack_f2(acc[r][2 * u + 1], f.z, f.w);
      f.x *= m; f.y *= m; f.z *= m; f.w *= m;
      *reinterpret_cast<float4*>(buf + (first + r) * X::kStride + (lane % X::kLanes) * 4 + u * 128) = f;
    }
  }
  cl.sync();
  // rank i finishes row groups of eight i, i + n_ranks, ...: one warp per row
  for (int r = rank * 8 + warp; r < rows; r += n_ranks * 8) {
    if (lane >= X::kLanes) continue;
    float4 f[X::kVec];
#pragma unroll
    for (int u = 0; u < X::kVec; ++u) f[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 0; i < n_ranks; ++i) {
      const float* src = cl.map_shared_rank(buf, i) + r * X::kStride + lane * 4;
#pragma unroll
      for (int u = 0; u < X::kVec; ++u) {
        const float4 x = *reinterpret_cast<const float4*>(src + u * 128);
        f[u].x += x.x; f[u].y += x.y; f[u].z += x.z; f[u].w += x.w;
      }
    }
#pragma unroll
    for (int u = 0; u < X::kVec; ++u) row_fin(r, f[u]);
    store_row<DP>(out + r * out_row, f, p.D, vec);
  }
  cl.sync();  // the other ranks may still be reading this CTA's part
}

// ---------------- forward -------------------------------------------------------------------------
template <int DP, bool kShared> constexpr int fwd_cols() { return DP == 256 && !kShared ? 32 : 64; }
template <int DP, bool kShared> constexpr size_t fwd_smem() {
  constexpr int C = fwd_cols<DP, kShared>();
  return sizeof(float) * ((size_t)Dim<DP>::kStride * (kRows + (kShared ? 1 : 2) * C) + kRows * (C + 4) + 4 * kRows);
}

template <typename T, int DP, bool kShared>
__global__ void __launch_bounds__(kThreads) tile_fwd_kernel(const TileParams p) {
  constexpr int C = fwd_cols<DP, kShared>(), J = C / 16;
  using X = Dim<DP>;
  extern __shared__ __align__(16) float smem[];
  float* sq = smem;
  float* sk = sq + kRows * X::kStride;
  float* sv = kShared ? sk : sk + C * X::kStride;
  float* sp = sv + C * X::kStride;
  float* st_m = sp + kRows * (C + 4);  // row maxima and sums of this CTA's share
  float* st_l = st_m + kRows;
  float* st_f = st_l + kRows;          // rescale factor of a block; later the factor of this CTA's share
  float* st_d = st_f + kRows;          // 1 / merged row sum, 0 for a row that saw no key
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane >> 4, cgl = lane & 15;

  const Tile t = find_tile(p, p.cu_q, p.stack);
  if (!t.any) return;  // the same for the whole cluster
  const int q0 = p.cu_q[t.seg], Lq = p.cu_q[t.seg + 1] - q0, k0 = p.cu_k[t.seg], Lk = p.cu_k[t.seg + 1] - k0;
  if (p.guard && (q0 < 0 || k0 < 0 || p.cu_q[t.seg + 1] < q0 || p.cu_q[t.seg + 1] > p.total_q ||
                  p.cu_k[t.seg + 1] < k0 || p.cu_k[t.seg + 1] > p.total_k))
    return;
  const long long row0 = (long long)q0 * p.stack + t.row0;  // first row of the tile in the whole batch
  const int rows = (int)min((long long)kRows, (long long)Lq * p.stack - t.row0);
  const int i0 = (int)t.row0;  // causal: stack is 1
  const int off = Lk - Lq;
  const int kmax = p.causal ? max(0, min(Lk, i0 + rows + off)) : Lk;  // keys the last row sees
  const int n_blk = (kmax + C - 1) / C;
  const int n_ranks = min(p.splits, max(1, n_blk));
  if (t.rank >= n_ranks) return;
  const float c = p.scale * kLog2e;

  const T* kb = (const T*)p.k + t.h * p.k_head + (int64_t)k0 * p.k_row;
  const T* vb = (const T*)p.v + t.h * p.v_head + (int64_t)k0 * p.v_row;
  load_tile<DP, kRows>(sq, (const T*)p.q + t.h * p.q_head + row0 * p.q_row, p.q_row, rows, p.D, p.vec_q, KeepAll());

  const bool live = warp * 8 < rows;
  float m[4], l[4];
  int kend[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    kend[i] = p.causal ? min(Lk, i0 + warp * 8 + rg * 4 + i + off + 1) : Lk;
  }
  uint64_t acc[X::kRpl][X::kVec * 2];
#pragma unroll
  for (int r = 0; r < X::kRpl; ++r)
#pragma unroll
    for (int u = 0; u < X::kVec * 2; ++u) acc[r][u] = 0ull;
  const int first = warp * 8 + (lane / X::kLanes) * X::kRpl;  // the lane's first row in the second product

  for (int b = t.rank; b < n_blk; b += p.splits) {
    const int j0 = b * C, n_keys = min(C, Lk - j0);
    __syncthreads();
    load_tile<DP, C>(sk, kb + (int64_t)j0 * p.k_row, p.k_row, n_keys, p.D, p.vec_k, KeepAll());
    if (!kShared) load_tile<DP, C>(sv, vb + (int64_t)j0 * p.v_row, p.v_row, n_keys, p.D, p.vec_v, KeepAll());
    tile_arrived();
    __syncthreads();
    if (!live) continue;
    float s[4][J];
    dot_block<DP, J>(sq + warp * 8 * X::kStride, sk, s);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        s[i][j] = (j0 + cgl + 16 * j < kend[i]) ? s[i][j] * c : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m[i], mx);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float corr = exp2f(m[i] - m_use);
      float* prow = sp + (warp * 8 + rg * 4 + i) * (C + 4);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const float x = exp2f(s[i][j] - m_use);
        sum += x;
        prow[cgl + 16 * j] = x;
      }
      l[i] = l[i] * corr + sum;
      m[i] = m_new;
      if (cgl == 0) st_f[warp * 8 + rg * 4 + i] = corr;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < X::kRpl; ++r) {
      const float f = st_f[first + r];
      const uint64_t f2 = ptx::pack_f2(f, f);
#pragma unroll
      for (int u = 0; u < X::kVec * 2; ++u) acc[r][u] = ptx::mul_f2(acc[r][u], f2);
    }
    const int n = (n_keys + 3) & ~3;
    if (p.causal && j0 + C > i0 + warp * 8 + off + 1) {
      int lo[X::kRpl], hi[X::kRpl];
#pragma unroll
      for (int r = 0; r < X::kRpl; ++r) {
        lo[r] = 0;
        hi[r] = i0 + first + r + off + 1 - j0;
      }
      add_weighted<DP, C, true>(acc, sp + warp * 8 * (C + 4), sv, n, lo, hi);
    } else {
      add_weighted<DP, C, false>(acc, sp + warp * 8 * (C + 4), sv, n, nullptr, nullptr);
    }
    __syncwarp();
  }
  tile_arrived();  // a share without a block has waited for nothing yet, and the rows' buffer is used again below

  // row statistics: the lanes of a row hold the sums of their own columns
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    if (cgl == 0) {
      st_m[warp * 8 + rg * 4 + i] = m[i];
      st_l[warp * 8 + rg * 4 + i] = l[i];
    }
  }
  if (n_ranks > 1) cg::this_cluster().sync(); else __syncthreads();
  if (threadIdx.x < kRows) {
    const int r = threadIdx.x;
    float mt = st_m[r], lt = st_l[r];
    if (n_ranks > 1) {
      cg::cluster_group cl = cg::this_cluster();
      mt = -INFINITY;
      for (int i = 0; i < n_ranks; ++i) mt = fmaxf(mt, *cl.map_shared_rank(st_m + r, i));
      const float mu = mt == -INFINITY ? 0.f : mt;
      lt = 0.f;
      for (int i = 0; i < n_ranks; ++i) lt += *cl.map_shared_rank(st_l + r, i) * exp2f(*cl.map_shared_rank(st_m + r, i) - mu);
      st_f[r] = exp2f(st_m[r] - mu);
    } else {
      st_f[r] = 1.f;
    }
    const bool dead = lt == 0.f;  // a NaN row sum is not a dead row: it goes out as NaN
    st_d[r] = dead ? 0.f : 1.f / lt;
    if (t.rank == 0 && r < rows)
      p.lse[p.stack > 1 ? row0 + r : (row0 + r) * p.H + t.h] = dead ? -INFINITY : mt + log2f(lt);
  }
  __syncthreads();
  reduce_store<DP>(p, acc, sq, n_ranks, t.rank, rows, (T*)p.o + t.h * p.q_head + row0 * p.q_row, p.q_row, p.vec_o,
                   [&](int r) { return st_f[r]; },
                   [&](int r, float4& f) {
                     const float d = st_d[r];
                     if (d == 0.f) { f = make_float4(0.f, 0.f, 0.f, 0.f); return; }
                     f.x *= d; f.y *= d; f.z *= d; f.w *= d;
                   });
}

// ---------------- dQ ------------------------------------------------------------------------------
template <int DP, bool kShared> constexpr int dq_cols() { return DP == 256 && !kShared ? 32 : 64; }
template <int DP, bool kShared> constexpr size_t dq_smem() {
  constexpr int C = dq_cols<DP, kShared>();
  return sizeof(float) * ((size_t)Dim<DP>::kStride * (2 * kRows + (kShared ? 1 : 2) * C) + kRows * (C + 4) + kRows);
}

template <typename T, typename TDO, int DP, bool kShared>
__global__ void __launch_bounds__(kThreads) tile_dq_kernel(const TileParams p) {
  constexpr int C = dq_cols<DP, kShared>(), J = C / 16;
  using X = Dim<DP>;
  extern __shared__ __align__(16) float smem[];
  float* sq = smem;
  float* sd = sq + kRows * X::kStride;
  float* sk = sd + kRows * X::kStride;
  float* sv = kShared ? sk : sk + C * X::kStride;
  float* sp = sv + C * X::kStride;
  float* st_z = sp + kRows * (C + 4);  // 0: the row saw no key
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane >> 4, cgl = lane & 15;

  const Tile t = find_tile(p, p.cu_q, p.stack);
  if (!t.any) return;
  const int q0 = p.cu_q[t.seg], Lq = p.cu_q[t.seg + 1] - q0, k0 = p.cu_k[t.seg], Lk = p.cu_k[t.seg + 1] - k0;
  const long long row0 = (long long)q0 * p.stack + t.row0;
  const int rows = (int)min((long long)kRows, (long long)Lq * p.stack - t.row0);
  const int i0 = (int)t.row0;
  const int off = Lk - Lq;
  const int kmax = p.causal ? max(0, min(Lk, i0 + rows + off)) : Lk;
  const int n_blk = (kmax + C - 1) / C;
  const int n_ranks = min(p.splits, max(1, n_blk));
  if (t.rank >= n_ranks) return;
  const float c = p.scale * kLog2e;

  const T* kb = (const T*)p.k + t.h * p.k_head + (int64_t)k0 * p.k_row;
  const T* vb = (const T*)p.v + t.h * p.v_head + (int64_t)k0 * p.v_row;
  load_tile<DP, kRows>(sq, (const T*)p.q + t.h * p.q_head + row0 * p.q_row, p.q_row, rows, p.D, p.vec_q, KeepAll());
  load_tile<DP, kRows>(sd, (const TDO*)p.d_o + t.h * p.do_head + row0 * p.do_row, p.do_row, rows, p.D, p.vec_do, KeepAll());
  const bool live = warp * 8 < rows;
  float lse[4], dl[4];
  int kend[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp * 8 + rg * 4 + i;
    lse[i] = -INFINITY;
    dl[i] = 0.f;
    if (r < rows) {
      const long long e = p.stack > 1 ? row0 + r : (row0 + r) * p.H + t.h;
      lse[i] = p.lse[e];
      dl[i] = p.delta[e];
    }
    kend[i] = p.causal ? min(Lk, i0 + r + off + 1) : Lk;
    if (lse[i] == -INFINITY) kend[i] = 0;
    if (cgl == 0) st_z[r] = lse[i] == -INFINITY ? 0.f : 1.f;
  }
  uint64_t acc[X::kRpl][X::kVec * 2];
#pragma unroll
  for (int r = 0; r < X::kRpl; ++r)
#pragma unroll
    for (int u = 0; u < X::kVec * 2; ++u) acc[r][u] = 0ull;
  const int first = warp * 8 + (lane / X::kLanes) * X::kRpl;

  for (int b = t.rank; b < n_blk; b += p.splits) {
    const int j0 = b * C, n_keys = min(C, Lk - j0);
    __syncthreads();
    load_tile<DP, C>(sk, kb + (int64_t)j0 * p.k_row, p.k_row, n_keys, p.D, p.vec_k, KeepAll());
    if (!kShared) load_tile<DP, C>(sv, vb + (int64_t)j0 * p.v_row, p.v_row, n_keys, p.D, p.vec_v, KeepAll());
    tile_arrived();
    __syncthreads();
    if (!live) continue;
    float s[4][J], dp[4][J];
    dot_block<DP, J>(sq + warp * 8 * X::kStride, sk, s);
    dot_block<DP, J>(sd + warp * 8 * X::kStride, sv, dp);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* prow = sp + (warp * 8 + rg * 4 + i) * (C + 4);
#pragma unroll
      for (int j = 0; j < J; ++j)
        prow[cgl + 16 * j] = (j0 + cgl + 16 * j < kend[i]) ? exp2f(s[i][j] * c - lse[i]) * (dp[i][j] - dl[i]) : 0.f;
    }
    __syncwarp();
    const int n = (n_keys + 3) & ~3;
    if (p.causal && j0 + C > i0 + warp * 8 + off + 1) {
      int lo[X::kRpl], hi[X::kRpl];
#pragma unroll
      for (int r = 0; r < X::kRpl; ++r) {
        lo[r] = 0;
        hi[r] = i0 + first + r + off + 1 - j0;
      }
      add_weighted<DP, C, true>(acc, sp + warp * 8 * (C + 4), sk, n, lo, hi);
    } else {
      add_weighted<DP, C, false>(acc, sp + warp * 8 * (C + 4), sk, n, nullptr, nullptr);
    }
    __syncwarp();
  }
  tile_arrived();  // a share without a block has waited for nothing yet
  __syncthreads();
  reduce_store<DP>(p, acc, sq, n_ranks, t.rank, rows, (T*)p.dq + t.h * p.q_head + row0 * p.q_row, p.q_row, p.vec_o,
                   [&](int) { return 1.f; },
                   [&](int r, float4& f) {
                     if (st_z[r] == 0.f) { f = make_float4(0.f, 0.f, 0.f, 0.f); return; }
                     f.x *= p.scale; f.y *= p.scale; f.z *= p.scale; f.w *= p.scale;
                   });
}

// ---------------- dK, dV (shared K/V rows: one output, the sum of both over all heads) --------------------------
template <int DP> constexpr int dkv_cols() { return DP == 256 ? 32 : 64; }
template <int DP, bool kShared> constexpr size_t dkv_smem() {
  constexpr int C = dkv_cols<DP>();
  return sizeof(float) * ((size_t)Dim<DP>::kStride * ((kShared ? 1 : 2) * kRows + 2 * C) + 2 * kRows * (C + 4) + 2 * C);
}

template <typename T, typename TDO, int DP, bool kShared>
__global__ void __launch_bounds__(kThreads) tile_dkv_kernel(const TileParams p) {
  constexpr int C = dkv_cols<DP>(), J = C / 16;
  using X = Dim<DP>;
  extern __shared__ __align__(16) float smem[];
  float* sk = smem;
  float* sv = kShared ? sk : sk + kRows * X::kStride;
  float* sq = sv + kRows * X::kStride;
  float* sd = sq + C * X::kStride;
  float* sp = sd + C * X::kStride;      // P^T
  float* ss = sp + kRows * (C + 4);     // dS^T
  float* st_lse = ss + kRows * (C + 4);
  float* st_dl = st_lse + C;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane >> 4, cgl = lane & 15;

  const Tile t = find_tile(p, p.cu_k, 1);
  if (!t.any) return;
  const int q0 = p.cu_q[t.seg], Lq = p.cu_q[t.seg + 1] - q0, k0 = p.cu_k[t.seg], Lk = p.cu_k[t.seg + 1] - k0;
  const long long krow0 = k0 + t.row0;
  const int rows = (int)min((long long)kRows, (long long)Lk - t.row0);
  const int j0 = (int)t.row0;
  const int off = Lk - Lq;
  const long long n_inner = (long long)Lq * p.stack;
  const int ibeg = p.causal ? max(0, j0 - off) : 0;  // first query row that sees the tile's first key
  const int n_blk = (int)max(0LL, (n_inner - ibeg + C - 1) / C);
  const int n_ranks = min(p.splits, max(1, n_blk));
  if (t.rank >= n_ranks) return;
  const float c = p.scale * kLog2e;

  load_tile<DP, kRows>(sk, (const T*)p.k + t.h * p.k_head + krow0 * p.k_row, p.k_row, rows, p.D, p.vec_k, KeepAll());
  if (!kShared) load_tile<DP, kRows>(sv, (const T*)p.v + t.h * p.v_head + krow0 * p.v_row, p.v_row, rows, p.D, p.vec_v, KeepAll());
  const bool live = warp * 8 < rows;
  uint64_t acc_k[X::kRpl][X::kVec * 2], acc_v[X::kRpl][X::kVec * 2];
#pragma unroll
  for (int r = 0; r < X::kRpl; ++r)
#pragma unroll
    for (int u = 0; u < X::kVec * 2; ++u) acc_k[r][u] = acc_v[r][u] = 0ull;
  const int first = warp * 8 + (lane / X::kLanes) * X::kRpl;
  const long long seg_row = (long long)q0 * p.stack;

  for (int b = t.rank; b < n_blk; b += p.splits) {
    const long long r0 = ibeg + (long long)b * C;  // first inner row of the block within the segment
    const int n_in = (int)min((long long)C, n_inner - r0);
    const long long g0 = seg_row + r0;
    __syncthreads();
    if (threadIdx.x < C) {
      float a = -INFINITY, d = 0.f;
      if ((int)threadIdx.x < n_in) {
        const long long e = p.stack > 1 ? g0 + threadIdx.x : (g0 + threadIdx.x) * p.H + t.h;
        a = p.lse[e];
        d = p.delta[e];
      }
      st_lse[threadIdx.x] = a;
      st_dl[threadIdx.x] = d;
    }
    __syncthreads();
    // rows that saw no key take no part, whatever they hold
    auto seen = [&](int r) { return st_lse[r] != -INFINITY; };
    load_tile<DP, C>(sq, (const T*)p.q + t.h * p.q_head + g0 * p.q_row, p.q_row, n_in, p.D, p.vec_q, seen);
    load_tile<DP, C>(sd, (const TDO*)p.d_o + t.h * p.do_head + g0 * p.do_row, p.do_row, n_in, p.D, p.vec_do, seen);
    tile_arrived();
    __syncthreads();
    if (!live) continue;
    float s[4][J], dp[4][J];
    dot_block<DP, J>(sk + warp * 8 * X::kStride, sq, s);
    dot_block<DP, J>(sv + warp * 8 * X::kStride, sd, dp);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = warp * 8 + rg * 4 + i;
      // causal: key j is seen by query rows i >= j - off
      const int lo = p.causal ? j0 + r - off - (int)r0 : 0;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int col = cgl + 16 * j;
        const float ls = st_lse[col];
        const bool ok = col >= lo && ls != -INFINITY;
        const float x = ok ? exp2f(s[i][j] * c - ls) : 0.f;
        const float y = ok ? x * (dp[i][j] - st_dl[col]) : 0.f;
        sp[r * (C + 4) + col] = x;
        ss[r * (C + 4) + col] = y;
      }
    }
    __syncwarp();
    const int n = (n_in + 3) & ~3;
    const float* wp = sp + warp * 8 * (C + 4);
    const float* ws = ss + warp * 8 * (C + 4);
    if (p.causal && j0 + warp * 8 + 7 - off - r0 > 0) {
      int lo[X::kRpl], hi[X::kRpl];
#pragma unroll
      for (int r = 0; r < X::kRpl; ++r) {
        lo[r] = j0 + first + r - off - (int)r0;
        hi[r] = C;
      }
      add_weighted<DP, C, true>(acc_v, wp, sd, n, lo, hi);
      add_weighted<DP, C, true>(acc_k, ws, sq, n, lo, hi);
    } else {
      add_weighted<DP, C, false>(acc_v, wp, sd, n, nullptr, nullptr);
      add_weighted<DP, C, false>(acc_k, ws, sq, n, nullptr, nullptr);
    }
    __syncwarp();
  }
  tile_arrived();  // a share without a block has waited for nothing yet
  __syncthreads();
  const float mul = kShared ? 1.f : p.scale;
  if (kShared) {
    // one output: scale * dK + dV
    const uint64_t s2 = ptx::pack_f2(p.scale, p.scale);
#pragma unroll
    for (int r = 0; r < X::kRpl; ++r)
#pragma unroll
      for (int u = 0; u < X::kVec * 2; ++u) acc_k[r][u] = ptx::fma_f2(acc_k[r][u], s2, acc_v[r][u]);
  }
  reduce_store<DP>(p, acc_k, sk, n_ranks, t.rank, rows, (T*)p.dk + t.h * p.k_head + krow0 * p.k_row, p.k_row, p.vec_o,
                   [&](int) { return 1.f; }, [&](int, float4& f) { f.x *= mul; f.y *= mul; f.z *= mul; f.w *= mul; });
  if constexpr (!kShared)
    reduce_store<DP>(p, acc_v, sv, n_ranks, t.rank, rows, (T*)p.dv + t.h * p.v_head + krow0 * p.v_row, p.v_row, p.vec_o,
                     [&](int) { return 1.f; }, [&](int, float4&) {});
}

// ---------------- launches ------------------------------------------------------------------------
inline int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  return n;
}

// Four elements at a time: base and both strides on a 4-element boundary, and a row that ends on one.
inline int vec4(const void* p, int64_t row, int64_t head, int D, int es) {
  return D % 4 == 0 && row % 4 == 0 && head % 4 == 0 && reinterpret_cast<uintptr_t>(p) % (4 * es) == 0;
}

inline long long max_slots(long long tokens, int stack, int n_seg) { return tokens * stack / kRows + n_seg; }

// Cluster size: CTAs that share an outer tile.  The lengths are not known here, only their mean, and the longest
// segment decides the time of a ragged batch, so the tile is shared while the mean segment has inner blocks of
// 64 rows for more than the ranks so far, until the grid holds eight tiles per SM.  With no more blocks than ranks
// the new ranks of most tiles return at once, and each costs a launch slot with the tile's shared memory: forward of
// users of one target, fp32, one rank more from as many blocks as ranks | from one more: 1024 users x 64 keys 267 | 153 us, 512 x 64
// 126 | 81, 1024 x 96 339 | 241; 64 users x 8 targets x 370 keys 128 | 130.
// (A grid of less than two CTAs per SM has room for them, and the segments above the mean use them.)
inline int pick_splits(long long tiles, long long inner_rows, int n_seg) {
  const long long mean = inner_rows / n_seg, sms = sm_count();
  int n = 1;
  while (n < kMaxSplits && tiles * n < 8 * sms && mean >= 64 * (tiles * n < 2 * sms ? n : n + 1)) n *= 2;
  return n;
}

inline TileParams tile_params(const SimtAttnParams& a) {
  TileParams p;
  p.q = a.q; p.k = a.k; p.v = a.v; p.d_o = a.d_o; p.o = a.o; p.dq = a.dq; p.dk = a.dk; p.dv = a.dv;
  p.lse = a.lse; p.delta = a.delta; p.cu_q = a.cu_q; p.cu_k = a.cu_k;
  p.n_seg = a.n_seg; p.D = a.D; p.H = a.H;
  p.heads = a.shared_kv ? 1 : a.H;
  p.stack = a.shared_kv ? a.H : 1;
  // stacked heads are consecutive rows of the [tokens * H, D] view
  p.q_row = a.shared_kv ? a.q_head : a.q_row;  p.q_head = a.shared_kv ? 0 : a.q_head;
  p.do_row = a.shared_kv ? a.do_head : a.do_row;  p.do_head = a.shared_kv ? 0 : a.do_head;
  p.k_row = a.k_row; p.k_head = a.k_head; p.v_row = a.v_row; p.v_head = a.v_head;
  const int es = elem_size(a.dtype);
  p.vec_q = vec4(a.q, p.q_row, p.q_head, a.D, es);
  p.vec_k = vec4(a.k, p.k_row, p.k_head, a.D, es);
  p.vec_v = vec4(a.v, p.v_row, p.v_head, a.D, es);
  p.vec_do = vec4(a.d_o, p.do_row, p.do_head, a.D, a.do_f32 ? 4 : es);
  p.vec_o = 0;
  p.causal = a.causal; p.scale = a.scale;
  p.total_q = a.total_q; p.total_k = a.total_k; p.guard = a.guard;
  p.splits = 1; p.slots = 0;
  return p;
}

template <typename K>
int launch(K kernel, size_t smem, const TileParams& p, const char* name, cudaStream_t s) {
  VAFA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.slots * p.heads * p.splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = p.splits;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  VAFA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, p));
  VAFA_LAUNCH_CHECK(name);
  return 0;
}

template <typename F>
int by_dim(int D, F f) {
  if (D <= 32) return f(std::integral_constant<int, 32>{});
  if (D <= 64) return f(std::integral_constant<int, 64>{});
  if (D <= 128) return f(std::integral_constant<int, 128>{});
  return f(std::integral_constant<int, 256>{});
}
template <typename F>
int by_type(int dtype, F f) {
  switch (dtype) {
    case VAFA_F32: return f(float{});
    case VAFA_BF16: return f(__nv_bfloat16{});
    case VAFA_F16: return f(__half{});
    default: return fail(VAFA_ERR_INVALID, "unknown dtype %d", dtype);
  }
}

}  // namespace tiles
}  // namespace vafa

// Absorb operator, backward core for users with at most 64 stacked query rows (64 / H queries): dU and dX of a user from one
// pass over the user's X rows (tcgen05 + TMA + TMEM).  Users with more queries keep the two kernels of sm100_varlen_bwd.cu.
//
// An item is a user.  U and dAlphaX (64 stacked rows each) stay in shared memory, X streams through it in tiles of 128 keys.
// Keys are the rows of all products (TMEM lanes), so nothing is computed for the 64 to 120 padding rows that a
// 128-row tile of the user's queries would have.  Per tile
//     S  = X U^T, Y = X dAlphaX^T                                    [128 keys, R query rows]
//     P  = 2^(c S - lse),  dS = P (Y - delta),  dS' = P (scale Y - scale delta)
//     dU^T += X^T dS                                                 [256, R]   TMEM, for the whole item; dU = scale (dU^T)^T
//     dX  = (w P dAlphaX + w dS' U) / w                              [128 keys, 256]
// What is rounded to 16 bits is what the pair rounds, P and dS' in dX, dS in dU, so the results differ from the pair's in the order
// of the fp32 sums alone.  w is a power of two that changes no bit of P or dS', but keeps dS' of fp16 out of the subnormal numbers
// when the scale is small (see range_factor).  dS lies in shared memory as a [key][row] tile
// with the 128-byte swizzle, the MN-major B operand of dU^T; P and dS' go over the columns of Y as those are read, as the
// A operands of dX.  S is free once it has been read, so that of the next tile runs under this one's element-wise work;
// Y follows dX, under its epilogue.  dX leaves through the slot of its X tile, which dU^T was the last to
// read: the rows of a tile are one piece of the output, and a warp of its own sends them off with one bulk copy.
// (Stored from registers, in pieces of 64 bytes per row, the 55 KB of a tile held the warps up for 4400 of 7500 cycles.)
// TMEM (512 columns): S [0,64) Y, later P and dS' [64,128) dX [128,384) dU^T [384,448) (d_kv 0-127) and [448,512) (128-255).
//
// The pair of kernels reads X twice, and its dU kernel multiplies 128-row query tiles by 64-key blocks: 4600 tensor cycles per 128
// keys where the three products here that replace it take 2300.  What bounds it: X in and dX out are 110 KB per tile at
// a width of 216, 4800 cycles of an SM's share of HBM, against about 3300 cycles of products.
// A step of 1137 users of 1-10 queries over 2048 keys of width 216: 1649 us with the pair for all, 1288 with this kernel for the 80 %
// it takes; of 1024 users of 1-16 queries over 8-2048 keys of width 256: 551 and 529.
// Rounding one P / scale and one dS for both results instead, with P as a second shared-memory tile, was 0.5 % faster (1175 and 1180 us of
// the first step as it is now, 421 and 424 of the second), but moved dX by 0.17 to 0.27 % and lost bits of fp16 at scales above 1.
//
// Reference: triton_target_attn_absorb/triton_target_attn_absorb/kernels.py:287-474 (dU, dX).
#include <cuda.h>
#include <type_traits>

#include "profile.cuh"
#include "sm100_common.cuh"
#include "sm100_kernels.cuh"

namespace vafa {
namespace {

using namespace ptx;

// Optional wait-time tracing (build with -DVAFA_TRACE), as in sm100_varlen_fwd.cu.
#ifdef VAFA_TRACE
#define TRACE_T0() const long long _t0 = clock64()
#define TRACE_ADD(slot) tr[slot] += clock64() - _t0
#else
#define TRACE_T0()
#define TRACE_ADD(slot)
#endif

constexpr int kDxuThreads = 352;  // 8 element-wise warps, 1 TMA warp, 1 MMA warp, 1 warp that stores dX
constexpr int kRows = 64;         // stacked query rows of an item
constexpr int kKv = 256;
constexpr int kRowSub = kRows * 128, kKeySub = kTile * 128;  // one 64-column sub tile of U / dAlphaX, of X
constexpr uint32_t kSCol = 0, kYCol = 64, kDxCol = 128, kDuCol = 384;

struct DxuSmem {
  alignas(1024) uint8_t u[4 * kRowSub];
  alignas(1024) uint8_t g[4 * kRowSub];
  alignas(1024) uint8_t x[2][4 * kKeySub];
  alignas(1024) uint8_t ds[kTile * 128];
  alignas(16) float nl[2][kRows], nd[2][kRows], nds[2][kRows];  // [item parity]: -lse (-inf past the last row), -delta, -scale delta
  alignas(8) uint64_t ug_full, ug_empty, x_full[2], x_empty[2];
  uint64_t sy_full, s_free, pds_full, dx_done, nl_full, stage_full[2];
  WorkQueue wq;
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;  // read by the bounded waits as abort_flag[1]: keep it right behind abort_flag
};
static_assert(sizeof(DxuSmem) + 1024 <= 227 * 1024, "shared memory budget");

struct DxuParams {
  void* du;
  void* dx;
  const float2* ld;  // (lse, delta) per stacked row
  const float* nl;   // the same planar, as -lse and -delta * scale
  const float* nds;
  const SchedHeader* header;
  const WorkItem* items;  // o_start / o_rows: the user's queries, i_start / i_len: the user's keys
  int H;
  int x_width;
  int which;  // 0: dU and dX; 1: dU only; 2: dX only (a backward in two phases; the same bits as both at once)
  float scale, scale_log2;
  float range, inv_range;  // w, 1 / w
  int32_t* status;
  int wait_limit;  // bound of every device-side wait, in units of 65536 cycles
  long long* trace;
};

// How dX of a tile lies in its slot: as the packed rows of the output, which one bulk copy sends off; or, where rows are a
// multiple of 128 bytes and would start in the same bank, as 64-column boxes with the 128-byte swizzle, which a tiled store takes
// (whole tiles only: a box has 128 rows).  Turning 4 x 4 pieces by shuffles between the lanes instead took three times as
// long as the writes, and a bulk copy per row longer than the tile's products.
__device__ __forceinline__ bool boxed_dx(int x_width, int rows) { return x_width % 64 == 0 && rows == kTile; }

template <typename T>
__global__ void __launch_bounds__(kDxuThreads, 1)
absorb_dxu_kernel(const __grid_constant__ CUtensorMap tmap_u, const __grid_constant__ CUtensorMap tmap_g,
                  const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_dx, const DxuParams p) {
  extern __shared__ uint8_t smem_raw[];
  DxuSmem& sm = *reinterpret_cast<DxuSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  volatile int* abort_flag = &sm.abort_flag;

  if (threadIdx.x == 0) {
    sm.abort_flag = 0;
    sm.wait_limit = p.wait_limit;
    wq_init(sm.wq, 10);
    mbar_init(smem_u32(&sm.ug_full), 1);
    mbar_init(smem_u32(&sm.ug_empty), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sm.x_full[i]), 1);
      mbar_init(smem_u32(&sm.x_empty[i]), 1);
      mbar_init(smem_u32(&sm.stage_full[i]), 8);  // one arrival per element-wise warp
    }
    mbar_init(smem_u32(&sm.sy_full), 1);
    mbar_init(smem_u32(&sm.s_free), 8);
    mbar_init(smem_u32(&sm.pds_full), 8);
    mbar_init(smem_u32(&sm.dx_done), 1);
    mbar_init(smem_u32(&sm.nl_full), kRows);
    fence_barrier_init();
  }
  if (warp == 8 && lane == 0) {
    prefetch_tensormap(&tmap_u);
    prefetch_tensormap(&tmap_g);
    prefetch_tensormap(&tmap_x);
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&sm.tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sm.tmem_base;

  const int n_items = p.header->n_items;
  const int total = max(n_items, 0);
  int* const next_item = const_cast<int*>(p.which == 2 ? &p.header->next_item_2 : &p.header->next_item);
  if (n_items < 0 && threadIdx.x == 0) report_error(p.status, 2, 150, n_items);
#ifdef VAFA_TRACE
  long long tr[16];
  for (int i = 0; i < 16; ++i) tr[i] = 0;
  const long long t_begin = clock64();
#endif

  if (warp == 8) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      constexpr int kPrefetch = 4;  // tiles of an item pulled into L2 ahead of their load
      uint32_t gk = 0, qi = 0;
      bool alive = true;
      WorkItem w;
      int idx = wq_produce_item(sm.wq, 0, next_item, total, p.items, w, abort_flag);
      for (uint32_t n = 0; alive && idx >= 0; ++n) {
        const int nt = (w.i_len + kTile - 1) / kTile;
        for (int t = 0; t < nt; ++t, ++gk) {
          const int st = gk & 1;
          const int row = w.i_start + t * kTile;
          if (t + kPrefetch < nt)
            for (int c = 0; c < 4; ++c) tma_prefetch_3d(&tmap_x, c * 64, 0, row + kPrefetch * kTile);
          { TRACE_T0(); if (!mbar_wait(smem_u32(&sm.x_empty[st]), ((gk >> 1) & 1) ^ 1, abort_flag)) { alive = false; break; } TRACE_ADD(0); }
          mbar_expect_tx(smem_u32(&sm.x_full[st]), 4 * kKeySub);
          for (int c = 0; c < 4; ++c) tma_load_3d(smem_u32(sm.x[st]) + c * kKeySub, &tmap_x, smem_u32(&sm.x_full[st]), c * 64, 0, row);
          if (t == 0) {
            { TRACE_T0(); if (!mbar_wait(smem_u32(&sm.ug_empty), (qi & 1) ^ 1, abort_flag)) { alive = false; break; } TRACE_ADD(1); }
            mbar_expect_tx(smem_u32(&sm.ug_full), 8 * kRowSub);
            for (int c = 0; c < 4; ++c) {
              tma_load_3d(smem_u32(sm.u) + c * kRowSub, &tmap_u, smem_u32(&sm.ug_full), c * 64, 0, w.o_start);
              tma_load_3d(smem_u32(sm.g) + c * kRowSub, &tmap_g, smem_u32(&sm.ug_full), c * 64, 0, w.o_start);
            }
          }
        }
        if (nt > 0) ++qi;
        // the next item is drawn while this one is worked on, and its first tiles pulled into L2
        idx = alive ? wq_produce_item(sm.wq, n + 1, next_item, total, p.items, w, abort_flag) : -1;
        if (idx >= 0) {
          for (int c = 0; c < 4; ++c) {
            tma_prefetch_3d(&tmap_u, c * 64, 0, w.o_start);
            tma_prefetch_3d(&tmap_g, c * 64, 0, w.o_start);
          }
          for (int t = 0; t < kPrefetch && t * kTile < w.i_len; ++t)
            for (int c = 0; c < 4; ++c) tma_prefetch_3d(&tmap_x, c * 64, 0, w.i_start + t * kTile);
        }
      }
    }
  } else if (warp == 10) {
    // ---------------- dX tiles to global memory ----------------
    uint32_t g = 0;
    bool alive = true;
    for (uint32_t n = 0; alive; ++n) {
      WorkItem w;
      if (wq_consume_item(sm.wq, n, w, abort_flag) < 0) break;
      for (int t = 0; t * kTile < w.i_len; ++t, ++g) {
        if (!mbar_wait(smem_u32(&sm.stage_full[g & 1]), (g >> 1) & 1, abort_flag)) { alive = false; break; }
        if (lane == 0 && p.which != 1) {
          const int row = w.i_start + t * kTile, rows = min(kTile, w.i_len - t * kTile);
          const uint32_t stage = smem_u32(sm.x[g & 1]);
          if (boxed_dx(p.x_width, rows)) {
            for (int c = 0; c < p.x_width / 64; ++c) tma_store_3d(&tmap_dx, stage + c * kKeySub, c * 64, 0, row);
            bulk_store_commit();
          } else {
            bulk_store_1d(reinterpret_cast<T*>(p.dx) + (long long)row * p.x_width, stage, (uint32_t)(rows * p.x_width * 2));
          }
          bulk_store_wait_read();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.x_empty[g & 1]));
      }
    }
    if (lane == 0) bulk_store_wait();
  } else if (warp == 9) {
    // ---------------- MMA issuer: the whole warp on warp-uniform values, one elected lane issues ----------------
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t idesc_du = make_idesc(kFmt, 1, 1, 128, kRows);  // both operands MN-major
    constexpr uint32_t idesc_dx = make_idesc(kFmt, 0, 1, 128, kKv);    // A from TMEM, B MN-major
    const uint32_t tm = warp_uniform(tbase);
    const uint32_t u_k = warp_uniform(desc_lo_sw128(smem_u32(sm.u), 16)), g_k = warp_uniform(desc_lo_sw128(smem_u32(sm.g), 16));
    const uint32_t u_mn = warp_uniform(desc_lo_sw128(smem_u32(sm.u), kRowSub)), g_mn = warp_uniform(desc_lo_sw128(smem_u32(sm.g), kRowSub));
    const uint32_t x_k0 = warp_uniform(desc_lo_sw128(smem_u32(sm.x[0]), 16)), x_mn0 = warp_uniform(desc_lo_sw128(smem_u32(sm.x[0]), kKeySub));
    const uint32_t ds_mn = warp_uniform(desc_lo_sw128(smem_u32(sm.ds), kKeySub));
    constexpr uint32_t kStage16 = 4 * kKeySub >> 4;
    uint32_t gk = 0, qi = 0;
    bool alive = true;

    // S or Y of tile g over the first `n` query rows
    auto issue_score = [&](uint32_t g, uint32_t n, uint32_t col, uint32_t b_lo) {
      const uint32_t x_lo = x_k0 + (g & 1) * kStage16;
      const uint32_t idesc = make_idesc(kFmt, 0, 0, 128, 0) | (n >> 3) << 17;
#pragma unroll
      for (int kk = 0; kk < kKv / 16; ++kk)
        mma_ss2(tm + col, x_lo + (kk >> 2) * (kKeySub >> 4) + (kk & 3) * 2, b_lo + (kk >> 2) * (kRowSub >> 4) + (kk & 3) * 2, idesc, kk > 0);
    };
    auto issue_s = [&](uint32_t g, uint32_t n) -> bool {
      { TRACE_T0(); if (!mbar_wait_warp(smem_u32(&sm.s_free), (g & 1) ^ 1, abort_flag)) return false; TRACE_ADD(5); }  // that of tile g - 1 has been read
      { TRACE_T0(); if (!mbar_wait_warp(smem_u32(&sm.x_full[0]) + (g & 1) * 8, (g >> 1) & 1, abort_flag)) return false; TRACE_ADD(4); }
      tc_fence_after();
      TRACE_T0();
      if (elect_one()) issue_score(g, n, kSCol, u_k);
      __syncwarp();
      TRACE_ADD(2);
      return true;
    };
    // (behind dX of tile g - 1, which reads P and dS' from these columns: the pipe runs in order)
    auto issue_y = [&](uint32_t g, uint32_t n) {
      if (elect_one()) {
        issue_score(g, n, kYCol, g_k);
        mma_commit(smem_u32(&sm.sy_full));
      }
      __syncwarp();
    };

    for (uint32_t n = 0; alive; ++n) {
      WorkItem w;
      const int idx = (int)warp_uniform((uint32_t)wq_consume_item(sm.wq, n, w, abort_flag));
      if (idx < 0) break;
      const int i_len = (int)warp_uniform((uint32_t)w.i_len);
      const int row_steps = (int)warp_uniform((uint32_t)((w.o_rows * p.H + 15) / 16));
      const int nt = (i_len + kTile - 1) / kTile;
      if (nt == 0) continue;
      { TRACE_T0(); if (!mbar_wait_warp(smem_u32(&sm.ug_full), qi & 1, abort_flag)) break; TRACE_ADD(3); }
      ++qi;
      tc_fence_after();
      if (!issue_s(gk, row_steps * 16)) break;
      issue_y(gk, row_steps * 16);
      for (int t = 0; t < nt; ++t) {
        const uint32_t g = gk + t;
        // the next tile's scores, where the tile is there before P and dS of this one
        bool s_due = t + 1 < nt;
        if (s_due) {
          const int first = (int)warp_uniform((uint32_t)mbar_wait_either(smem_u32(&sm.x_full[0]) + ((g + 1) & 1) * 8, ((g + 1) >> 1) & 1,
                                                                         smem_u32(&sm.pds_full), g & 1, abort_flag));
          if (first == 0 || (first == 1 && !issue_s(g + 1, row_steps * 16))) { alive = false; break; }
          s_due = first != 1;
        }
        { TRACE_T0(); if (!mbar_wait_warp(smem_u32(&sm.pds_full), g & 1, abort_flag)) { alive = false; break; } TRACE_ADD(6); }
        tc_fence_after();
        // keys past the user's last are zeros in dS; those past the 16-key step of the last are not multiplied
        const int key_steps = (min(kTile, i_len - t * kTile) + 15) / 16;
        const uint32_t x_lo = x_mn0 + (g & 1) * kStage16;
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk)
              if (kk < key_steps && p.which != 2) mma_ss2(tm + kDuCol + h * kRows, x_lo + h * (2 * kKeySub >> 4) + kk * (2048 >> 4), ds_mn + kk * (2048 >> 4), idesc_du,
                      (t > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < kRows / 16; ++kk) {
            if (kk >= row_steps || p.which == 1) break;
            const uint32_t a = tm + kYCol + (kk >> 1) * 32 + (kk & 1) * 8;  // a thread's 32 columns: 16 of P, 16 of dS'
            mma_ts2(tm + kDxCol, a, g_mn + kk * (2048 >> 4), idesc_dx, kk > 0 ? 1u : 0u);
            mma_ts2(tm + kDxCol, a + 16, u_mn + kk * (2048 >> 4), idesc_dx, 1u);
          }
          mma_commit(smem_u32(&sm.dx_done));
          if (t + 1 == nt) mma_commit(smem_u32(&sm.ug_empty));
        }
        __syncwarp();
        if (s_due && !issue_s(g + 1, row_steps * 16)) { alive = false; break; }
        if (t + 1 < nt) issue_y(g + 1, row_steps * 16);
      }
      gk += nt;
    }
  } else {
    // ---------------- element-wise warps + epilogues (warps 0-7) ----------------
    // thread -> key row r of the tile (TMEM lane; a warp may only touch lane quadrant warp % 4); warps 0-3 take the query
    // rows [0,32) and the output columns [0,128), warps 4-7 the others
    const int r = threadIdx.x & 127;
    const int half = threadIdx.x >> 7;
    const uint32_t lane_base = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    const uint64_t c2 = pack_f2(p.scale_log2, p.scale_log2), s2 = pack_f2(p.scale, p.scale), w2 = pack_f2(p.range, p.range);
    uint32_t gk = 0, par = 0;
    bool alive = true;
    // dX of the tile, scaled back and rounded, over its X tile (see boxed_dx)
    auto epilogue_dx = [&](uint8_t* stage, int rows) {
      if (p.which == 1) return;
      const bool boxed = boxed_dx(p.x_width, rows);
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4) {
        const int cc = half * 4 + c4;
        const int pieces = min(4, (p.x_width - cc * 32) / 8);
        if (pieces <= 0) continue;
        uint32_t t[32], pw[16];
        tmem_ld32(lane_base + kDxCol + cc * 32, t);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          pw[i] = pack2_out<T>(__uint_as_float(t[2 * i]) * p.inv_range, __uint_as_float(t[2 * i + 1]) * p.inv_range);
        // (rows past the last are left out: with rows of 512 bytes each is a bank conflict)
        uint8_t* const dst = boxed ? stage + (cc >> 1) * kKeySub + r * 128 : stage + (r * p.x_width + cc * 32) * 2;
        const int turn = boxed ? r & 7 : 0, first = boxed ? (cc & 1) * 4 : 0;
        if (r < rows) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < pieces) *reinterpret_cast<uint4*>(dst + ((first + k) ^ turn) * 16) = make_uint4(pw[4 * k], pw[4 * k + 1], pw[4 * k + 2], pw[4 * k + 3]);
        }
      }
      fence_proxy_async();
    };
    // lane = column of dU here: neighbouring lanes swap, so that each writes two columns of every second row
    auto epilogue_du = [&](int item_q, int item_rows) {
      if (p.which == 2) return;
      T* const out = reinterpret_cast<T*>(p.du) + (long long)item_q * p.H * kKv + ((half * 128 + r) & ~1);
      const bool odd = (lane & 1) != 0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (c * 32 >= item_rows) break;
        uint32_t t[32];
        tmem_ld32(lane_base + kDuCol + half * kRows + c * 32, t);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = __uint_as_float(t[2 * i]), b = __uint_as_float(t[2 * i + 1]);
          const float recv = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
          const int row = c * 32 + 2 * i + (odd ? 1 : 0);
          if (row < item_rows)
            *reinterpret_cast<uint32_t*>(out + (long long)row * kKv) =
                odd ? pack2_out<T>(recv * p.scale, b * p.scale) : pack2_out<T>(a * p.scale, recv * p.scale);
        }
      }
    };

    for (uint32_t n = 0; alive; ++n) {
      WorkItem w;
      if (wq_consume_item(sm.wq, n, w, abort_flag) < 0) break;
      const int rows = w.o_rows * p.H;
      const int nt = (w.i_len + kTile - 1) / kTile;
      if (nt == 0) continue;
      if (threadIdx.x < kRows) {
        const int t = threadIdx.x;
        const long long at = (long long)w.o_start * p.H + t;
        sm.nl[par][t] = t < rows ? p.nl[at] : -INFINITY;
        sm.nd[par][t] = t < rows ? -p.ld[at].y : 0.f;
        sm.nds[par][t] = t < rows ? p.nds[at] : 0.f;
        mbar_arrive(smem_u32(&sm.nl_full));
      }
      if (!mbar_wait(smem_u32(&sm.nl_full), par, abort_flag)) break;
      const bool active = half * 32 < rows;

      for (int t = 0; t < nt; ++t) {
        const uint32_t g = gk + t;
        const int keys = min(kTile, w.i_len - t * kTile);
        { TRACE_T0(); if (!mbar_wait(smem_u32(&sm.sy_full), g & 1, abort_flag)) { alive = false; break; } TRACE_ADD(8); }
        tc_fence_after();
#ifdef VAFA_TRACE
        tr[11] += 1;
        long long t_c = clock64();
#endif
        uint32_t pd[32], dd[16];  // w P and w dS', dS
        uint32_t xs[32], ys[32];
        if (active) {
          tmem_ld32(lane_base + kSCol + half * 32, xs);
          tmem_ld32(lane_base + kYCol + half * 32, ys);
          tmem_wait_ld();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.s_free));
        if (active) {
          const float2* nlp = reinterpret_cast<const float2*>(&sm.nl[par][half * 32]);
          const float2* ndp = reinterpret_cast<const float2*>(&sm.nd[par][half * 32]);
          const float2* ndsp = reinterpret_cast<const float2*>(&sm.nds[par][half * 32]);
          const bool row_ok = r < keys;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 n2 = nlp[i], d2 = ndp[i], ds2 = ndsp[i];
            const uint64_t y2 = pack_f2(__uint_as_float(ys[2 * i]), __uint_as_float(ys[2 * i + 1]));
            float t0, t1, w0, w1, e0, e1, f0, f1;
            unpack_f2(fma_f2(pack_f2(__uint_as_float(xs[2 * i]), __uint_as_float(xs[2 * i + 1])), c2, pack_f2(n2.x, n2.y)), t0, t1);
            const uint64_t p2 = pack_f2(ex2(t0), ex2(t1)), wp2 = mul_f2(p2, w2);
            unpack_f2(wp2, w0, w1);
            unpack_f2(mul_f2(wp2, fma_f2(y2, s2, pack_f2(ds2.x, ds2.y))), e0, e1);
            unpack_f2(mul_f2(p2, add_f2(y2, pack_f2(d2.x, d2.y))), f0, f1);
            pd[i] = row_ok ? pack2_out<T>(w0, w1) : 0u;
            pd[16 + i] = row_ok ? pack2_out<T>(e0, e1) : 0u;
            dd[i] = row_ok ? pack2_out<T>(f0, f1) : 0u;
          }
        }
#ifdef VAFA_TRACE
        tr[12] += clock64() - t_c;
#endif
        if (active) {
          tmem_st32(lane_base + kYCol + half * 32, pd);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t off = r * 128 + (((half * 4 + j) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(sm.ds + off) = make_uint4(dd[4 * j], dd[4 * j + 1], dd[4 * j + 2], dd[4 * j + 3]);
          }
          tmem_wait_st();
          fence_proxy_async();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.pds_full));
        // the tile's products: they have read P, dS' and dS and, with dU^T, the X tile
        { TRACE_T0(); if (!mbar_wait(smem_u32(&sm.dx_done), g & 1, abort_flag)) { alive = false; break; } TRACE_ADD(9); }
        tc_fence_after();
        {
          TRACE_T0();
          epilogue_dx(sm.x[g & 1], keys);
          TRACE_ADD(14);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.stage_full[g & 1]));
      }
      if (!alive) break;
      epilogue_du(w.o_start, rows);
      // (both accumulators are written again only after this thread's next arrival at pds_full)
      tc_fence_before();
      gk += nt;
      par ^= 1;
    }
  }

#ifdef VAFA_TRACE
  if (p.trace != nullptr && (threadIdx.x == 0 || threadIdx.x == 256 || threadIdx.x == 288)) {
    tr[15] = clock64() - t_begin;
    for (int i = 0; i < 16; ++i)
      if (tr[i] != 0) p.trace[(long long)blockIdx.x * 16 + i] = tr[i];
  }
#endif
  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (sm.abort_flag != 0) {
    if (threadIdx.x == 0) report_error(p.status, 1, 151, blockIdx.x);
    // let copies that are still in flight land before shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) { }
    __syncthreads();
  }
  if (warp == 9) tmem_dealloc(tbase, 512);
}

#ifdef VAFA_TRACE
}  // namespace
long long* vafa_trace_buffer_dxu = nullptr;
namespace {
#endif

// The smallest power of two at or above the scale, upside down, between 1 and 2^8.  From a scale of 1 on dS' is no smaller than dS.
// Below, w dS' lies between dS / 2 and dS, so that it leaves the range of fp16 on either side no sooner than dS in dU does; w P
// ends at 2^8.
float range_factor(float scale) {
  int e;
  const float f = frexpf(scale, &e);
  if (f == 0.5f) --e;
  return ldexpf(1.f, e >= 0 ? 0 : e <= -8 ? 8 : -e);
}

template <typename T>
int launch_dxu(const AbsorbDxuLaunch& L, cudaStream_t s) {
  CUtensorMap tu, tg, tx, tdx;
  int rc;
  if ((rc = encode_tmap_rows(&tu, L.u, L.dtype, L.total_q, L.H, kKv, kRows / L.H, L.H))) return rc;
  if ((rc = encode_tmap_rows(&tg, L.dax, L.dtype, L.total_q, L.H, kKv, kRows / L.H, L.H))) return rc;
  if ((rc = encode_tmap_rows(&tx, L.x, L.dtype, L.total_k, 1, L.x_width, kTile))) return rc;
  if ((rc = encode_tmap_rows(&tdx, L.dx, L.dtype, L.total_k, 1, L.x_width, kTile))) return rc;
  DxuParams p;
  p.du = L.du; p.dx = L.dx; p.ld = L.ld; p.nl = L.nl; p.nds = L.nds;
  p.header = (const SchedHeader*)L.header; p.items = (const WorkItem*)L.items;
  p.H = L.H; p.x_width = L.x_width; p.which = L.which;
  p.scale = L.scale; p.scale_log2 = L.scale * kLog2e; p.range = range_factor(L.scale); p.inv_range = 1.f / p.range;
  p.status = L.status;
  p.wait_limit = wait_limit_units();
  p.trace = nullptr;
#ifdef VAFA_TRACE
  {
    static long long* g_trace = nullptr;  // debugging aid only
    if (!g_trace) cudaMalloc(&g_trace, 512 * 16 * sizeof(long long));
    cudaMemsetAsync(g_trace, 0, 512 * 16 * sizeof(long long), s);
    p.trace = g_trace;
    vafa_trace_buffer_dxu = g_trace;
  }
#endif
  const size_t smem = sizeof(DxuSmem) + 1024;
  VAFA_CUDA_CHECK(cudaFuncSetAttribute(absorb_dxu_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LaunchScope scope(kKAbsorbBwdDxu, s);
  absorb_dxu_kernel<T><<<L.sms, kDxuThreads, smem, s>>>(tu, tg, tx, tdx, p);
  VAFA_LAUNCH_CHECK("absorb_dxu_kernel");
  return 0;
}

}  // namespace

int sm100_absorb_dxu_launch(const AbsorbDxuLaunch& L, cudaStream_t s) {
  return L.dtype == VAFA_BF16 ? launch_dxu<__nv_bfloat16>(L, s) : launch_dxu<__half>(L, s);
}

}  // namespace vafa

#ifdef VAFA_TRACE
extern "C" __attribute__((visibility("default"))) int vafa_trace_read_dxu(long long* host, int n) {
  if (!vafa::vafa_trace_buffer_dxu) return -1;
  return (int)cudaMemcpy(host, vafa::vafa_trace_buffer_dxu, (size_t)n * 16 * sizeof(long long), cudaMemcpyDeviceToHost);
}
#endif

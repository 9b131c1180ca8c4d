// Dense product for the absorb operator's prologue and epilogue:
//   C[M, N] = A[M, K] . B[K, N]        (16-bit operands, fp32 accumulation, 16-bit result; K = 256 k)
// One persistent CTA per SM owns a 256-column slice of C and walks 128-row tiles of it.  K is taken 64 deep: a chunk of A
// (16 KB) has a slot of its own, so the loads of the next tile start while the current one is multiplied.  K = 256: the
// CTA's 256 x 256 slice of B stays in shared memory (128 KB, MN-major) beside five slots; K = 512, 768, ...: a slot holds the
// chunk of B (32 KB) too, and there are four.  The accumulator (256 TMEM columns) is double buffered, so the epilogue
// of tile i overlaps the products of tile i + 1; a row's pieces leave through the lane transpose of common.cuh.
// Bound by L2 and HBM (a row of the stacked operands is 4 KB).  With one 64 KB tile of A at a time its load, its products and the
// next load ran one after the other: the six products of a training step of 1024 users 113 -> 90 us, at raw widths 968 / 216
// 134 -> 99.
// It stands in for the two torch matmuls of the reference's prologue
// (triton_target_attn_absorb/triton_target_attn_absorb/interface.py:434-435, here as one product
// with the pre-multiplied W_Q W_K^T) and for the per-head W_V projection the reference does at the
// end of its forward kernel (triton_target_attn_absorb/triton_target_attn_absorb/kernels.py:273-279).
#include <cuda.h>
#include <type_traits>

#include "profile.cuh"
#include "sm100_common.cuh"
#include "sm100_kernels.cuh"

namespace vafa {
namespace {

using namespace ptx;

constexpr int kGemmThreads = 192;
constexpr int kK = 256;
constexpr int kNTile = 256;
constexpr int kChunk = 64;                       // depth of a slot
constexpr int kAChunk = 128 * 128;               // 128 rows x 64 of A
constexpr int kBSub = kChunk * 128;              // 64 k-rows x 64 columns of B
constexpr int kBChunk = 4 * kBSub;
constexpr int kResidentSlots = 5, kStreamSlots = 4, kMaxSlots = 5;
constexpr int kBufBytes = 4 * kBChunk + kResidentSlots * kAChunk;
static_assert(kStreamSlots * (kAChunk + kBChunk) <= kBufBytes, "streamed slots fit where the resident slice and its slots do");

struct GemmSmem {
  alignas(1024) uint8_t buf[kBufBytes];  // resident: B slice, then A slots; streamed: slots of A chunk and B chunk
  alignas(8) uint64_t b_full[4], full[kMaxSlots], empty[kMaxSlots], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int wait_limit;  // read by the bounded waits as abort_flag[1]: keep it right behind abort_flag
};
static_assert(sizeof(GemmSmem) + 1024 <= 227 * 1024, "shared memory budget");

struct GemmParams {
  void* C;
  long long M;
  int ldc;
  int n_tiles;     // N / 256
  int m_tiles;     // ceil(M / 128)
  int k_chunks;    // K / 64, or those of a column tile's block
  int k_block;     // rows of B between the blocks of neighbouring column tiles, 0: B is full
  int diag_heads;  // 0: full rows
  int wait_limit;  // bound of every device-side wait, in units of 65536 cycles
};

template <typename T, bool kResident>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_nn_k256_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
  constexpr uint32_t kSlots = kResident ? kResidentSlots : kStreamSlots;
  constexpr uint32_t kFirst = kResident ? 4 * kBChunk : 0, kSlot = kResident ? kAChunk : kAChunk + kBChunk;
  extern __shared__ uint8_t smem_raw[];
  GemmSmem& sm = *reinterpret_cast<GemmSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = (int)warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  volatile int* abort_flag = &sm.abort_flag;
  if (threadIdx.x == 0) {
    sm.abort_flag = 0;
    sm.wait_limit = p.wait_limit;
    for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&sm.b_full[i]), 1);
    for (int i = 0; i < kMaxSlots; ++i) {
      mbar_init(smem_u32(&sm.full[i]), 1);
      mbar_init(smem_u32(&sm.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sm.acc_full[i]), 1);
      mbar_init(smem_u32(&sm.acc_empty[i]), 128);
    }
    fence_barrier_init();
  }
  if (warp == 4 && lane == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sm.tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = sm.tmem_base;

  // CTA -> (column tile, first row tile, row tile stride)
  const int groups = gridDim.x / p.n_tiles;  // CTAs per column tile (grid is a multiple of n_tiles)
  const int n_tile = blockIdx.x % p.n_tiles;
  const int m_first = blockIdx.x / p.n_tiles;
  const int kc0 = n_tile * p.k_block / kChunk;
  const uint32_t buf0 = smem_u32(sm.buf);

  if (warp == 4) {
    if (lane == 0) {
      auto load_b = [&](uint32_t dst, uint32_t bar, int kc) {
        for (int c = 0; c < 4; ++c) tma_load_3d(dst + c * kBSub, &tmap_b, bar, n_tile * kNTile + c * 64, 0, (kc0 + kc) * kChunk);
      };
      uint32_t it = 0;
      bool alive = true;
      for (int m = m_first; alive && m < p.m_tiles; m += groups) {
        for (int kc = 0; kc < p.k_chunks; ++kc, ++it) {
          const uint32_t slot = it % kSlots, bar = smem_u32(&sm.full[0]) + slot * 8, dst = buf0 + kFirst + slot * kSlot;
          if (!mbar_wait(smem_u32(&sm.empty[0]) + slot * 8, ((it / kSlots) & 1) ^ 1, abort_flag)) { alive = false; break; }
          mbar_expect_tx(bar, kSlot);
          tma_load_3d(dst, &tmap_a, bar, (kc0 + kc) * kChunk, 0, m * 128);
          if (!kResident) load_b(dst + kAChunk, bar, kc);
          if (kResident && m == m_first) {
            const uint32_t b_bar = smem_u32(&sm.b_full[kc]);
            mbar_expect_tx(b_bar, kBChunk);
            load_b(buf0 + kc * kBChunk, b_bar, kc);
          }
        }
      }
    }
  } else if (warp == 5) {
    // the whole warp on warp-uniform values, one elected lane issues (see varlen_fwd_kernel)
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t idesc = make_idesc(kFmt, 0, 1, 128, kNTile);
    const uint32_t tm = warp_uniform(tbase);
    const uint32_t a_lo0 = warp_uniform(desc_lo_sw128(buf0 + kFirst, 16));
    const uint32_t b_lo0 = warp_uniform(desc_lo_sw128(buf0 + (kResident ? 0 : kAChunk), kBSub));
    bool ok = true;
    uint32_t it = 0, tile = 0;
    for (int m = m_first; ok && m < p.m_tiles; m += groups, ++tile) {
      const uint32_t buf = tile & 1;
      if (!mbar_wait_warp(smem_u32(&sm.acc_empty[0]) + buf * 8, ((tile >> 1) & 1) ^ 1, abort_flag)) break;
      for (int kc = 0; kc < p.k_chunks; ++kc, ++it) {
        const uint32_t slot = it % kSlots;
        if (kResident && tile == 0 && !mbar_wait_warp(smem_u32(&sm.b_full[0]) + kc * 8, 0, abort_flag)) { ok = false; break; }
        if (!mbar_wait_warp(smem_u32(&sm.full[0]) + slot * 8, (it / kSlots) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_lo = a_lo0 + slot * (kSlot >> 4), b_lo = b_lo0 + (kResident ? (uint32_t)kc * (kBChunk >> 4) : slot * (kSlot >> 4));
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kChunk / 16; ++kk)
            mma_ss2(tm + buf * kNTile, a_lo + kk * 2, b_lo + kk * (2048 >> 4), idesc, (kc > 0 || kk > 0) ? 1u : 0u);
          mma_commit(smem_u32(&sm.empty[0]) + slot * 8);
          if (kc == p.k_chunks - 1) mma_commit(smem_u32(&sm.acc_full[0]) + buf * 8);
        }
        __syncwarp();
      }
    }
  } else {
    const int r = threadIdx.x;
    const uint32_t lane_base = tbase + ((uint32_t)(warp * 32) << 16);
    T* const C = reinterpret_cast<T*>(p.C);
    uint32_t it = 0;
    for (int m = m_first; m < p.m_tiles; m += groups, ++it) {
      const uint32_t buf = it & 1;
      if (!mbar_wait(smem_u32(&sm.acc_full[buf]), (it >> 1) & 1, abort_flag)) break;
      tc_fence_after();
      const long long row = (long long)m * 128 + r;
      const int rows = (int)min(128LL, p.M - (long long)m * 128);
      auto ld = [&](int cc, uint32_t (&pw)[16]) {
        uint32_t t[32];
        tmem_ld32(lane_base + buf * kNTile + cc * 32, t);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) pw[i] = pack2_out<T>(__uint_as_float(t[2 * i]), __uint_as_float(t[2 * i + 1]));
      };
      if (p.diag_heads == 0) {
#pragma unroll 2
        for (int cc = 0; cc < kNTile / 32; ++cc) {
          uint32_t pw[16];
          ld(cc, pw);
          store_chunk_coalesced<T>(pw, C + row * p.ldc + (long long)n_tile * kNTile + cc * 32, p.ldc, r, rows, 4);
        }
      } else {
        // row m keeps the 256 / diag_heads columns of its own head.  tcgen05.ld is warp-collective: all chunks are walked
        // and each lane keeps its own, so that a chunk of all rows leaves in one go
        const int per = (kNTile / p.diag_heads) / 32;  // 32-column chunks per head
        const int mine = (int)(row % p.diag_heads);
        for (int j = 0; j < per; ++j) {
          uint32_t keep[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) keep[i] = 0u;
          for (int h = 0; h < p.diag_heads; ++h) {
            if (!__any_sync(0xffffffffu, mine == h)) continue;
            uint32_t pw[16];
            ld(h * per + j, pw);
#pragma unroll
            for (int i = 0; i < 16; ++i) keep[i] = mine == h ? pw[i] : keep[i];
          }
          store_chunk_coalesced<T>(keep, C + row * p.ldc + j * 32, p.ldc, r, rows, 4);
        }
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&sm.acc_empty[buf]));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (sm.abort_flag != 0) {
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) { }
    __syncthreads();
  }
  if (warp == 5) tmem_dealloc(tbase, 512);
}

template <typename T, bool kResident>
int launch_gemm_nn(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid, cudaStream_t s) {
  const size_t smem = sizeof(GemmSmem) + 1024;
  VAFA_CUDA_CHECK(cudaFuncSetAttribute(gemm_nn_k256_kernel<T, kResident>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gemm_nn_k256_kernel<T, kResident><<<grid, kGemmThreads, smem, s>>>(ta, tb, p);
  VAFA_LAUNCH_CHECK("gemm_nn_k256_kernel");
  return 0;
}

}  // namespace

int sm100_gemm_nn_k256(const GemmNNArgs& g, cudaStream_t s) {
  if (g.M <= 0) return 0;
  if (g.N % kNTile != 0 || (g.diag_heads > 0 && (g.N != kNTile || (kNTile / g.diag_heads) % 32 != 0)))
    return fail(VAFA_ERR_UNSUPPORTED, "gemm_nn_k256: N=%d diag_heads=%d not supported", g.N, g.diag_heads);
  if (g.k_block > 0 && (g.lda != kK || (g.N / kNTile) * g.k_block != kK || (kChunk % g.k_block != 0 && g.k_block % kChunk != 0)))
    return fail(VAFA_ERR_UNSUPPORTED, "gemm_nn_k256: blocks of %d rows not supported", g.k_block);
  int sms = g.sm_count;
  if (sms <= 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  GemmParams p;
  p.wait_limit = wait_limit_units();
  p.C = g.C; p.M = g.M; p.ldc = g.ldc; p.n_tiles = g.N / kNTile; p.m_tiles = (int)((g.M + 127) / 128);
  p.diag_heads = g.diag_heads;
  p.k_block = g.k_block;
  p.k_chunks = g.k_block > 0 ? (g.k_block + kChunk - 1) / kChunk : g.lda / kChunk;
  int groups = sms / p.n_tiles;
  if (groups < 1) groups = 1;
  if (groups > p.m_tiles) groups = p.m_tiles;
  const int grid = groups * p.n_tiles;
  CUtensorMap ta, tb;
  int rc;
  // K = lda (A rows densely packed), a multiple of 256; B is [K, N] densely packed
  if (g.lda < kK || g.lda % kK != 0 || g.ldb != g.N) return fail(VAFA_ERR_UNSUPPORTED, "gemm_nn_k256: K=%d ldb=%d not supported", g.lda, g.ldb);
  if ((rc = encode_tmap_rows(&ta, g.A, g.dtype, g.M, 1, g.lda, 128))) return rc;
  if ((rc = encode_tmap_rows(&tb, g.B, g.dtype, g.lda, 1, g.N, kChunk))) return rc;
  LaunchScope scope(kKAbsorbGemm, s);
  const bool resident = g.lda == kK;
  if (g.dtype == VAFA_BF16)
    return resident ? launch_gemm_nn<__nv_bfloat16, true>(ta, tb, p, grid, s) : launch_gemm_nn<__nv_bfloat16, false>(ta, tb, p, grid, s);
  return resident ? launch_gemm_nn<__half, true>(ta, tb, p, grid, s) : launch_gemm_nn<__half, false>(ta, tb, p, grid, s);
}

}  // namespace vafa

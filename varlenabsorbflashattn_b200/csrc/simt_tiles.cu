// Tiled fp32-arithmetic attention (simt_tiles.cuh): which calls it takes, and the forward.
#include "simt_tiles.cuh"

namespace vafa {

using namespace tiles;

bool simt_tiles_ok(const SimtAttnParams& a) {
  if (a.D > 256 || a.total_q <= 0 || a.total_k <= 0) return false;
  if (a.shared_kv && (a.q_row != a.H * a.q_head || a.do_row != a.H * a.do_head || a.causal || !a.do_f32)) return false;
  if (!a.shared_kv && a.do_f32) return false;
  const int stack = a.shared_kv ? a.H : 1;
  const long long rows = (long long)a.total_q * stack;
  if (rows < (long long)kTileMinRows * a.n_seg || a.total_k < (long long)kTileMinRows * a.n_seg) return false;
  if ((double)rows * a.total_k < kTileMinScores * a.n_seg * a.n_seg) return false;
  const long long heads = a.shared_kv ? 1 : a.H;
  return max_slots(a.total_q, stack, a.n_seg) * heads < (1LL << 31) / kMaxSplits &&
         max_slots(a.total_k, 1, a.n_seg) * heads < (1LL << 31) / kMaxSplits;
}

int simt_tiles_fwd(const SimtAttnParams& a, cudaStream_t s) {
  TileParams p = tile_params(a);
  p.vec_o = vec4(a.o, p.q_row, p.q_head, a.D, elem_size(a.dtype));
  p.slots = max_slots(a.total_q, p.stack, a.n_seg);
  p.splits = pick_splits(p.slots * p.heads, a.total_k, a.n_seg);
  return by_type(a.dtype, [&](auto tag) {
    using T = decltype(tag);
    return by_dim(a.D, [&](auto d) {
      constexpr int DP = decltype(d)::value;
      return a.shared_kv ? launch(tile_fwd_kernel<T, DP, true>, fwd_smem<DP, true>(), p, "tile_fwd_kernel", s)
                         : launch(tile_fwd_kernel<T, DP, false>, fwd_smem<DP, false>(), p, "tile_fwd_kernel", s);
    });
  });
}

}  // namespace vafa

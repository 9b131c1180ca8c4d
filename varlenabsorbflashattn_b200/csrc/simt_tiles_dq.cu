// Tiled fp32-arithmetic attention (simt_tiles.cuh): dQ.
#include "simt_tiles.cuh"

namespace vafa {

using namespace tiles;

int simt_tiles_dq(const SimtAttnParams& a, cudaStream_t s) {
  TileParams p = tile_params(a);
  p.vec_o = vec4(a.dq, p.q_row, p.q_head, a.D, elem_size(a.dtype));
  p.slots = max_slots(a.total_q, p.stack, a.n_seg);
  p.splits = pick_splits(p.slots * p.heads, a.total_k, a.n_seg);
  return by_type(a.dtype, [&](auto tag) {
    using T = decltype(tag);
    return by_dim(a.D, [&](auto d) {
      constexpr int DP = decltype(d)::value;
      return a.shared_kv ? launch(tile_dq_kernel<T, float, DP, true>, dq_smem<DP, true>(), p, "tile_dq_kernel", s)
                         : launch(tile_dq_kernel<T, T, DP, false>, dq_smem<DP, false>(), p, "tile_dq_kernel", s);
    });
  });
}

}  // namespace vafa

// Tiled fp32-arithmetic attention (simt_tiles.cuh): dK and dV, or their sum over the heads.
#include "simt_tiles.cuh"

namespace vafa {

using namespace tiles;

int simt_tiles_dkv(const SimtAttnParams& a, cudaStream_t s) {
  TileParams p = tile_params(a);
  p.vec_o = vec4(a.dk, p.k_row, p.k_head, a.D, elem_size(a.dtype)) && (a.shared_kv || vec4(a.dv, p.v_row, p.v_head, a.D, elem_size(a.dtype)));
  p.slots = max_slots(a.total_k, 1, a.n_seg);
  p.splits = pick_splits(p.slots * p.heads, (long long)a.total_q * p.stack, a.n_seg);
  return by_type(a.dtype, [&](auto tag) {
    using T = decltype(tag);
    return by_dim(a.D, [&](auto d) {
      constexpr int DP = decltype(d)::value;
      return a.shared_kv ? launch(tile_dkv_kernel<T, float, DP, true>, dkv_smem<DP, true>(), p, "tile_dkv_kernel", s)
                         : launch(tile_dkv_kernel<T, T, DP, false>, dkv_smem<DP, false>(), p, "tile_dkv_kernel", s);
    });
  });
}

}  // namespace vafa

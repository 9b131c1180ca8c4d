"""Dispatch branches of the tile kernels at the sizes where they can go wrong: stacks of heads that do and do not
divide a 128-row tile, segments around the tile's query count, rows of padding in whole warps, slices of a
lone long segment."""
import pytest
import torch

import varlenabsorbflashattn_b200 as vb
from oracle import make_absorb_inputs, make_varlen_inputs, target_attn_ref_fwd_bwd, varlen_attn_ref
from helpers import LN2, check_close, check_lse

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,H_kv,D,dtype,causal", [
    (8, 2, 128, torch.bfloat16, False), (12, 4, 128, torch.bfloat16, True), (10, 2, 64, torch.float16, True),
    (16, 1, 128, torch.float16, False), (7, 1, 64, torch.bfloat16, False), (128, 1, 64, torch.bfloat16, True),
    (4, 4, 128, torch.bfloat16, False)])
def test_few_queries_per_segment(H, H_kv, D, dtype, causal):
    """Fewer than 128 queries per segment on average: the query heads of a K/V head share a tile."""
    G = H // H_kv
    t = 128 // G  # queries per tile
    ql = [1, t, t + 1, 0, max(1, t - 1), 3, 2 * t + 1, 1, 9, 2]
    kl = [1, 200, t + 1, 7, 127, 129, 2 * t + 1, 5000, 0, 33]
    if causal:
        kl = [max(a, b) for a, b in zip(ql, kl)]
    q, _, _, _, cu_q, cu_k = make_varlen_inputs(ql, kl, H, D, dtype, 11, with_do=False)
    g = torch.Generator().manual_seed(12)
    k, v = (torch.randn(sum(kl), H_kv, D, generator=g).to(dtype) for _ in range(2))
    with torch.no_grad():
        o, lse = vb.packed_varlen_attn_with_lse(q.to(DEV), k.to(DEV), v.to(DEV), cu_seqlens_q=cu_q, cu_seqlens_k=cu_k,
                                                causal=causal)
    ro, rlse = varlen_attn_ref(q, k.repeat_interleave(G, dim=1), v.repeat_interleave(G, dim=1), cu_q, cu_k, causal=causal)
    check_close("o", o, ro, dtype)
    check_lse(lse / LN2, rlse)


@pytest.mark.parametrize("ql,kl,H", [
    ([1] * 80, [300] * 79 + [30000], 8),         # many tiles, one of them longer than an SM's share
    ([130, 1, 500], [20000, 9000, 40000], 2),    # full tiles and a single row cut side by side
    ([1, 2], [257, 129], 1)])                    # slices of two blocks
def test_long_segments_are_cut(ql, kl, H):
    q, k, v, _, cu_q, cu_k = make_varlen_inputs(ql, kl, H, 64, torch.bfloat16, 13, with_do=False)
    with torch.no_grad():
        o, lse = vb.packed_varlen_attn_with_lse(q.to(DEV), k.to(DEV), v.to(DEV), cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)
    ro, rlse = varlen_attn_ref(q, k, v, cu_q, cu_k)
    check_close("o", o, ro, torch.bfloat16)
    check_lse(lse / LN2, rlse)


@pytest.mark.parametrize("ql,kl,H", [
    ([16], [5000], 8),                                      # one user, one full tile
    ([1, 16, 17, 0, 3], [700, 2048, 2047, 5, 0], 8),        # cut and uncut tiles, a second tile of one query
    ([5, 40], [3000, 97], 4), ([3] * 24, [8] * 23 + [2048], 8)])
def test_few_users_with_long_histories_are_cut(ql, kl, H):
    """Absorb: up to four tiles per SM the histories are cut and the parts merged (also read by the backward)."""
    ql = [a if b else 0 for a, b in zip(ql, kl)]
    ins = make_absorb_inputs(ql, kl, 256, 256, H, 256 // H, torch.bfloat16, 14, x_std=0.3, w_std=0.1)
    q_raw, X, W_Q, W_K, W_V, dO, cu_q, cu_k = ins
    g = [t.to(DEV).requires_grad_(True) for t in (q_raw, X, W_Q, W_K, W_V)]
    O = vb.packed_target_attn(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)
    O.backward(dO.to(DEV))
    ref = target_attn_ref_fwd_bwd(*ins)
    check_close("O", O, ref[0], torch.bfloat16, scale_abs=True)
    for name, t, r in zip(("dq_raw", "dX", "dW_Q", "dW_K", "dW_V"), g, ref[2:]):
        check_close(name, t.grad, r, torch.bfloat16, scale_abs=True)

"""Dispatch branches of the tile kernels at the sizes where they can go wrong: stacks of heads that do and do not
divide a 128-row tile, segments around the tile's query count, rows of padding in whole warps, slices of a
lone long segment."""
import math

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
    ([1, 16, 17, 0, 3], [700, 2048, 2047, 5, 0], 8),        # a second tile of one query
    ([5, 40], [3000, 97], 4), ([3] * 24, [8] * 23 + [2048], 8)])
def test_few_users_with_long_histories(ql, kl, H):
    """Absorb: fewer tiles than SMs, histories of many blocks and of one, a tile of one query."""
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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("n_seg,H,climb", [(3, 2, 12.0), (3, 2, 130.0), (160, 8, 130.0)])
def test_scores_that_climb_past_the_first_block(dtype, D, n_seg, H, climb):
    """Scores of later blocks far above those of the first one (by `climb` log2 units and more, in steps): tiles whose
    reference maximum is left are done again; with many of them a CTA stops trying."""
    L = 700
    q, k, v, _, cu_q, cu_k = make_varlen_inputs([L] * n_seg, [L] * n_seg, H, D, dtype, 21, with_do=False)
    # a common direction: q[..., 0] = 1, and k[..., 0] steps up every 128 keys in every other segment
    q[..., 0] = 1.0
    step = torch.arange(L).div(128, rounding_mode="floor").float() * climb * math.log(2.0) * math.sqrt(D) / 4
    for s in range(0, n_seg, 2):
        k[s * L:(s + 1) * L, :, 0] = step[:, None].to(dtype)
    with torch.no_grad():
        o, lse = vb.packed_varlen_attn_with_lse(q.to(DEV), k.to(DEV), v.to(DEV), cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, causal=True)
    n = min(n_seg, 4) * L
    ro, rlse = varlen_attn_ref(q[:n], k[:n], v[:n], cu_q[:min(n_seg, 4) + 1], cu_k[:min(n_seg, 4) + 1], causal=True)
    check_close("o", o[:n], ro, dtype)
    # each of the D / 16 accumulation steps of a score can lose a unit in the last place of the running fp32 sum, and the
    # exponent, the logarithm and the conversion of the LSE one more each: scores reach 110 here
    assert ((lse[:n].cpu() - rlse).abs() <= 1e-4 + (D // 16 + 4) * 2.0 ** -23 * rlse.abs()).all()
    assert torch.isfinite(o).all()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nan_and_infinite_scores_behind_the_first_block(bad):
    """Only the rows that see the bad key are touched by it."""
    L, H, D = 400, 2, 64
    q, k, v, _, cu_q, cu_k = make_varlen_inputs([L, L], [L, L], H, D, torch.bfloat16, 22, with_do=False)

    def run(kk):
        with torch.no_grad():
            return vb.packed_varlen_attn(q.to(DEV), kk.to(DEV), v.to(DEV), cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, causal=True)

    o0 = run(k)
    k2 = k.clone()
    k2[300] = bad
    o1 = run(k2)
    # (with an infinite score the rest of the tile is done again: equal at least up to the rounding of P and O, 2^-8 each)
    assert (o1[:300] - o0[:300]).abs().max() <= 2e-2 and torch.equal(o1[L:], o0[L:])
    assert torch.isnan(o1[300:L].float()).any(dim=-1).all()

"""The tiled fp32-arithmetic attention kernels at the edges of their 64-row tiles, their inner blocks and their
cluster splits, for every padded head dim and for rows that cannot be read four elements at a time."""
import pytest
import torch

import varlenabsorbflashattn_b200 as vb
from oracle import make_absorb_inputs, make_varlen_inputs, target_attn_ref_fwd_bwd, varlen_attn_ref_fwd_bwd
from helpers import LN2, check_close, check_lse

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("ql,kl", [
    ([64, 65, 63, 1, 0, 129], [64, 63, 65, 33, 7, 0]),
    ([100, 8, 31], [1000, 513, 32]),           # several ranks of a cluster per tile
    ([300], [20]),                             # more queries than keys: causal rows without a key
    ([8] * 40, [31] * 40), ([8] * 40, [32] * 40), ([16] * 9, [15] * 9), ([16] * 9, [16] * 9),  # either side of the line
    ([20] * 3, [127] * 3), ([20] * 3, [128] * 3), ([20] * 3, [320] * 3)])  # one rank, two, eight
def test_varlen_fp32(D, causal, ql, kl):
    q, k, v, do, cu_q, cu_k = make_varlen_inputs(ql, kl, 3, D, torch.float32, 5)
    g = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    o, lse = vb.packed_varlen_attn_with_lse(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, causal=causal)
    o.backward(do.to(DEV))
    ref = varlen_attn_ref_fwd_bwd(q, k, v, do, cu_q, cu_k, causal=causal)
    check_close("o", o, ref[0], torch.float32)
    check_lse(lse / LN2, ref[1])
    for name, t, r in zip(("dq", "dk", "dv"), g, ref[2:]):
        check_close(name, t.grad, r, torch.float32, scale_abs=True)


@pytest.mark.parametrize("d_kv,H,dtype", [(256, 8, torch.float32), (216, 8, torch.float32), (130, 4, torch.float32),
                                          (37, 3, torch.float32), (64, 6, torch.bfloat16)])
def test_absorb_shared_rows(d_kv, H, dtype):
    ins = make_absorb_inputs([16, 1, 9, 7, 0, 33], [700, 64, 65, 63, 5, 1], 72, d_kv, H, 32, dtype, 6, x_std=0.1, w_std=0.1)
    q_raw, X, W_Q, W_K, W_V, dO, cu_q, cu_k = ins
    g = [t.to(DEV).requires_grad_(True) for t in (q_raw, X, W_Q, W_K, W_V)]
    O = vb.packed_target_attn(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)
    O.backward(dO.to(DEV))
    ref = target_attn_ref_fwd_bwd(q_raw, X, W_Q, W_K, W_V, dO, cu_q, cu_k)
    check_close("O", O, ref[0], dtype, scale_abs=True)
    for name, t, r in zip(("dq_raw", "dX", "dW_Q", "dW_K", "dW_V"), g, ref[2:]):
        if dtype != torch.float32 and name in ("dq_raw", "dW_Q", "dW_K"):
            # delta = rowsum(dO * O) is formed from the 16-bit O: the score gradient of a user with one key (33 of
            # these 66 rows), exactly zero in truth, is |dO| 2^-9 |O| of noise, so only the absolute error is bounded
            assert (t.grad.float().cpu() - r.float()).abs().max() <= 2e-2 * max(1.0, r.abs().max().item())
            continue
        check_close(name, t.grad, r, dtype, scale_abs=True)


def test_rows_that_are_not_seen_may_hold_anything():
    """Infinities and NaN in keys and values that the causal mask hides, and behind a segment, change nothing."""
    ql = kl = [70, 90]
    q, k, v, do, cu_q, cu_k = make_varlen_inputs(ql, kl, 2, 64, torch.float32, 7)

    def run(kk, vv):
        g = [t.to(DEV).requires_grad_(True) for t in (q, kk, vv)]
        o = vb.packed_varlen_attn(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, causal=True)
        return o.detach(), torch.autograd.grad(o, g, do.to(DEV))[0]

    o0, dq0 = run(k, v)
    k2, v2 = k.clone(), v.clone()
    k2[60:70], v2[60:70] = float("nan"), float("inf")   # keys 60.. of the first segment
    o1, dq1 = run(k2, v2)
    for a, b in ((o0, o1), (dq0, dq1)):
        assert torch.equal(a[:60], b[:60]) and torch.equal(a[70:], b[70:])


@pytest.mark.parametrize("dtype,D", [(torch.float32, 32), (torch.float32, 64), (torch.float32, 256), (torch.bfloat16, 32), (torch.float16, 256)])
@pytest.mark.parametrize("Lk", [40, 900])  # one CTA of a cluster, several
@pytest.mark.parametrize("where", ["q nan", "k nan", "k inf"])
def test_a_visible_nan_or_infinity_does_not_vanish(dtype, D, Lk, where):
    """It reaches the rows that see it in O, LSE and dQ, and no others."""
    H = 2
    q, k, v, do, cu_q, cu_k = make_varlen_inputs([16, 20], [Lk, 30], H, D, dtype, 8)
    if where == "q nan":
        q[5, 1, 3] = float("nan")
        rows = [5]
    else:
        q[..., 3] = 1.0
        k[Lk - 3, 1, 3] = float(where[2:])
        rows = list(range(16))
    g = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    o, lse = vb.packed_varlen_attn_with_lse(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)
    o.backward(do.to(DEV))
    hit = torch.zeros(36, H, dtype=torch.bool, device=DEV)
    hit[rows, 1] = True
    for t in (o, g[0].grad):
        assert torch.isnan(t[hit].float()).all() and torch.isfinite(t[~hit].float()).all()
    assert torch.isnan(lse[hit]).all() and torch.isfinite(lse[~hit]).all()


def test_a_visible_nan_does_not_vanish_absorb():
    ins = make_absorb_inputs([16, 3], [700, 64], 72, 130, 4, 32, torch.float32, 9, x_std=0.1, w_std=0.1)
    q_raw, X, W_Q, W_K, W_V, _, cu_q, cu_k = ins
    X[690, 7] = float("nan")
    with torch.no_grad():
        O = vb.packed_target_attn(*(t.to(DEV) for t in (q_raw, X, W_Q, W_K, W_V)), cu_seqlens_q=cu_q, cu_seqlens_k=cu_k)
    assert torch.isnan(O[:16]).all() and torch.isfinite(O[16:]).all()

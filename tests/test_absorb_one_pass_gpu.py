"""dU and dX of users with at most 64 stacked query rows from one kernel: the edges of its key tiles (128), of the
16-key and 16-row steps of its products, users without keys or queries, and users one query too many beside them."""
import pytest
import torch

import varlenabsorbflashattn_b200 as vb
from oracle import make_absorb_inputs, target_attn_ref_fwd_bwd
from helpers import check_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,dtype,d_kv,scale", [
    (8, torch.bfloat16, 256, None), (8, torch.float16, 216, None), (4, torch.bfloat16, 192, None), (2, torch.float16, 256, None),
    (1, torch.bfloat16, 256, None), (8, torch.bfloat16, 256, 1.0 / 512)])
@pytest.mark.parametrize("long_users", [False, True])
def test_users_of_few_queries(H, dtype, d_kv, scale, long_users):
    t = 64 // H  # queries that fill the 64 rows
    kl = [1, 15, 16, 17, 127, 128, 129, 300, 0, 5, 640, 97, 31]
    ql = [1, t, 2, t, max(1, t - 1), t, 3, t, 0, 0, 1, t, t]
    if long_users:
        ql = [a + t if i % 3 == 1 else a for i, (a, b) in enumerate(zip(ql, kl))]
    ins = make_absorb_inputs(ql, kl, 256, d_kv, H, 256 // H, dtype, 21)
    q_raw, X, W_Q, W_K, W_V, dO, cu_q, cu_k = ins
    g = [x.cuda().requires_grad_(True) for x in (q_raw, X, W_Q, W_K, W_V)]
    out = vb.packed_target_attn(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, scale=scale)
    first = torch.autograd.grad(out, g, dO.cuda(), retain_graph=True)
    ref = target_attn_ref_fwd_bwd(q_raw, X, W_Q, W_K, W_V, dO, cu_q, cu_k, scale=scale)
    check_close("O", out, ref[0], dtype, scale_abs=True)
    for name, mine, r in zip(("dq_raw", "dX", "dW_Q", "dW_K", "dW_V"), first, ref[2:]):
        check_close(name, mine, r, dtype, scale_abs=True)
    second = torch.autograd.grad(out, g, dO.cuda())
    assert all(torch.equal(a, b) for a, b in zip(first, second))  # no order depends on timing


@pytest.mark.parametrize("dtype,eps", [(torch.float16, 2.0 ** -11), (torch.bfloat16, 2.0 ** -8)])
@pytest.mark.parametrize("scale", [1.0 / 256, 32 ** -0.5, 4.0, 16.0, 64.0, 256.0])
def test_what_is_rounded_keeps_its_bits_at_any_scale(dtype, eps, scale):
    """Long, nearly even rows of P.  dX meets three roundings to the type: P, dAlphaX and its own.  One rounding of values whose
    logarithms are spread evenly is 0.7355 / sqrt(3) eps in the 2-norm, the three 0.736 eps; a quarter is added to that."""
    H, n, t, L = 8, 4, 8, 2048
    gen = torch.Generator(device="cuda").manual_seed(11)
    r = lambda std, *s: (torch.randn(s, device="cuda", generator=gen) * std).to(dtype).requires_grad_(True)
    u, X, W_V, dO = r(0.3 / 16 / scale, n * t, H, 256), r(1, n * L, 256), r(1 / 16, 256, H, 32), r(1, n * t, H, 32).detach()
    cu_q, cu_k = (torch.arange(n + 1, device="cuda", dtype=torch.int32) * x for x in (t, L))
    out = vb.target_attn_inner(u, X, W_V, cu_q, cu_k, scale=scale)
    dX = torch.autograd.grad(out, X, dO)[0].double()
    U, x, G = u.detach().double().view(n, t * H, 256), X.detach().double().view(n, L, 256), \
        torch.einsum("thd,khd->thk", dO.double(), W_V.detach().double()).reshape(n, t * H, 256)
    P = torch.softmax(scale * U @ x.mT, -1)
    dP = G @ x.mT
    dS = P * (dP - (P * dP).sum(-1, keepdim=True))
    want = (P.mT @ G + scale * dS.mT @ U).view(n * L, 256)
    assert float((dX - want).norm() / want.norm()) <= 1.25 * 0.736 * eps

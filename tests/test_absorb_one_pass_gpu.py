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
    (1, torch.bfloat16, 256, None), (8, torch.bfloat16, 256, 1.0 / 512)])  # the last scale keeps to the pair of kernels
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

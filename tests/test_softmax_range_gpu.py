"""The forward's softmax against a fixed reference, on scores that leave its range: every further block of an item runs
against the maximum of the first one, so what lies far above it has to be noticed, in whichever column it stands."""
import math
import os
import subprocess
import sys

import pytest
import torch

import varlenabsorbflashattn_b200 as vb

pytestmark = pytest.mark.gpu
DEV = "cuda"
GAPS = (14.0, 59.0, 100.0, 128.6, 150.0, 200.0, 255.0, 300.0, 400.0)  # log2 units above the first block


def _cu(lens):
    return torch.tensor([0] + list(lens), dtype=torch.int64).cumsum(0).int().to(DEV)


def _ref(q, k, v, scale):
    """Every segment with the same lengths, [n, Lq, H, D] x [n, Lk, H, D], in 64 bits."""
    S = torch.einsum("nqhd,nkhd->nhqk", q.double(), k.double()) * scale
    return torch.einsum("nhqk,nkhd->nqhd", S.softmax(-1), v.double()), S.logsumexp(-1).transpose(1, 2)


def _lse_tol(ref, D):
    # each of the D / 16 accumulation steps of a score can lose a unit in the last place of the running fp32 sum, and the
    # exponent, the logarithm and the conversion of the LSE one more each
    return 1e-4 + (D // 16 + 4) * 2.0 ** -23 * ref.abs()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lq", [1, 130])
def test_one_key_far_above_the_first_block(dtype, D, Lq):
    """One key of the second of three blocks stands alone, segment by segment in another column of its block."""
    n, L, H = 128, 384, 2
    g = torch.Generator(device=DEV).manual_seed(31)
    q, k, v = (torch.randn(n, m, H, D, device=DEV, generator=g).to(dtype) for m in (Lq, L, L))
    q[..., 0] = 8.0
    k[..., 0] = 0.0
    at = torch.arange(n, device=DEV)
    for gap in GAPS:
        k[at, 128 + at, :, 0] = gap * math.log(2.0) * math.sqrt(D) / 8.0
        with torch.no_grad():
            o, lse = vb.packed_varlen_attn_with_lse(q.view(-1, H, D), k.view(-1, H, D), v.view(-1, H, D),
                                                    cu_seqlens_q=_cu([Lq] * n), cu_seqlens_k=_cu([L] * n))
        ro, rlse = _ref(q, k, v, D ** -0.5)
        # P and O are rounded to the type, half an eps each
        assert (o.view_as(q).double() - ro).abs().max() <= torch.finfo(dtype).eps * v.abs().max() + 1e-3, gap
        err = (lse.view(n, Lq, H).double() - rlse).abs()
        assert (err <= _lse_tol(rlse, D)).all(), (gap, err.max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_one_key_far_above_the_first_block_absorb(dtype):
    """The same in the absorb kernel's 96-key blocks, whose keys are the values."""
    n, L, H, D_H, d = 96, 288, 8, 32, 256
    g = torch.Generator(device=DEV).manual_seed(32)
    u = (0.3 * torch.randn(n, 2, H, d, device=DEV, generator=g)).to(dtype)
    X = torch.randn(n, L, d, device=DEV, generator=g).to(dtype)
    W_V = (torch.randn(d, H, D_H, device=DEV, generator=g) / 16.0).to(dtype)
    u[..., 0] = 8.0
    X[..., 0] = 0.0
    W_V[0] = 0.0  # the column that raises a key is not seen in its value
    at = torch.arange(n, device=DEV)
    for gap in GAPS:
        X[at, 96 + at, 0] = gap * math.log(2.0) * math.sqrt(D_H) / 8.0
        with torch.no_grad():
            O = vb.target_attn_inner(u.view(-1, H, d), X.view(-1, d), W_V, _cu([2] * n), _cu([L] * n))
        xs = X.unsqueeze(2).expand(n, L, H, d)
        ro = torch.einsum("nqhk,khd->nqhd", _ref(u, xs, xs, D_H ** -0.5)[0], W_V.double())
        assert (O.view_as(ro).double() - ro).abs().max() <= 3e-2, gap  # alphaX is rounded as well


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lq,L", [(3, 128), (3, 384), (200, 384)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_nan_or_infinite_score_reaches_its_rows_from_every_column(dtype, D, Lq, L, bad):
    """Softmax of a row with a NaN or +inf score is NaN; the key stands in another column of the last block of each segment."""
    n, H = 128, 2
    g = torch.Generator(device=DEV).manual_seed(33)
    q, k, v = (torch.randn(n, m, H, D, device=DEV, generator=g).to(dtype) for m in (Lq, L, L))
    q[..., 0] = 1.0
    at = torch.arange(n, device=DEV)
    k[at, L - 128 + at, 0, 0] = bad
    with torch.no_grad():
        o, lse = vb.packed_varlen_attn_with_lse(q.view(-1, H, D), k.view(-1, H, D), v.view(-1, H, D),
                                                cu_seqlens_q=_cu([Lq] * n), cu_seqlens_k=_cu([L] * n))
    o, lse = o.view(n, Lq, H, D), lse.view(n, Lq, H)
    assert torch.isnan(o[:, :, 0]).all() and torch.isnan(lse[:, :, 0]).all()
    assert torch.isfinite(o[:, :, 1]).all() and torch.isfinite(lse[:, :, 1]).all()


def test_the_same_in_the_two_tile_kernel():
    """Segments of more than 160 query rows go there with VAFA_FWD_PAIR=1 (read once per process)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", __file__, "-q", "-x", "-m", "gpu", "-k", "from_every_column and 200",
                        "-p", "no:cacheprovider"], env=dict(os.environ, VAFA_FWD_PAIR="1"), cwd=root, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and "8 passed" in r.stdout, r.stdout[-3000:] + r.stderr[-2000:]


def _climbing(dtype, D, n, L, H, climb, every):
    """Self-attention batch in which every `every`-th segment climbs by `climb` log2 units from block to block."""
    g = torch.Generator(device=DEV).manual_seed(34)
    q, k, v = (torch.randn(n, L, H, D, device=DEV, generator=g).to(dtype) for _ in range(3))
    q[..., 0] = 1.0
    step = torch.arange(L, device=DEV).div(128, rounding_mode="floor").float() * climb * math.log(2.0) * math.sqrt(D)
    k[::every, :, :, 0] = step[:, None].to(dtype)
    return q, k, v


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,climb,every", [(64, 30.0, 2), (128, 30.0, 7), (128, 12.0, 2)])
def test_results_do_not_depend_on_the_rest_of_the_batch(dtype, D, climb, every):
    """Where a few segments leave the range, all come out with the same bits in every run and in a batch of their own."""
    n, L, H = 96, 640, 4
    q, k, v = _climbing(dtype, D, n, L, H, climb, every)

    def run(a, b):
        with torch.no_grad():
            return vb.packed_varlen_attn_with_lse(*(t[a:b].reshape(-1, H, D) for t in (q, k, v)),
                                                  cu_seqlens_q=_cu([L] * (b - a)), cu_seqlens_k=_cu([L] * (b - a)), causal=True)

    full = run(0, n)
    for _ in range(4):
        assert all(torch.equal(x, y) for x, y in zip(run(0, n), full))
    for a, b in ((0, 12), (12, 13), (13, 60), (60, n)):
        assert all(torch.equal(x, y[a * L:b * L]) for x, y in zip(run(a, b), full)), (a, b)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lq,n", [(640, 8), (640, 90), (2, 90)])
def test_large_values_under_climbing_scores(D, Lq, n):
    """bf16 values near 2^100 under scores that climb by up to 40: P.V stays finite, as P does not grow with them."""
    L, H = 640, 2
    q, k, v = _climbing(torch.bfloat16, D, n, L, H, 10.0, 2)
    q = q[:, :Lq].contiguous()
    v = (v.float() * 2.0 ** 100).to(torch.bfloat16)

    def run(a, b):
        with torch.no_grad():
            return vb.packed_varlen_attn(*(t[a:b].reshape(-1, H, D) for t in (q, k, v)), cu_seqlens_q=_cu([Lq] * (b - a)),
                                         cu_seqlens_k=_cu([L] * (b - a)), split_k_block=L)  # (how keys are cut depends on the batch)

    o = run(0, n)
    ro, _ = _ref(q[:8], k[:8], v[:8], D ** -0.5)
    # P and O are rounded to the type, half an eps each
    assert (o[:8 * Lq].view_as(ro).double() - ro).abs().max() <= (torch.finfo(o.dtype).eps + 1e-3) * v.abs().max().double()
    for _ in range(3):
        assert torch.equal(run(0, n), o)
    assert torch.equal(run(3, 8), o[3 * Lq:8 * Lq])

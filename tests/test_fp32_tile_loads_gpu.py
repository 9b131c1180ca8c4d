"""fp32 rows copied asynchronously and rows read element by element give the same bits: more segments than a block has
threads, shares of a tile without a block, tile edges."""
import pytest
import torch

import varlenabsorbflashattn_b200 as vb

pytestmark = pytest.mark.gpu


def _off(t):
    """The same rows, one element off the 16-byte boundary: they cannot be read four at a time."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("D", [32, 64, 128, 256])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("ql,kl", [([i % 5 for i in range(600)], [(i * 7) % 11 for i in range(600)]),
                                   ([70, 1, 300], [1300, 64, 20]), ([64], [65])])
def test_same_bits(D, causal, ql, kl):
    gen = torch.Generator(device="cuda").manual_seed(3)
    cu = [torch.tensor([0] + n, device="cuda").cumsum(0).to(torch.int32) for n in (ql, kl)]
    q, d_o = (torch.randn(sum(ql), 2, D, generator=gen, device="cuda") for _ in range(2))
    k, v = (torch.randn(sum(kl), 2, D, generator=gen, device="cuda") for _ in range(2))
    outs = []
    for place in (lambda t: t, _off):
        g = [place(t).detach().requires_grad_(True) for t in (q, k, v)]
        o = vb.packed_varlen_attn(*g, cu_seqlens_q=cu[0], cu_seqlens_k=cu[1], causal=causal)
        outs.append([o] + list(torch.autograd.grad(o, g, place(d_o))))
    for a, b in zip(*outs):
        assert torch.equal(a, b) and torch.isfinite(a).all()


def test_thousands_of_segments_as_in_pieces():
    """5000 segments (two rounds of the search for a tile's segment) against calls on 125 of them (one round).  Sums over the
    same rows in another order: a few ulps."""
    ql, kl, n = [8 + i % 60 for i in range(5000)], [8 + i % 41 for i in range(5000)], 125
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, d_o = (torch.randn(sum(ql), 1, 64, generator=gen, device="cuda") for _ in range(2))
    k, v = (torch.randn(sum(kl), 1, 64, generator=gen, device="cuda") for _ in range(2))

    def call(a, b):
        cu = [torch.tensor([0] + x[a:b], device="cuda").cumsum(0).to(torch.int32) for x in (ql, kl)]
        rq, rk = slice(sum(ql[:a]), sum(ql[:b])), slice(sum(kl[:a]), sum(kl[:b]))
        g = [t.detach().requires_grad_(True) for t in (q[rq], k[rk], v[rk])]
        o = vb.packed_varlen_attn(*g, cu_seqlens_q=cu[0], cu_seqlens_k=cu[1])
        return [o.detach()] + list(torch.autograd.grad(o, g, d_o[rq]))

    whole = call(0, 5000)
    pieces = [torch.cat(x) for x in zip(*(call(a, a + n) for a in range(0, 5000, n)))]
    for a, b in zip(whole, pieces):
        assert torch.isfinite(a).all() and float((a - b).norm() / b.norm()) < 1e-6 and float((a - b).abs().max()) < 1e-5

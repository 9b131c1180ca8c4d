"""The check of cu_seqlens on the GPU: what a checked call refuses, and with which error; vafa_check_cu_seqlens on its own."""
import pytest
import torch

import varlenabsorbflashattn_b200 as vb
from varlenabsorbflashattn_b200 import _lib

pytestmark = pytest.mark.gpu


def _cu(*v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("cu_q,cu_k,text", [
    ((1, 4), (0, 6), "cu_seqlens_q"), ((0, 3), (0, 6), "cu_seqlens_q"), ((0, 4), (0, 7), "cu_seqlens_k"),
    ((0, 5, 4), (0, 2, 6), "cu_seqlens_q"), ((0, 2, 4), (0, 7, 6), "cu_seqlens_k"), ((0,), (0,), "at least 2")])
def test_bad_arrays_are_refused(cu_q, cu_k, text):
    q, k, v = (torch.randn(n, 1, 64, device="cuda", dtype=torch.bfloat16) for n in (4, 6, 6))
    with pytest.raises(ValueError, match=text):
        vb.packed_varlen_attn(q, k, v, cu_seqlens_q=_cu(*cu_q), cu_seqlens_k=_cu(*cu_k))


@pytest.mark.parametrize("n_seg", [1, 5000])
def test_good_arrays_pass(n_seg):
    x = torch.randn(3 * n_seg, 1, 64, device="cuda", dtype=torch.bfloat16)
    cu = torch.arange(0, 3 * n_seg + 1, 3, device="cuda", dtype=torch.int64)
    a = vb.packed_varlen_attn(x, x, x, cu_seqlens_q=cu, cu_seqlens_k=cu.clone())
    c32 = cu.to(torch.int32)
    assert torch.equal(a, vb.packed_varlen_attn(x, x, x, cu_seqlens_q=c32, cu_seqlens_k=c32))


def test_more_rows_than_32_bits_count_are_refused():
    """2^32 + 1 keys (17 GB that nobody writes or reads) must not arrive in the library as one."""
    torch.cuda.empty_cache()
    X = torch.empty(2 ** 32 + 1, 1, device="cuda")
    q_raw, W = torch.randn(3, 8, device="cuda"), [torch.randn(d, 1, 16, device="cuda") for d in (8, 1, 1)]
    for validate in (True, False):
        with pytest.raises(ValueError, match="int32"):
            vb.packed_target_attn(q_raw, X, *W, cu_seqlens_q=_cu(0, 3), cu_seqlens_k=_cu(0, 1), validate=validate)
    with pytest.raises(ValueError, match="int32"):
        vb.target_attn_inner(torch.randn(3, 1, 1, device="cuda"), X, W[2], _cu(0, 3), _cu(0, 1))
    del X
    torch.cuda.empty_cache()


@pytest.mark.parametrize("cu_q,cu_k,need_keys,rc", [
    ((0, 4), (0, 6), 0, 0), ((0, 2, 2, 4), (0, 0, 6, 6), 0, 0), ((0, 2, 4), (0, 3, 6), 1, 0), ((0, 0, 4), (0, 0, 6), 1, 0),
    ((1, 4), (0, 6), 0, 1), ((0, 4), (1, 6), 0, 1), ((0, 3), (0, 6), 0, 1), ((0, 4), (0, 7), 0, 1), ((0, 5, 4), (0, 2, 6), 0, 1),
    ((0, 2, 4), (0, 7, 6), 0, 1), ((0, 2, 4), (0, 0, 6), 1, 1), ((0, 2, 4), (0, 6, 6), 1, 1)])
def test_the_check_as_a_call_of_its_own(cu_q, cu_k, need_keys, rc):
    a, b = _cu(*cu_q), _cu(*cu_k)
    stream = _lib.raw_stream(a.device)
    assert _lib.load().vafa_check_cu_seqlens(a.data_ptr(), b.data_ptr(), len(cu_q) - 1, 4, 6, need_keys, stream) == rc


def test_the_check_as_a_call_of_its_own_wants_arrays():
    a = _cu(0, 4)
    lib, stream = _lib.load(), _lib.raw_stream(a.device)
    assert lib.vafa_check_cu_seqlens(a.data_ptr(), None, 1, 4, 4, 0, stream) < 0
    assert lib.vafa_check_cu_seqlens(a.data_ptr(), a.data_ptr(), 0, 4, 4, 0, stream) < 0

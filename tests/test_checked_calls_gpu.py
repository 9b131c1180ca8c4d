"""Forward calls that look over cu_seqlens on the device: what they refuse, that a refused call leaves nothing behind, and that
good calls give what unchecked ones give, from several threads and streams."""
import os
import threading
import time

import pytest
import torch

import varlenabsorbflashattn_b200 as vb

pytestmark = pytest.mark.gpu
QL, KL = [3, 0, 130, 1], [5, 0, 300, 128]
TQ, TK = sum(QL), sum(KL)
BAD = [((1, 3, 133, 134), None), ((0, 3, 3, 133, 135), None), ((0, 3, 200, 133, 134), None), ((0, -5, 3, 133, 134), None),
       ((0, 3, 3, 2 ** 30, 134), None), (None, (0, 5, 5, 434, 433)), (None, (0, 5, 5, 305, 2 ** 31 - 1)), (None, (7, 5, 5, 305, 433))]


def _cu(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _sum(lens):
    return torch.tensor([0] + lens).cumsum(0).tolist()


def _operators():
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = r(TQ, 2, 128), r(TK, 2, 128), r(TK, 2, 128)
    q_raw, X, u = r(TQ, 256), r(TK, 256), r(TQ, 8, 256)
    W = [r(256, 8, 32) / 16 for _ in range(3)]

    def varlen(cq, ck, check):
        if not check:
            vb.set_validate_cu_seqlens(False)
        try:
            return vb.packed_varlen_attn(q, k, v, cu_seqlens_q=cq, cu_seqlens_k=ck)
        finally:
            vb.set_validate_cu_seqlens(True)

    return {"varlen": varlen,
            "varlen fp32": lambda cq, ck, check: vb.packed_varlen_attn(q.float(), k.float(), v.float(), cu_seqlens_q=cq, cu_seqlens_k=ck),
            "absorb": lambda cq, ck, check: vb.packed_target_attn(q_raw, X, *W, cu_seqlens_q=cq, cu_seqlens_k=ck, validate=check),
            "inner": lambda cq, ck, check: vb.target_attn_inner(u, X, W[2], cq, ck, validate=check)}


@pytest.mark.parametrize("name", ["varlen", "varlen fp32", "absorb", "inner"])
def test_bad_arrays_are_refused_and_leave_nothing_behind(name):
    call, good = _operators()[name], (_cu(_sum(QL)), _cu(_sum(KL)))
    want = call(*good, False)
    for bq, bk in BAD:
        if bq is not None and len(bq) == 4:
            with pytest.raises((ValueError, AssertionError)):
                call(_cu(bq), good[1], True)
            continue
        with pytest.raises(ValueError):
            call(_cu(bq) if bq else good[0], _cu(bk) if bk else good[1], True)
        assert torch.equal(call(*good, True), want)


@pytest.mark.parametrize("name", ["varlen", "absorb"])
def test_sums_that_fall_and_rise_again(name):
    """Two batches put together whose second was not offset: a tile of the fp32 kernels lies in two segments, and clusters
    (several hundred keys a segment, one head) share it."""
    rng = torch.Generator().manual_seed(4)
    lens = torch.randint(150, 450, (130,), generator=rng).tolist()
    qlens = lens if name == "varlen" else torch.randint(8, 24, (130,), generator=rng).tolist()
    good = _cu(_sum(qlens)), _cu(_sum(lens))
    T, Tk, g = sum(qlens), sum(lens), torch.Generator(device="cuda").manual_seed(4)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    if name == "varlen":
        q, k, v = r(T, 1, 64), r(Tk, 1, 64), r(Tk, 1, 64)
        call = lambda cq, ck: vb.packed_varlen_attn(q, k, v, cu_seqlens_q=cq, cu_seqlens_k=ck)
    else:
        q_raw, X, W = r(T, 64), r(Tk, 64), [r(64, 2, 32) / 8 for _ in range(3)]
        call = lambda cq, ck: vb.packed_target_attn(q_raw, X, *W, cu_seqlens_q=cq, cu_seqlens_k=ck)
    want = call(*good)

    def twice(cu, at):  # rises for `at` segments, starts again, ends where it should
        v = cu.tolist()
        return _cu(v[:at + 1] + [x - v[at] for x in v[at + 1:-1]] + [v[-1]])

    for at in (40, 64, 65, 100, 128):
        for bad in ((twice(good[0], at), good[1]), (good[0], twice(good[1], at)), (twice(good[0], at), twice(good[1], at))):
            with pytest.raises(ValueError):
                call(*bad)
        assert torch.equal(call(*good), want)


def test_threads_and_streams():
    call, good, bad = _operators()["absorb"], (_cu(_sum(QL)), _cu(_sum(KL))), _cu((0, 3, 200, 133, 134))
    want, errors = call(*good, False), []
    torch.cuda.synchronize()

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                out = call(*good, True)
                try:
                    call(bad, good[1], True)
                    errors.append("not refused")
                except ValueError:
                    pass
                torch.cuda.current_stream().synchronize()
                if not torch.equal(out, want):
                    errors.append("other result")

    threads = [threading.Thread(target=work) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors[:3]


def test_a_threads_end_does_not_wait_for_the_gpu():
    """The end of a thread that has made checked calls, while the GPU is busy for about a second."""
    call, good = _operators()["varlen fp32"], (_cu(_sum(QL)), _cu(_sum(KL)))
    want, got, ids = call(*good, True), [], []
    called, leave = threading.Event(), threading.Event()

    def work():
        ids.append(threading.get_native_id())
        with torch.cuda.stream(torch.cuda.Stream()):
            got.append(call(*good, True))
            torch.cuda.current_stream().synchronize()
        called.set()
        leave.wait(10)

    thread = threading.Thread(target=work)
    thread.start()
    assert called.wait(60)
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(2_000_000_000)
        end = torch.cuda.current_stream().record_event()
    leave.set()
    thread.join()
    t0 = time.monotonic()
    while time.monotonic() - t0 < 0.4 and os.path.exists(f"/proc/self/task/{ids[0]}"):
        time.sleep(0.01)
    gone, asleep = not os.path.exists(f"/proc/self/task/{ids[0]}"), not end.query()
    torch.cuda.synchronize()
    assert asleep, "the sleep was too short for the test"
    assert gone and torch.equal(got[0], want)

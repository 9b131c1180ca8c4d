"""Absorb calls from several streams and threads: side streams are not shared between callers, results stay what they are."""
import threading
import time

import pytest
import torch

import varlenabsorbflashattn_b200 as vb
from oracle import make_absorb_inputs

pytestmark = pytest.mark.gpu


def _step(seed=3, n=24):
    ql, kl = [1 + (5 * i) % 20 for i in range(n)], [8 + (97 * i) % 700 for i in range(n)]
    ins = make_absorb_inputs(ql, kl, 256, 256, 8, 32, torch.bfloat16, seed)
    g = [t.cuda().requires_grad_(True) for t in ins[:5]]
    dO, cu_q, cu_k = ins[5].cuda(), ins[6].cuda(), ins[7].cuda()

    def step(check=False):
        o = vb.packed_target_attn(*g, cu_seqlens_q=cu_q, cu_seqlens_k=cu_k, validate=check)
        return [o.detach()] + list(torch.autograd.grad(o, g, dO))
    return step


def test_a_stream_does_not_wait_for_another_ones_backlog():
    """One stream sleeps for about a second and has a step behind that; steps on other streams are done meanwhile.  (Streams can
    meet in a hardware queue: it is enough that half of them get through.)"""
    step = _step()
    streams = [torch.cuda.Stream() for _ in range(7)]
    torch.cuda.synchronize()
    for s in streams:  # what is made on first use
        with torch.cuda.stream(s):
            step()
    torch.cuda.synchronize()
    busy, others = streams[0], streams[1:]
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)
        step()
        end = busy.record_event()
    done = []
    for s in others:
        with torch.cuda.stream(s):
            step()
            done.append(s.record_event())
    t0 = time.monotonic()
    while time.monotonic() - t0 < 0.4 and not all(e.query() for e in done):
        time.sleep(0.01)
    through, asleep = sum(e.query() for e in done), not end.query()
    torch.cuda.synchronize()
    assert asleep, "the sleep was too short for the test"
    assert through >= len(others) // 2, f"{through} of {len(others)} got through"


def test_steps_from_threads_on_streams_of_both_priorities():
    steps = [_step(seed) for seed in range(3)]
    want = [s() for s in steps]
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            for k in range(12):  # more streams than are kept, one after another
                with torch.cuda.stream(torch.cuda.Stream(priority=-1 if (i + k) % 2 else 0)):
                    got = steps[i](check=k % 3 == 0)
                    torch.cuda.current_stream().synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                        errors.append(f"thread {i}, call {k}: other result")
        except Exception as e:  # noqa: BLE001 - a thread's error has to reach the test
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors[:3]


def test_a_call_beside_a_capture_of_another_stream():
    """While one stream is captured with an absorb call in it, a call on another stream goes on, and both give their results."""
    inside, beside = _step(7), _step(8)
    want = inside(), beside()
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    for st, step in ((s, inside), (other, beside)):
        with torch.cuda.stream(st):
            for _ in range(3):
                step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
        captured = inside()
        with torch.cuda.stream(other):
            got = beside()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip((captured, got), want):
        assert all(torch.equal(x, y) for x, y in zip(a, b))

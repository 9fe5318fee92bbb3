"""Prefill calls that could meet in a buffer of the library: several host threads, streams and recordings."""
import threading

import pytest

from tests.util import D, SCALE, TYPES

pytestmark = pytest.mark.gpu
HKV, HQ = 2, 12
SHAPES = [(48, 6000), (5, 9000), (130, 4000)]   # rows, history: cut row tiles


class _Call:
    """one prefill call with inputs of its own; scratch: "library", or "caller" for the smallest that takes the context in one pass"""

    def __init__(self, cuda, seed, shape, scratch):
        import torch
        from p100e_engine_b200 import fast
        self.T, self.p0 = shape
        n = self.T + self.p0
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.c = fast.kv_alloc(TYPES["q8_0"], n, HKV, D)
        assert fast.kv_fill_random(self.c, 0, n, seed)
        self.q, self.gate = torch.randn(self.T, HQ, D, generator=g, device=cuda), torch.randn(self.T, HQ * D, generator=g, device=cuda)
        self.out = torch.full((self.T, HQ, D), float("nan"), device=cuda)
        self.nb = fast.attn_fold_scratch_bytes(self.T, HKV, n) if scratch == "caller" else 0
        self.scratch = torch.empty(self.nb, dtype=torch.uint8, device=cuda) if self.nb else None
        self.want = None

    def __call__(self, s=None):
        from p100e_engine_b200 import fast
        assert fast.attn_prefill_gated(self.q, self.c, self.out, self.gate, self.T, self.p0, HQ, SCALE, self.scratch, self.nb, s=s)

    def alone(self):
        import torch
        self()
        torch.cuda.synchronize()
        self.want = self.out.clone()
        self.out.fill_(float("nan"))
        torch.cuda.synchronize()


def _in_threads(calls, streams, rounds=40):
    import torch
    failed = []

    def work(call, stream):
        try:
            torch.cuda.set_device(0)
            for _ in range(rounds):
                call(stream)
        except BaseException as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=x) for x in zip(calls, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    for c in calls:
        assert torch.equal(c.out, c.want)


@pytest.mark.parametrize("scratch", ["library", "caller"])
def test_threads_on_one_stream_and_on_several(cuda, lib, scratch):
    import torch
    from p100e_engine_b200 import fast
    calls = [_Call(cuda, i, SHAPES[i % 3], scratch) for i in range(4)]
    for c in calls:
        c.alone()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    _in_threads(calls, [a, a, b, b])
    assert fast.device_status() == 0


def test_threads_on_the_per_thread_stream(cuda, lib):
    """cudaStreamPerThread is one handle and a stream per thread"""
    from p100e_engine_b200 import fast
    calls = [_Call(cuda, i, SHAPES[i % 3], "caller") for i in range(3)]
    for c in calls:
        c.alone()
    _in_threads(calls, [2, 2, 2])
    assert fast.device_status() == 0


def test_replay_elsewhere_beside_a_call_on_the_recording_stream(cuda, lib):
    """a recorded call with the library's scratch, replayed on another stream, and a call with the caller's scratch on the stream it was recorded
    on share nothing"""
    import torch
    from p100e_engine_b200 import fast
    rec, own = _Call(cuda, 1, SHAPES[0], "library"), _Call(cuda, 2, SHAPES[1], "caller")
    rec.alone()
    own.alone()
    a, b, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(a):
        rec(a)                                   # sizes the stream's scratch
        a.synchronize()
        with torch.cuda.graph(graph, stream=a):
            rec(a)
    torch.cuda.synchronize()
    for _ in range(30):
        with torch.cuda.stream(b):
            graph.replay()
        own(a)
    torch.cuda.synchronize()
    assert torch.equal(rec.out, rec.want) and torch.equal(own.out, own.want)
    assert fast.device_status() == 0


@pytest.mark.parametrize("shape", SHAPES)
def test_room_in_the_callers_scratch(cuda, lib, shape):
    """with room for images and partial sums a call is the same, recorded or not, with the library's scratch or its own; without, a recorded
    call runs a row tile per CTA: the same attention, to f16 operands and fp32 sums (2e-3 of the largest output)"""
    import torch
    from p100e_engine_b200 import fast
    call = _Call(cuda, 3, shape, "library")
    call.alone()
    n = shape[0] + shape[1]
    small = fast.attn_fold_scratch_bytes(shape[0], HKV, n)
    for nb in (small, small + (40 << 20)):
        call.nb, call.scratch = nb, torch.empty(nb, dtype=torch.uint8, device=cuda)
        call.out.fill_(float("nan"))
        call()
        torch.cuda.synchronize()
        assert torch.equal(call.out, call.want)
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            call(side)
        call.out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        if nb == small:
            assert (call.out - call.want).abs().max() <= 2e-3 * call.want.abs().max()
        else:
            assert torch.equal(call.out, call.want)
    assert fast.device_status() == 0


def test_an_earlier_larger_call_does_not_change_a_call(cuda, lib):
    """165000 keys of four heads are more images than one pass of the library's scratch holds; a call with 20000 rows in between needs a little
    more of it, which makes the buffer larger, not the passes"""
    import torch
    from p100e_engine_b200 import fast
    n, T, hkv, hq = 165000, 5, 4, 24
    c = fast.kv_alloc(TYPES["q4_0"], n, hkv, D)
    assert fast.kv_fill_random(c, 0, n, 5)
    q = torch.randn(T, hq, D, device=cuda, generator=torch.Generator(device="cuda").manual_seed(1))
    big = torch.zeros(20000, hq, D, device=cuda)
    big_out, outs = torch.empty_like(big), [torch.full((T, hq, D), float("nan"), device=cuda) for _ in range(2)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(2):
        n0 = lib.b200_launch_count()
        assert fast.attn_prefill(q, c, outs[i], T, n - T, hq, SCALE, s=s)
        assert lib.b200_launch_count() - n0 == 4     # two passes
        assert fast.attn_prefill(big, c, big_out, big.shape[0], n - big.shape[0], hq, SCALE, s=s)
    s.synchronize()
    assert torch.equal(outs[0], outs[1])
    assert fast.device_status() == 0

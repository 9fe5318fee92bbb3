"""Run plans that the calls of a declared step share, with CUDA graphs recorded and replayed in between: every call and every replay equals
the same call without a declared step, bit for bit."""
import numpy as np
import pytest

from tests.util import D, SCALE, TYPES

pytestmark = pytest.mark.gpu
HKV, HQ, CAP = 4, 24, 6144
SHORT, LONG = [700, 65, 1500, 300, 2049, 64], [1900, 4000, 1501, 6000, 2050, 5000]


class _Batch:
    """six sequences in one pool; a call of one kind over their last rows"""

    def __init__(self, lib, cuda, tname, kind, q_len):
        import torch
        from p100e_engine_b200 import fast
        from p100e_engine_b200.pool import Pool
        n = len(LONG)
        self.lib, self.kind, self.q_len, self.n, self.s = lib, kind, q_len, n, torch.cuda.Stream()
        self.pool = Pool(TYPES[tname], HKV, 1, n * CAP // 256, 8, D, max_slots=n, max_pages=CAP // 256, max_rows=4 * n, device=0)
        with torch.cuda.stream(self.s):
            for i in range(n):
                assert self.pool.ensure(i, CAP, self.s.cuda_stream) == 0
                assert fast.kv_fill_random(self.pool.view(0, i), 0, CAP, 17 + i)
            self.q = torch.randn(4 * n, HQ, D, device=cuda, generator=torch.Generator(device="cuda").manual_seed(3))
        assert fast.attn_reserve(TYPES[tname], n, 4, CAP, CAP, HKV, 64, s=self.s)   # the largest call: nothing is allocated in a recording
        self.s.synchronize()

    def step(self, lens):
        past = np.array([x - self.q_len for x in lens], np.int32)
        assert self.pool.step(np.arange(self.n, dtype=np.int32), past, self.q_len, stream=self.s.cuda_stream) == 0

    def call(self, out, kind=None):
        from p100e_engine_b200 import fast
        view, pos = self.pool.view(0, -1), self.pool.step_arrays()[1]
        kind = kind or self.kind
        n0 = self.lib.b200_launch_count()
        if kind == "rows":
            assert fast.attn_decode_rows(self.q, view, out, self.n, pos, HQ, SCALE, s=self.s)
        else:
            assert fast.attn_decode_slots(self.q, view, out, None, self.n, self.q_len, pos, CAP, HQ, SCALE, kind, s=self.s)
        return self.lib.b200_launch_count() - n0

    def new_out(self):
        import torch
        return torch.full((self.n * self.q_len, HQ, D), float("nan"), device="cuda")

    def want(self, lens):
        from p100e_engine_b200 import fast
        out = self.new_out()
        self.step(lens)
        assert fast.attn_step_end(self.s)
        self.call(out)
        self.s.synchronize()
        return out

    def record(self, out, kind=None):
        import torch
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=self.s):
            launches = self.call(out, kind)
        return g, launches

    def replay(self, g):
        import torch
        with torch.cuda.stream(self.s):
            g.replay()


KINDS = [("f16", "rows", 1), ("q8_0", 64, 1), ("q8_0", 64, 4), ("f16", -1, 1), ("q8_0", -1, 4)]   # -1 with 4 rows of q8_0: the verify kernel


@pytest.mark.parametrize("tname,kind,q_len", KINDS)
def test_calls_then_recording_then_the_next_step(cuda, lib, tname, kind, q_len):
    import torch
    b = _Batch(lib, cuda, tname, kind, q_len)
    short, long = b.want(SHORT), b.want(LONG)
    out, rec = b.new_out(), b.new_out()
    torch.cuda.synchronize()
    b.step(SHORT)
    full = b.call(out)
    assert b.call(out) == full - 1                   # the plan is shared
    g, launches = b.record(rec)
    assert launches == full                          # a recording brings its own
    for lens, want in ((LONG, long), (SHORT, short)):
        b.step(lens)
        b.replay(g)
        b.s.synchronize()
        assert torch.equal(rec, want)
    assert torch.equal(out, short)


@pytest.mark.parametrize("tname,kind,q_len", KINDS)
def test_recording_then_the_call_itself(cuda, lib, tname, kind, q_len):
    import torch
    b = _Batch(lib, cuda, tname, kind, q_len)
    long = b.want(LONG)
    out, rec = b.new_out(), b.new_out()
    torch.cuda.synchronize()
    b.step(LONG)
    g, full = b.record(rec)
    assert b.call(out) == full                       # nothing has run yet that could have left a plan
    b.s.synchronize()
    assert torch.equal(out, long)
    b.replay(g)
    b.s.synchronize()
    assert torch.equal(rec, long)


@pytest.mark.parametrize("tname,kind,q_len", KINDS)
def test_replay_between_two_calls_of_a_step(cuda, lib, tname, kind, q_len):
    import torch
    b = _Batch(lib, cuda, tname, kind, q_len)
    want = b.want(SHORT)
    out, rec = b.new_out(), b.new_out()
    torch.cuda.synchronize()
    b.step(LONG)
    other = 128 if kind != 128 else 256
    g, _ = b.record(rec, other)                      # another shape: partials of another layout
    b.step(SHORT)
    full = b.call(out)
    b.replay(g)
    out.fill_(float("nan"))
    torch.cuda.synchronize()
    assert b.call(out) == full - 1
    b.s.synchronize()
    assert torch.equal(out, want)


def test_two_layers_of_one_recording_share_a_plan(cuda, lib):
    import torch
    b = _Batch(lib, cuda, "q8_0", "rows", 1)
    long, short = b.want(LONG), b.want(SHORT)
    outs = [b.new_out(), b.new_out()]
    torch.cuda.synchronize()
    b.step(SHORT)
    b.call(outs[0])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=b.s):
        first, second = b.call(outs[0]), b.call(outs[1])
    assert second == first - 1
    for lens, want in ((LONG, long), (SHORT, short)):
        b.step(lens)
        b.replay(g)
        b.s.synchronize()
        assert all(torch.equal(o, want) for o in outs)


def test_even_split_and_fixed_chunks_of_one_geometry(cuda, lib):
    """f16, 4 kv heads, two slots of up to 2432 keys in 64-key chunks: as many partials as the even split over 74 CTAs per head, the same
    chunk and the same chunk count.  Each kind computes its own plan."""
    import torch
    from p100e_engine_b200 import fast
    n = 2432
    c = fast.kv_alloc(TYPES["f16"], n, HKV, D)
    g = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    assert fast.kv_append(c, rn(n, HKV, D), rn(n, HKV, D), 0, n)
    q, pos = rn(2, HQ, D), torch.tensor([n - 1, 2400], dtype=torch.int32, device=cuda)

    def call(chunk):
        out = torch.full((2, HQ, D), float("nan"), device=cuda)
        n0 = lib.b200_launch_count()
        assert fast.attn_decode_slots(q, c, out, None, 2, 1, pos, n, HQ, SCALE, chunk)
        launches = lib.b200_launch_count() - n0
        torch.cuda.synchronize()
        return out, launches

    want = {chunk: call(chunk)[0] for chunk in (64, -1)}
    assert fast.attn_step_begin(pos)
    try:
        for chunk, launches in ((64, 3), (64, 2), (-1, 3), (-1, 2), (64, 3)):
            out, k = call(chunk)
            assert k == launches, chunk
            assert torch.equal(out, want[chunk]), chunk
    finally:
        assert fast.attn_step_end()
    assert fast.device_status() == 0

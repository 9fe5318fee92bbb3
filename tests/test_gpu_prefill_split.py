"""Prefill attention where row tiles are cut between CTAs: few row tiles behind a long history, runs that start or end inside a tile, a
last step with a single 64-key image, rows that see none of a piece's keys; every form of the result."""
import numpy as np
import pytest

from oracle import orc
from tests import util
from tests.util import D, SCALE, TYPES

pytestmark = pytest.mark.gpu


def _filled(kt, n, cuda, seed, hkv):
    import torch
    from p100e_engine_b200 import fast
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = fast.kv_alloc(kt, n, hkv, D)
    assert fast.kv_append(c, torch.randn(n, hkv, D, generator=g, device=cuda), torch.randn(n, hkv, D, generator=g, device=cuda), 0, n)
    torch.cuda.synchronize()
    return c, orc.Cache(kt, n, hkv, D, c.k.cpu().numpy(), c.v.cpu().numpy())


# operands in f16, sums in fp32, in any split of the keys: held to the usual bar (2e-3 of the largest output, 1e-2 rms)
@pytest.mark.parametrize("tname,hkv,p0,T", [
    ("q8_0", 1, 6000, 1),        # one tile over every CTA that gets work
    ("q8_0", 4, 5000, 22),       # two tiles per head, the second with 4 rows
    ("q4_0", 2, 8191, 5),        # the last step holds one 64-key image
    ("f16", 1, 4031, 43),        # tile of 128 rows + tile of 130: ends inside an image
    ("q8_0", 1, 0, 700),         # causal ramp: tiles of 1 .. 6 steps, rows that see none of a piece's keys
    ("q8_0", 3, 1000, 130),
    ("q8_0", 2, 2685, 174),      # runs that start at the last step of a tile, which its first rows do not see
    ("f16", 2, 3055, 174),
    ("q4_0", 1, 40, 1500),       # left whole: the first runs would cross many tiles of one step
])
def test_cut_row_tiles_vs_oracle(cuda, lib, tname, hkv, p0, T):
    import torch
    from p100e_engine_b200 import fast
    hq = 6 * hkv
    c, oc = _filled(TYPES[tname], p0 + T, cuda, p0 + T, hkv)
    q = util.rng_normal(p0 + 7, (T, hq, D))
    gate = util.rng_normal(p0 + 8, (T, hq * D))
    qd, gd = util.to_dev(q, cuda), util.to_dev(gate, cuda)
    ref = orc.attention(q, oc, T, hq, SCALE, p0=p0, gate=gate)
    what = "%s hkv=%d p0=%d T=%d" % (tname, hkv, p0, T)
    out, a16 = torch.full((T, hq, D), float("nan"), device=cuda), torch.zeros(T * hq * 8 * 17, 2, dtype=torch.float16, device=cuda)
    assert fast.attn_prefill_gated_a16(qd, c, out, gd, a16, T, p0, hq, SCALE, None, 0)
    # the caller's scratch, with and without recording (a recorded call runs one tile per CTA)
    nb = fast.attn_fold_scratch_bytes(T, hkv, p0 + T)
    scratch = torch.empty(nb, dtype=torch.uint8, device=cuda)
    own, rec = torch.full_like(out, float("nan")), torch.full_like(out, float("nan"))
    assert fast.attn_prefill_gated(qd, c, own, gd, T, p0, hq, SCALE, scratch, nb)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        assert fast.attn_prefill_gated(qd, c, rec, gd, T, p0, hq, SCALE, scratch, nb)
    graph.replay()
    # passes of few keys carry their state through the result
    few = fast.attn_fold_scratch_bytes(T, hkv, 512)
    passes = torch.full_like(out, float("nan"))
    assert fast.attn_prefill_gated(qd, c, passes, gd, T, p0, hq, SCALE, scratch, min(few, nb))
    torch.cuda.synchronize()
    assert fast.device_status() == 0
    util.check_close(out.cpu().numpy(), ref, what)
    assert torch.equal(own, out), what
    util.check_close(rec.cpu().numpy(), ref, "recorded " + what)
    util.check_close(passes.cpu().numpy(), ref, "passes " + what)
    # the a16 copy is that of the result
    x, y, copy = out.reshape(T, hq * D), torch.empty(T, hq * D, device=cuda), torch.zeros_like(a16)
    big = torch.full_like(x, 200.0)   # sigmoid = 1
    assert fast.ew_quant(fast.EW_SIGMOID_MUL, x, big, y, copy, T, hq * D)
    torch.cuda.synchronize()
    assert torch.equal(copy.view(torch.int16), a16.view(torch.int16)), what


@pytest.mark.parametrize("p0,T", [(3000, 50), (0, 300)])
def test_cut_row_tiles_bf16_form(cuda, lib, p0, T):
    """bf16 rows in, bf16 result and gate: the rounding of the result (2^-9 relative) on top of the usual bar"""
    import torch
    from p100e_engine_b200 import fast
    hkv, hq = 2, 12
    c, _ = _filled(TYPES["q8_0"], p0 + T, cuda, 3, hkv)
    bf = lambda seed, h: util.to_dev(util.rng_normal(seed, (T, h, D)), cuda).to(torch.bfloat16)
    q, k, v, gate = bf(1, hq), bf(2, hkv), bf(3, hkv), bf(4, hq)
    nb = fast.attn_prefill_bf16_scratch_bytes(T, hkv, p0 + T, True)
    scratch = torch.empty(nb, dtype=torch.uint8, device=cuda)
    out = torch.zeros(T, hq, D, dtype=torch.bfloat16, device=cuda)
    assert fast.attn_prefill_bf16(q, k, v, None, gate, None, out, None, c, p0, T, hq, 64, 1e7, SCALE, scratch, nb)
    qr = torch.zeros(T, hq, D, device=cuda)
    assert fast.rope_append_bf16(q, k, v, qr, c, p0, T, hq, hkv, D, 64, 1e7)
    torch.cuda.synchronize()
    assert fast.device_status() == 0
    oc = orc.Cache(TYPES["q8_0"], p0 + T, hkv, D, c.k.cpu().numpy(), c.v.cpu().numpy())
    ref = orc.attention(qr.cpu().numpy(), oc, T, hq, SCALE, p0=p0, gate=gate.float().reshape(T, -1).cpu().numpy())
    util.check_close(out.float().cpu().numpy(), ref, "bf16 p0=%d T=%d" % (p0, T), 2e-3 + 2.0 ** -9, 1e-2)

"""Decode attention where the key split can go wrong: ends of contexts inside a 64-key tile, with page rows past the end that
hold anything; boundaries of the default chunk grid; one slot with the even split; the allocation-free entry in head groups."""
import numpy as np
import pytest

from oracle import orc
from tests import util
from tests.util import D, HKV, HQ, SCALE, TYPES

pytestmark = pytest.mark.gpu


def _paged(cuda, kt, n, seed, hkv=HKV, extra_pages=0):
    """one sequence of n positions in 256-row pages; every byte of the pool that is not a stored row is 0xff (f16 NaN)"""
    import torch
    from p100e_engine_b200 import fast
    npg = (n + 255) // 256
    pool = util.PagedPool(kt, npg + 1, psh=8, hkv=hkv, seed=seed)
    pt = pool.take(n, npg + extra_pages)
    pool_t = torch.full((pool.bytes,), 0xff, dtype=torch.uint8, device=cuda)
    c = util.dev_cache(pool_t, pool, util.to_dev(pt, cuda), None, (npg + extra_pages) << 8)
    g = torch.Generator(device="cuda").manual_seed(seed)
    for p in range(0, n, 8192):
        T = min(8192, n - p)
        assert fast.kv_append(c, torch.randn(T, hkv, D, generator=g, device=cuda), torch.randn(T, hkv, D, generator=g, device=cuda), p, T)
    torch.cuda.synchronize()
    pool.host[:pool.bytes] = pool_t.cpu().numpy()
    return c, pool.host_cache(pt), pool_t


@pytest.mark.parametrize("tname", ["q8_0", "f16", "q4_0"])
@pytest.mark.parametrize("n", [1, 63, 65, 257, 4095, 4097, 8193, 16385 + 31])
def test_ragged_ends_and_grid_boundaries(cuda, lib, tname, n):
    """f16 products of f16 operands summed in fp32: held to the usual bar (2e-3 of the largest output, 1e-2 rms)"""
    import torch
    from p100e_engine_b200 import fast
    c, hc, _keep = _paged(cuda, TYPES[tname], n, n)
    for T in (1, 4):
        if T > n:
            continue
        q = util.rng_normal(n + T, (T, HQ, D))
        qd, pos = util.to_dev(q, cuda), torch.arange(n - T, n, dtype=torch.int32, device=cuda)
        ref = orc.attention(q, hc, T, HQ, SCALE, p0=n - T)
        a, b = (torch.full((T, HQ, D), float("nan"), device=cuda) for _ in range(2))
        assert fast.attn_decode(qd, c, a, T, n - T, HQ, SCALE)                                   # default grid
        assert fast.attn_decode_slots(qd, c, b, None, 1, T, pos, n, HQ, SCALE, -1)                # even split of one slot
        torch.cuda.synchronize()
        util.check_close(a.cpu().numpy(), ref, "default grid %s n=%d T=%d" % (tname, n, T))
        util.check_close(b.cpu().numpy(), ref, "even split %s n=%d T=%d" % (tname, n, T))
    assert fast.device_status() == 0


def test_rows_do_not_depend_on_the_call_across_grid_boundaries(cuda, lib):
    """row t of a call that straddles a boundary of the chunk grid == the one-row call, bit for bit, also as one of several
    slots (a run plan) and through the allocation-free entry, whose kv heads then go in groups"""
    import torch
    from p100e_engine_b200 import fast
    n = 12000
    c, _, _keep = _paged(cuda, TYPES["q8_0"], n, 5, extra_pages=50)
    q = util.to_dev(util.rng_normal(6, (4, HQ, D)), cuda)
    for p0 in (4094, 8190, n - 4):
        out, one = torch.zeros(4, HQ, D, device=cuda), torch.zeros(4, HQ, D, device=cuda)
        assert fast.attn_decode(q, c, out, 4, p0, HQ, SCALE)
        for t in range(4):
            assert fast.attn_decode(q[t:t + 1], c, one[t:t + 1], 1, p0 + t, HQ, SCALE)
        rows = torch.zeros(8, HQ, D, device=cuda)
        pos8 = torch.tensor([p0 + t for t in range(4)] + [n - 1 - t for t in range(4)], dtype=torch.int32, device=cuda)
        c.rtab = torch.zeros(8, dtype=torch.int32, device=cuda)
        assert fast.attn_decode_rows(torch.cat([q, q]), c, rows, 8, pos8, HQ, SCALE)
        pos4 = pos8[:4].contiguous()
        free = torch.zeros(4, HQ, D, device=cuda)
        assert fast.attn_decode_slots_noalloc(q, c, free, None, 1, 4, pos4, n, HQ, SCALE, 64) == 0    # 188 chunks: three heads fit
        pinned = torch.zeros(4, HQ, D, device=cuda)
        assert fast.attn_decode_slots(q, c, pinned, None, 1, 4, pos4, n, HQ, SCALE, 64)
        torch.cuda.synchronize()
        assert torch.equal(out, one), p0
        assert torch.equal(rows[:4], out), p0
        assert torch.equal(free, pinned), p0
    assert fast.device_status() == 0
    assert fast.noalloc_device_status() == 0


@pytest.mark.parametrize("tname", ["q8_0", "f16", "q4_0"])
@pytest.mark.parametrize("n_slots", [5, 2100, 8200])   # few units; a plan of runs; more slots than a plan holds
def test_many_slots_of_fixed_chunks(cuda, lib, tname, n_slots):
    """fixed chunks of many ragged slots, some of them without a key: every row equals the one-row call, bit for bit"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv = 400, 1
    g = torch.Generator(device="cuda").manual_seed(n_slots)
    c = fast.kv_alloc(TYPES[tname], n, hkv, D)
    assert fast.kv_append(c, torch.randn(n, hkv, D, generator=g, device=cuda), torch.randn(n, hkv, D, generator=g, device=cuda), 0, n)
    q = torch.randn(n_slots, 6 * hkv, D, generator=g, device=cuda)
    pos = torch.randint(-1, n, (n_slots,), generator=g, device=cuda, dtype=torch.int32)
    pos[:5] = torch.tensor([n - 1, 63, 64, -1, 0], dtype=torch.int32)
    out = torch.full_like(q, float("nan"))
    assert fast.attn_decode_slots(q, c, out, None, n_slots, 1, pos, n, 6 * hkv, SCALE, 64)
    picked = list(range(5)) + list(range(5, n_slots, max(1, n_slots // 40)))
    for i in picked:
        one = torch.full_like(q[:1], float("nan"))
        assert fast.attn_decode_slots(q[i:i + 1], c, one, None, 1, 1, pos[i:i + 1], n, 6 * hkv, SCALE, 64)
        assert torch.equal(one, out[i:i + 1]), (i, int(pos[i]))
    assert torch.isfinite(out).all()
    assert fast.device_status() == 0


@pytest.mark.parametrize("tname,n_slots,q_len,n,hkv", [
    ("q8_0", 64, 1, 4096, 1), ("f16", 16, 4, 8192, 1), ("q4_0", 100, 4, 512, 4), ("q8_0", 100, 4, 512, 1), ("q8_0", 64, 4, 1024, 2),
    ("q4_0", 300, 1, 1024, 2), ("q8_0", 64, 1, 4096, 4), ("q8_0", 1353, 1, 1024, 1)])
def test_default_chunk_of_batches(cuda, lib, tname, n_slots, q_len, n, hkv):
    """chunk_keys = 0 is the chunk that b200_attn_fixed_chunk names: 512 keys here, few enough partials for the allocation-free entry, even
    where they fill its array to the last value and leave no room for a run plan"""
    import torch
    from p100e_engine_b200 import fast
    g = torch.Generator(device="cuda").manual_seed(n_slots)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    c = fast.kv_alloc(TYPES[tname], n, hkv, D)
    assert fast.kv_append(c, rn(n, hkv, D), rn(n, hkv, D), 0, n)
    assert lib.b200_attn_fixed_chunk(n) == lib.b200_attn_chunk_keys() == 512
    rows, hq = n_slots * q_len, 6 * hkv
    q = rn(rows, hq, D)
    last = torch.randint(q_len - 1, n, (n_slots, 1), generator=g, device=cuda, dtype=torch.int32)
    pos = (last - q_len + 1 + torch.arange(q_len, device=cuda, dtype=torch.int32)).reshape(-1).contiguous()
    outs = [torch.full((rows, hq, D), float("nan"), device=cuda) for _ in range(3)]
    assert fast.attn_decode_slots(q, c, outs[0], None, n_slots, q_len, pos, n, hq, SCALE, 0)
    assert fast.attn_decode_slots(q, c, outs[1], None, n_slots, q_len, pos, n, hq, SCALE, 512)
    assert fast.attn_decode_slots_noalloc(q, c, outs[2], None, n_slots, q_len, pos, n, hq, SCALE, 0) == 0
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert fast.device_status() == 0 and fast.noalloc_device_status() == 0


@pytest.mark.parametrize("chunk", [0, -1])
def test_reservation_covers_the_position_grid(cuda, lib, chunk):
    """after attn_reserve for 8 slots, one slot with -1 and the row entry points are recorded without a call before (a recording cannot allocate)"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv = 4096, 4
    c = fast.kv_alloc(TYPES["q8_0"], n, hkv, D)
    assert fast.kv_fill_random(c, 0, n, 3)
    c.rtab = None
    q, pos = torch.randn(8, 6 * hkv, D, device=cuda), torch.arange(n - 8, n, dtype=torch.int32, device=cuda)
    a, b = torch.zeros_like(q), torch.zeros_like(q)
    assert fast.attn_decode_rows(q, c, torch.zeros_like(q), 8, pos, 6 * hkv, SCALE)          # kernels loaded
    assert fast.attn_decode_slots(q, c, torch.zeros_like(q), None, 1, 4, pos, n, 6 * hkv, SCALE, -1)
    want, want1 = torch.zeros_like(q), torch.zeros_like(q)
    assert fast.attn_decode_rows(q, c, want, 8, pos, 6 * hkv, SCALE)
    assert fast.attn_decode_slots(q, c, want1, None, 1, 4, pos, n, 6 * hkv, SCALE, -1)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    assert fast.attn_reserve(TYPES["q8_0"], 8, 4, n, n, hkv, chunk, s=side)
    with torch.cuda.graph(graph, stream=side):
        assert fast.attn_decode_rows(q, c, a, 8, pos, 6 * hkv, SCALE)
        assert fast.attn_decode_slots(q, c, b, None, 1, 4, pos, n, 6 * hkv, SCALE, -1)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b[:4], want1[:4])


@pytest.mark.parametrize("n_slots,chunks", [(2, 4), (2, 5), (60, 16), (200, 16), (60, 17), (20, 40), (60, 40), (60, 150), (200, 150)])
def test_merge_forms_agree(cuda, lib, n_slots, chunks):
    """the merge runs one, four or sixteen groups of threads per row and head, by partials and grid: the bits of a row are those of the row
    alone (24 heads x 1 row: the smallest grid)"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv = 64 * chunks, 4
    c = fast.kv_alloc(TYPES["q8_0"], n, hkv, D)
    g = torch.Generator(device="cuda").manual_seed(chunks)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    assert fast.kv_append(c, rn(n, hkv, D), rn(n, hkv, D), 0, n)
    q, gate = rn(n_slots, 6 * hkv, D), rn(n_slots, 6 * hkv * D)
    pos = torch.randint(0, n, (n_slots,), generator=g, device=cuda, dtype=torch.int32)
    pos[0], pos[1] = n - 1, -1
    out = torch.full_like(q, float("nan"))
    assert fast.attn_decode_slots(q, c, out, gate, n_slots, 1, pos, n, 6 * hkv, SCALE, 64)
    for i in {0, 1, n_slots // 2, n_slots - 1}:
        one = torch.full_like(q[:1], float("nan"))
        assert fast.attn_decode_slots(q[i:i + 1], c, one, gate[i:i + 1], 1, 1, pos[i:i + 1], n, 6 * hkv, SCALE, 64)
        assert torch.equal(one, out[i:i + 1]), (i, int(pos[i]))
    assert fast.device_status() == 0


@pytest.mark.parametrize("tname", ["q8_0", "f16"])
@pytest.mark.parametrize("longest", [64, 1000, 4096])
def test_short_slots_in_a_long_cache(cuda, lib, tname, longest):
    """room for more chunks than CTAs, slots that fill few of them: a CTA per chunk (64, 1000 keys) or runs of chunks"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv, n_slots = 4096, 1, 300
    c = fast.kv_alloc(TYPES[tname], n, hkv, D)
    g = torch.Generator(device="cuda").manual_seed(longest)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    assert fast.kv_append(c, rn(n, hkv, D), rn(n, hkv, D), 0, n)
    q = rn(n_slots, 6 * hkv, D)
    pos = torch.randint(-1, 64, (n_slots,), generator=g, device=cuda, dtype=torch.int32)
    pos[7:300:19] = longest - 1
    pos[11], pos[299] = -1, longest - 30
    out = torch.full_like(q, float("nan"))
    assert fast.attn_decode_slots(q, c, out, None, n_slots, 1, pos, n, 6 * hkv, SCALE, 64)
    for i in (0, 7, 8, 11, 26, 150, 298, 299):
        one = torch.full_like(q[:1], float("nan"))
        assert fast.attn_decode_slots(q[i:i + 1], c, one, None, 1, 1, pos[i:i + 1], n, 6 * hkv, SCALE, 64)
        assert torch.equal(one, out[i:i + 1]), (i, int(pos[i]))
    assert torch.isfinite(out).all() and fast.device_status() == 0


@pytest.mark.parametrize("tname", ["q8_0", "q4_0", "f16"])
@pytest.mark.parametrize("chunk,n_slots", [(512, 8), (512, 9), (256, 3), (64, 8), (128, 8)])
def test_long_slots_in_fixed_chunks(cuda, lib, tname, chunk, n_slots):
    """more chunks than CTAs (f16: 296 CTAs of one head, q8_0 and q4_0: 888), whole ones and ragged last ones: listed (up to eight slots of a quantised
    cache) or in runs; also through the row entry point, whose chunks grow with the position"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv = 70000, 1
    c = fast.kv_alloc(TYPES[tname], n, hkv, D)
    assert fast.kv_fill_random(c, 0, n, chunk)
    g = torch.Generator(device="cuda").manual_seed(n_slots)
    q = torch.randn(n_slots, 6 * hkv, D, generator=g, device=cuda)
    pos = torch.tensor([n - 1, 65535, 65536, n - 1, -1, 63, 40000, n - 5, n - 1][:n_slots], dtype=torch.int32, device=cuda)
    out, one = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    assert fast.attn_decode_slots(q, c, out, None, n_slots, 1, pos, n, 6 * hkv, SCALE, chunk)
    for i in range(n_slots):
        assert fast.attn_decode_slots(q[i:i + 1], c, one[i:i + 1], None, 1, 1, pos[i:i + 1], n, 6 * hkv, SCALE, chunk)
    torch.cuda.synchronize()
    assert torch.equal(one, out)
    if n_slots == 8:
        assert fast.attn_decode_rows(q, c, out, 8, pos, 6 * hkv, SCALE)
        for i in (0, 1, 2, 5, 6):
            assert fast.attn_decode(q[i:i + 1], c, one[i:i + 1], 1, int(pos[i]), 6 * hkv, SCALE)
            assert torch.equal(one[i], out[i]), i
    assert torch.isfinite(out).all() and fast.device_status() == 0


@pytest.mark.parametrize("n_ctx", [131072, 131328, 229376, 229632])
def test_rows_around_capacities_where_the_grid_changes(cuda, lib, n_ctx):
    """row t of a call == the one-row call where the longest chunk doubles; against an even split of two slots (rounding: the usual bar)"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv = 70000, 1
    c = fast.kv_alloc(TYPES["q4_0"], n_ctx, hkv, D)
    g = torch.Generator(device="cuda").manual_seed(1)
    for p in range(0, n, 10000):
        assert fast.kv_append(c, torch.randn(10000, hkv, D, generator=g, device=cuda), torch.randn(10000, hkv, D, generator=g, device=cuda), p, 10000)
    q = torch.randn(4, 6 * hkv, D, generator=g, device=cuda)
    out, one, two = torch.zeros_like(q), torch.zeros_like(q), torch.zeros(8, 6 * hkv, D, device=cuda)
    for p0 in (n - 4, 65534, 32766):
        assert fast.attn_decode(q, c, out, 4, p0, 6 * hkv, SCALE)
        for t in range(4):
            assert fast.attn_decode(q[t:t + 1], c, one[t:t + 1], 1, p0 + t, 6 * hkv, SCALE)
        pos = torch.arange(p0, p0 + 4, dtype=torch.int32, device=cuda).repeat(2)
        assert fast.attn_decode_slots(torch.cat([q, q]), c, two, None, 2, 4, pos, n, 6 * hkv, SCALE, -1)
        torch.cuda.synchronize()
        assert torch.equal(out, one), p0
        util.check_close(out.cpu().numpy(), two[:4].cpu().numpy(), "n_ctx %d p0 %d" % (n_ctx, p0))
    assert fast.device_status() == 0

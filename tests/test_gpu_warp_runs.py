"""Batched decode of quantised caches on the kernel whose warps walk their keys by themselves (one row of q8_0, one or two of q4_0, even split): ends of
contexts inside a warp's 32 keys, runs that cross slots, small pages, V scales that a plain f16 product would not hold."""
import numpy as np
import pytest

from tests import util
from tests.test_gpu_one_slot import _dequant
from tests.util import D, SCALE, TYPES

pytestmark = pytest.mark.gpu
HKV, HQ = 2, 12


def _batch(cuda, tname, lens, seed, psh=8, v_of=lambda v: v, page_slack=3):
    """paged caches of the given lengths, pages dealt out in turn, all other bytes 0xff (f16 NaN); returns the view and each slot's rows (K, V) in 64 bits"""
    import torch
    from p100e_engine_b200 import fast
    kt, ps = TYPES[tname], 1 << psh
    need = [(n + ps - 1) // ps for n in lens]
    pool = util.PagedPool(kt, sum(need), psh=psh, hkv=HKV, seed=seed)
    tabs = np.stack([pool.take(n, max(need) + page_slack) for n in lens])
    pool_t = torch.full((pool.bytes,), 0xff, dtype=torch.uint8, device=cuda)
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    rows = []
    for s, n in enumerate(lens):
        one = util.dev_cache(pool_t, pool, util.to_dev(tabs[s], cuda))
        flat = fast.kv_alloc(kt, n, HKV, D)
        k, v = rn(n, HKV, D), v_of(rn(n, HKV, D))
        assert fast.kv_append(one, k, v, 0, n) and fast.kv_append(flat, k, v, 0, n)
        torch.cuda.synchronize()
        rows.append((_dequant(flat.k, tname, n), _dequant(flat.v, tname, n)))
    return tabs, pool, pool_t, rows, rn


def _view(cuda, pool, pool_t, tabs, q_len):
    m = tabs.shape[1]
    rtab = np.repeat(np.arange(len(tabs), dtype=np.int32) * m, q_len)
    return util.dev_cache(pool_t, pool, util.to_dev(tabs.reshape(-1), cuda), util.to_dev(rtab, cuda))


def _exact(q, k, v, n_seen):
    """[HQ][D] for one row that sees n_seen keys"""
    import torch
    out = torch.empty(HQ, D, dtype=torch.float64, device=q.device)
    for h in range(HKV):
        s = q[6 * h:6 * h + 6].double() @ k[:n_seen, h].T * SCALE
        out[6 * h:6 * h + 6] = s.softmax(-1) @ v[:n_seen, h]
    return out


def _check(cuda, tname, q_len, lens, seed, psh=8, v_of=lambda v: v, skip=None):
    import torch
    from p100e_engine_b200 import fast
    tabs, pool, pool_t, rows, rn = _batch(cuda, tname, lens, seed, psh, v_of)
    c, q = _view(cuda, pool, pool_t, tabs, q_len), rn(len(lens) * q_len, HQ, D)
    pos = util.to_dev(np.concatenate([np.arange(n - q_len, n) for n in lens]).astype(np.int32), cuda)
    # the bound on the keys is far above the contexts: runs of at least two tiles are possible, so that q4_0 takes the kernel too
    cap = 1 << 18
    out, fixed = (torch.full((len(lens) * q_len, HQ, D), float("nan"), device=cuda) for _ in range(2))
    assert fast.attn_decode_slots(q, c, out, None, len(lens), q_len, pos, cap, HQ, SCALE, -1)
    assert fast.attn_decode_slots(q, c, fixed, None, len(lens), q_len, pos, cap, HQ, SCALE, 4096)
    torch.cuda.synchronize()
    assert fast.device_status() == 0
    err = np.zeros(2)
    for i, p in enumerate(pos.tolist()):
        ref = _exact(q[i], *rows[i // q_len], p + 1)
        for j, o in enumerate((out, fixed)):
            err[j] += float((o[i].double() - ref).norm() / ref.norm()) / len(pos)
            # three f16 roundings (Q, P, P d) of 2^-12 rms at most each; single values against the row's largest
            assert float((o[i].double() - ref).abs().max() / ref.abs().max()) < 4 * 2.0 ** -11, (i, j)
    return err


@pytest.mark.parametrize("tname,q_len", [("q8_0", 1), ("q4_0", 1), ("q4_0", 2)])
def test_ragged_contexts_and_runs_across_slots(cuda, lib, tname, q_len):
    lens = [2, 31, 32, 33, 34, 63, 64, 65, 95, 96, 97, 129, 255, 257, 513, 1000, 8191, 20011]
    err = _check(cuda, tname, q_len, lens, 3 + q_len)
    print("%s q_len %d: %.3e, fixed chunks %.3e" % (tname, q_len, *err))
    assert err[0] <= 1.02 * err[1]


@pytest.mark.parametrize("tname,q_len", [("q8_0", 1), ("q4_0", 2)])
@pytest.mark.parametrize("psh", [3, 5, 6])
def test_small_pages(cuda, lib, tname, q_len, psh):
    _check(cuda, tname, q_len, [70, 301, 2500], 9, psh)


@pytest.mark.parametrize("tname,q_len", [("q8_0", 1), ("q4_0", 1), ("q4_0", 2)])
@pytest.mark.parametrize("what", ["all", "late", "one block"])
def test_large_values(cuda, lib, tname, q_len, what):
    """V of up to 30000: all of it, from key 500 on, or one block of 32 dims beside blocks a million times smaller"""
    import torch

    def v_of(v):
        v = v.clone()
        if what == "all":
            v *= 6000.0
        elif what == "late":
            v[500:] *= 300.0
            v[700:] *= 20.0
        else:
            v *= 0.01
            v[:, :, 64:96] *= 6e5
        return v.clamp(-30000.0, 30000.0)

    err = _check(cuda, tname, q_len, [300, 600, 1200, 3000], 21, v_of=v_of)
    print("%s q_len %d %s: %.3e, fixed chunks %.3e" % (tname, q_len, what, *err))
    assert err[0] <= 1.05 * err[1]
    if what != "one block":
        return
    # the small blocks by themselves
    from p100e_engine_b200 import fast
    lens = [600, 3000]
    tabs, pool, pool_t, rows, rn = _batch(cuda, tname, lens, 22, v_of=v_of)
    q = rn(2 * q_len, HQ, D)
    pos = util.to_dev(np.concatenate([np.arange(n - q_len, n) for n in lens]).astype(np.int32), cuda)
    out = torch.full((2 * q_len, HQ, D), float("nan"), device=cuda)
    assert fast.attn_decode_slots(q, _view(cuda, pool, pool_t, tabs, q_len), out, None, 2, q_len, pos, 1 << 18, HQ, SCALE, -1)
    torch.cuda.synchronize()
    for i, p in enumerate(pos.tolist()):
        ref = _exact(q[i], *rows[i // q_len], p + 1)[:, 128:]
        assert float((out[i, :, 128:].double() - ref).norm() / ref.norm()) < 3 ** 0.5 * 2.0 ** -11


@pytest.mark.parametrize("tname,q_len", [("q8_0", 1), ("q4_0", 1)])
def test_an_infinite_scale_stays_in_its_block(cuda, lib, tname, q_len):
    import torch
    from p100e_engine_b200 import fast
    tabs, pool, pool_t, rows, rn = _batch(cuda, tname, [200, 900], 5)
    page = int(tabs[1][1])   # keys 256 .. of slot 1: block 3 of head 0 of key 300 gets an infinite V scale
    off = pool.voff + page * pool.pstride + (300 - 256) * pool.rowb + (2 * 3 if tname == "q8_0" else 18 * 3)
    pool_t[off:off + 2] = torch.tensor([0x00, 0x7c], dtype=torch.uint8, device=cuda)
    q, pos = rn(2, HQ, D), util.to_dev(np.array([199, 899], np.int32), cuda)
    out = torch.full((2, HQ, D), float("nan"), device=cuda)
    assert fast.attn_decode_slots(q, _view(cuda, pool, pool_t, tabs, 1), out, None, 2, 1, pos, 1 << 18, HQ, SCALE, -1)
    torch.cuda.synchronize()
    assert not torch.isfinite(out[1, :6, 96:128]).any()
    for i, n in enumerate((200, 900)):
        ref = _exact(q[i], *rows[i], n)
        keep = torch.ones(HQ, D, dtype=torch.bool, device=cuda)
        if i:
            keep[:6, 96:128] = False
        assert torch.isfinite(out[i][keep]).all()
        assert float((out[i].double() - ref)[keep].norm() / ref[keep].norm()) < 3 ** 0.5 * 2.0 ** -11


def test_allocation_free_call_takes_as_many_slots_as_its_array_ever_held(cuda, lib):
    """450 slots of q4_0 with four heads: partials of decode_part_k's runs fit the built-in array, those of the longer list of runs would not"""
    import torch
    from p100e_engine_b200 import fast
    n, hkv, hq = 450, 4, 24
    c = fast.kv_alloc(TYPES["q4_0"], 4096, hkv, D)
    assert fast.kv_fill_random(c, 0, 4096, 2)
    q = torch.randn(n, hq, D, device=cuda)
    pos = torch.arange(n, dtype=torch.int32, device=cuda) * 9
    a, b = (torch.full_like(q, float("nan")) for _ in range(2))
    assert fast.attn_decode_slots_noalloc(q, c, a, None, n, 1, pos, 4096, hq, SCALE, -1) == 0
    assert fast.attn_decode_slots(q, c, b, None, n, 1, pos, 4096, hq, SCALE, -1)
    torch.cuda.synchronize()
    assert float((a - b).norm() / b.norm()) < 3 ** 0.5 * 2.0 ** -11

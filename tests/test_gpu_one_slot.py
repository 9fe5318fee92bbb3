"""One slot through the batched entry point with chunk_keys = -1: no further from 64-bit attention than equal chunks on the kernel that keeps K
integer."""
import numpy as np
import pytest

from tests.util import D, SCALE, TYPES

pytestmark = pytest.mark.gpu
HKV, HQ = 2, 12


def _dequant(raw, tname, n):
    """stored rows in 64 bits [n][Hkv][D]"""
    import torch
    if tname == "f16":
        return raw.view(torch.float16).view(n, HKV, D).double()
    if tname == "q8_0":
        r = raw.view(n, HKV, 272)
        return (r[..., 16:].contiguous().view(torch.int8).double().view(n, HKV, 8, 32) *
                r[..., :16].contiguous().view(torch.float16).double()[..., None]).view(n, HKV, D)
    r = raw.view(n, HKV, 8, 18)
    b = r[..., 2:].to(torch.int32)
    return (torch.cat([(b & 15) - 8, (b >> 4) - 8], -1).double() * r[..., :2].contiguous().view(torch.float16).double()).view(n, HKV, D)


def _attention64(q, c, tname, n, p0):
    import torch
    k, v = _dequant(c.k, tname, n), _dequant(c.v, tname, n)
    T, out = q.shape[0], torch.empty(q.shape, dtype=torch.float64, device=q.device)
    hidden = torch.arange(n, device=q.device)[None, None] > (p0 + torch.arange(T, device=q.device))[:, None, None]
    for h in range(HKV):
        s = torch.einsum("tgd,nd->tgn", q[:, 6 * h:6 * h + 6].double(), k[:, h]) * SCALE
        out[:, 6 * h:6 * h + 6] = torch.einsum("tgn,nd->tgd", s.masked_fill(hidden, float("-inf")).softmax(-1), v[:, h])
    return out


@pytest.mark.parametrize("tname", ["q8_0", "f16", "q4_0"])
@pytest.mark.parametrize("n", [100, 5000, 30011, 65536, 70001])
@pytest.mark.parametrize("T", [1, 2, 4])
def test_one_slot_keeps_the_precision_of_fixed_chunks(cuda, lib, tname, n, T):
    import torch
    from p100e_engine_b200 import fast
    c = fast.kv_alloc(TYPES[tname], n, HKV, D)
    g = torch.Generator(device="cuda").manual_seed(n + T)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    assert fast.kv_append(c, rn(n, HKV, D), rn(n, HKV, D), 0, n)
    p0 = n - T
    pos = torch.arange(p0, n, dtype=torch.int32, device=cuda)
    err = np.zeros(2)
    for _ in range(3):
        q = rn(T, HQ, D)
        one, fixed = (torch.full((T, HQ, D), float("nan"), device=cuda) for _ in range(2))
        assert fast.attn_decode_slots(q, c, one, None, 1, T, pos, n, HQ, SCALE, -1)
        assert fast.attn_decode_slots(q, c, fixed, None, 1, T, pos, n, HQ, SCALE, 256)
        torch.cuda.synchronize()
        ref = _attention64(q, c, tname, n, p0)
        err += [float((o.double() - ref).norm() / ref.norm()) for o in (one, fixed)]
    print("%s n=%d T=%d: one slot %.3e, chunks of 256 %.3e" % (tname, n, T, *(err / 3)))
    assert fast.device_status() == 0
    # chunks that are nowhere longer, so that the roundings of P are those of reference maxima that are nowhere further away
    assert err[0] <= 1.002 * err[1]


@pytest.mark.parametrize("q_len", [2, 4])
def test_verify_kernel_error(cuda, lib, q_len):
    """two slots of the same rows on the verify kernel (K rounded to f16) and on the mma.sync kernel (K integer): both within the f16 bound"""
    import torch
    from p100e_engine_b200 import fast
    n = 30011
    c = fast.kv_alloc(TYPES["q8_0"], n, HKV, D)
    g = torch.Generator(device="cuda").manual_seed(n)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    assert fast.kv_append(c, rn(n, HKV, D), rn(n, HKV, D), 0, n)
    q = rn(2 * q_len, HQ, D)
    pos = torch.arange(n - q_len, n, dtype=torch.int32, device=cuda).repeat(2)
    ref = torch.cat([_attention64(x, c, "q8_0", n, n - q_len) for x in (q[:q_len], q[q_len:])])
    err = []
    try:
        for tc in (1, 0):
            lib.b200_attn_dec_set_tc(tc)
            out = torch.full((2 * q_len, HQ, D), float("nan"), device=cuda)
            assert fast.attn_decode_slots(q, c, out, None, 2, q_len, pos, n, HQ, SCALE, -1)
            torch.cuda.synchronize()
            err.append(float((out.double() - ref).norm() / ref.norm()))
    finally:
        lib.b200_attn_dec_set_tc(-1)
    print("q_len %d: verify kernel %.3e, mma.sync kernel %.3e" % (q_len, *err))
    assert fast.device_status() == 0
    # three f16 roundings (K, P, V scaled) of 2^-12 rms at most each, sums over independent errors
    assert max(err) < 3 ** 0.5 * 2.0 ** -11


@pytest.mark.parametrize("hkv", [1, 2, 8])
def test_one_slot_after_a_reservation(cuda, lib, hkv):
    """attn_reserve(-1) covers one slot of any length up to its max_n: a call that allocates cannot be recorded"""
    import torch
    from p100e_engine_b200 import fast
    cap = 140000
    c = fast.kv_alloc(TYPES["q4_0"], cap, hkv, D)
    assert fast.kv_fill_random(c, 0, cap, 2)
    q = torch.randn(4, 6 * hkv, D, device=cuda)
    lens = [1, 4096, 30000, 37891, 65536, 65537, 75800, 75900, 131072, cap]
    want = []
    for n in lens:
        pos = torch.full((4,), n - 1, dtype=torch.int32, device=cuda)
        want.append(torch.full_like(q, float("nan")))
        assert fast.attn_decode_slots(q, c, want[-1], None, 1, 4, pos, n, 6 * hkv, SCALE, -1)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert fast.attn_reserve(TYPES["q4_0"], 2, 4, cap, cap, hkv, -1, s=side)
    for n, w in zip(lens, want):
        pos = torch.full((4,), n - 1, dtype=torch.int32, device=cuda)
        out, graph = torch.full_like(q, float("nan")), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            assert fast.attn_decode_slots(q, c, out, None, 1, 4, pos, n, 6 * hkv, SCALE, -1)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, w), n


@pytest.mark.parametrize("q_len", [2, 4])
@pytest.mark.parametrize("n", [128, 129, 300, 2049, 20011])
@pytest.mark.parametrize("trend", ["rising", "falling", "one peak", "large q"])
def test_one_slot_verify_with_scores_that_drift(cuda, lib, q_len, n, trend):
    """scores whose maxima move by hundreds over the context, up, down, or at one key only, and query sums beyond f16 times 128: the reference maxima of
    the exact verify form follow without leaving f16 and fp32"""
    import torch
    from p100e_engine_b200 import fast
    c = fast.kv_alloc(TYPES["q8_0"], n, HKV, D)
    g = torch.Generator(device="cuda").manual_seed(n + q_len)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    k, q = rn(n, HKV, D), rn(q_len, HQ, D)
    along = q[0, ::6][None] / 16.0        # a direction that the first head of each group sees
    ramp = torch.linspace(0.0, 40.0, n, device=cuda)[:, None, None]
    if trend == "rising":
        k += ramp * along
    elif trend == "falling":
        k += (40.0 - ramp) * along
    elif trend == "one peak":
        k[n // 2] += 60.0 * along[0]
    else:
        q = q * 40.0 + 300.0
    assert fast.kv_append(c, k, rn(n, HKV, D), 0, n)
    pos = torch.arange(n - q_len, n, dtype=torch.int32, device=cuda)
    one, fixed = (torch.full((q_len, HQ, D), float("nan"), device=cuda) for _ in range(2))
    assert fast.attn_decode_slots(q, c, one, None, 1, q_len, pos, n, HQ, SCALE, -1)
    assert fast.attn_decode_slots(q, c, fixed, None, 1, q_len, pos, n, HQ, SCALE, 256)
    torch.cuda.synchronize()
    assert fast.device_status() == 0
    ref = _attention64(q, c, "q8_0", n, n - q_len)
    err = [float((o.double() - ref).norm() / ref.norm()) for o in (one, fixed)]
    print("%s n=%d q_len=%d: one slot %.3e, chunks of 256 %.3e" % (trend, n, q_len, *err))
    # the rounding of Q to f16 (2^-12 rms of scores of up to some hundreds) is common to both; beyond it three roundings of 2^-12 rms
    assert err[0] <= 1.05 * err[1] + 3 ** 0.5 * 2.0 ** -12

"""The merge of a row's partials: numbers of partials around one per summation stream, around the partials that are fetched before the row's
length is known, and scratch whose unused partials hold NaN."""
import pytest

from oracle import orc
from tests import util
from tests.util import D, HKV, HQ, SCALE, TYPES
from tests.test_gpu_chunk_grid import _paged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 5, 15, 16, 17, 63, 64, 65, 129])
def test_merge_of_n_partials(cuda, lib, parts):
    """chunks of 64 keys; the bound on the keys says exactly what the row has, or 140 chunks, of which the rest holds NaN from a call before;
    and the row in a batch large enough for one group of threads per head.  All bitwise equal, and close to the oracle (f16 operands, fp32 sums:
    the usual bar)."""
    import torch
    from p100e_engine_b200 import fast
    cap, n = 140 * 64, 64 * parts - 3
    c, hc, _keep = _paged(cuda, TYPES["q8_0"], cap, 3)
    q = util.to_dev(util.rng_normal(4, (1, HQ, D)), cuda)
    gate = util.to_dev(util.rng_normal(5, (1, HQ * D)), cuda)
    pos, last = (torch.tensor([p], dtype=torch.int32, device=cuda) for p in (n - 1, cap - 1))
    a, b, junk = (torch.empty(1, HQ, D, device=cuda) for _ in range(3))
    assert fast.attn_decode_slots(torch.full_like(q, float("nan")), c, junk, None, 1, 1, last, cap, HQ, SCALE, 64)
    assert fast.attn_decode_slots(q, c, a, gate, 1, 1, pos, cap, HQ, SCALE, 64)
    assert fast.attn_decode_slots(q, c, b, gate, 1, 1, pos, n, HQ, SCALE, 64)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
    m = 60
    many = torch.empty(m, HQ, D, device=cuda)
    rows = torch.zeros(m, dtype=torch.int32, device=cuda)
    cm = fast.kv_cache(c.type, c.n_ctx, c.Hkv, c.D, c.k, c.v, c.pt, rows, c.psh, c.pstride)
    assert fast.attn_decode_slots(q.repeat(m, 1, 1), cm, many, gate.repeat(m, 1), m, 1, pos.repeat(m), n, HQ, SCALE, 64)
    torch.cuda.synchronize()
    assert fast.device_status() == 0
    assert all(torch.equal(many[i], a[0]) for i in range(m))
    ref = orc.attention(q.cpu().numpy(), hc, 1, HQ, SCALE, pos=pos.cpu().numpy(), gate=gate.cpu().numpy())
    util.check_close(a.cpu().numpy(), ref, "%d partials" % parts)

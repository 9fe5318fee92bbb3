"""The step descriptor's upload: one copy through the unused rows of a small descriptor, one 2D copy of a large one.  Rows that a step does not have keep what
an earlier step put there, as in a replayed recording that covers more rows than the step."""
import numpy as np
import pytest

from tests.util import TYPES

pytestmark = pytest.mark.gpu


class _Ints:
    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (address, False), "version": 3}


@pytest.mark.parametrize("max_rows", [8, 5461 + 8, 5462 + 9, 40000])   # 8 rows used: no gap worth a word, gaps of 64 KiB, just above, far above
def test_step_arrays(cuda, lib, max_rows):
    import torch
    from p100e_engine_b200 import lib as L
    from p100e_engine_b200.pool import Pool
    pool = Pool(TYPES["q8_0"], 1, 1, 64, 8, 256, max_slots=8, max_pages=8, max_rows=max_rows, device=0)
    dev = [torch.as_tensor(_Ints(a, 8), device=cuda) for a in pool.step_arrays()]
    held = np.zeros((4, 8), np.int32)
    rng = np.random.default_rng(max_rows)
    for slots, q_len in ([0, 1, 2, 3, 4, 5, 6, 7], 1), ([3, 1], 2), ([5], 1), ([2, 7, 0], 2), ([4], 3), ([6, 5], 4):
        n_past = rng.integers(0, 1000, len(slots)).astype(np.int32)
        L.check("pool_step", pool.step(np.array(slots, np.int32), n_past, q_len))
        torch.cuda.synchronize()
        rows = len(slots) * q_len
        pos = (n_past[:, None] + np.arange(q_len)).reshape(-1)
        held[:3, :rows] = pos
        held[3, :rows] = np.repeat(np.array(slots) * 8, q_len)
        assert np.array_equal(np.stack([d.cpu().numpy() for d in dev]), held)

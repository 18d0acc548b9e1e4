"""The sort's look-back reads eight earlier partitions a step: sorts whose
partition counts (of 3072 keys) lie around two and four steps, and whole waves
of partitions that publish at once, order stably and lose nothing."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PARTITION = 3072


@pytest.mark.parametrize("with_values", [False, True], ids=["keys", "values"])
@pytest.mark.parametrize("count", [16 * PARTITION, 16 * PARTITION + 1, 17 * PARTITION, 18 * PARTITION + 1,
                                   33 * PARTITION - 1, 33 * PARTITION + 1, 592 * PARTITION, 700 * PARTITION + 5])
def test_sorts_around_a_look_back_step(rasterizer, count, with_values):
    rng = np.random.default_rng(count)
    keys = rng.integers(0, 1 << 20, count, dtype=np.uint64) | (np.uint64(7) << np.uint64(40))
    kt = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    vt = torch.arange(count, dtype=torch.int32, device="cuda") if with_values else None
    rasterizer.radix_sort(kt, vt, 16)
    order = np.argsort(keys & np.uint64(0xFFFF), kind="stable")
    assert np.array_equal(kt.cpu().numpy().view(np.uint64), keys[order])
    if with_values:
        assert np.array_equal(vt.cpu().numpy(), order.astype(np.int32))

"""The most components whose labels fit 32-bit integers: 2^31 of them are returned,
one more is an error."""
from __future__ import annotations

import os

import numpy as np
import pytest

import knappnet_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1])
def test_the_largest_label(more):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("less than 80 GB of device memory")
    if os.sysconf("SC_AVPHYS_PAGES") * os.sysconf("SC_PAGE_SIZE") < 24 << 30:
        pytest.skip("less than 24 GB of host memory")
    pairs = 1 << 20
    n = (1 << 31) + pairs + more
    a = np.arange(pairs, dtype=np.int64) * 2048
    g = K.Graph(n, a, a + 1, None, False)
    if more:
        with pytest.raises(K.EngineError, match="component count .* is too large"):
            g.components(strong=False)
    else:
        label, count = g.components(strong=False)
        assert count == 1 << 31
        assert label[-1] == (1 << 31) - 1 and label[0] == label[1] == 0 and label[2] == 1
    del g
    K.device_sync()

"""Device memory the library keeps between calls: bounded, given back, and
safe for handles that one thread builds and another uses or frees."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import knappnet_b200 as K

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KEPT = 512 << 20


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_is_bounded_and_given_back():
    K.generate_rmat(10, 8, seed=1).close()  # context, kernels and pool exist
    K.device_sync()
    before = free_bytes()
    g = K.generate_rmat(20, 16, seed=3, clean=True, lognormal=True)  # over 1 GB while it is built
    g.pagerank(weighted=True)
    g.close()
    slack = 64 << 20  # what the driver rounds and kernels' local memory add
    assert before - free_bytes() <= KEPT + slack
    K.device_sync()
    assert before - free_bytes() <= slack


def test_threads_share_and_free_each_others_handles():
    """Every thread builds graphs of its own sizes; another thread solves on
    them and frees them while the first builds on in the memory that comes
    free. Scores equal those of a quiet solve, bit for bit."""
    rng = np.random.default_rng(5)
    made = []
    for k in range(6):
        n = 3000 + 700 * k
        made.append((n, rng.integers(0, n, 9 * n), rng.integers(0, n, 9 * n),
                     rng.lognormal(size=9 * n)))
    alone = [K.Graph(*t, True).pagerank(weighted=True, precision=K.PREC_MIXED) for t in made]
    box, errors = [], []
    ready = threading.Condition()

    def build():
        for r in range(5):
            for k, t in enumerate(made):
                with ready:
                    box.append((k, K.Graph(*t, True)))
                    ready.notify_all()

    def use(count):
        for _ in range(count):
            with ready:
                while not box:
                    ready.wait(30)
                k, g = box.pop()
            try:
                got = g.pagerank(weighted=True, precision=K.PREC_MIXED)
                if not np.array_equal(got, alone[k]):
                    errors.append(k)
            except Exception as e:  # noqa: BLE001
                errors.append(e)
            g.close()

    ts = [threading.Thread(target=build) for _ in range(2)]
    ts += [threading.Thread(target=use, args=(20,)) for _ in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(60)
    assert not errors and not box

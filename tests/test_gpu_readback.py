"""Reads of whole states: the small path, the pinned slots with one and with several threads, and the pool."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from celeris_b200 import cases

pytestmark = pytest.mark.gpu


def _waves(shape, seed):
    rng = np.random.default_rng(seed)
    s = rng.standard_normal(shape + (4,)).astype(np.float32)
    s[..., 3] = 0
    return s


# 16-byte texels: under 1 MB, just over it, a ragged last slot, several threads
@pytest.mark.parametrize("nx, ny", [(2, 2), (252, 252), (253, 254), (300, 601), (1021, 777)])
@pytest.mark.parametrize("form", ["plain", "fused", "mixed"])
def test_state_reads_back_what_was_set(celeris, nx, ny, form):
    p, z, _, _ = cases.small_case(nx, ny, "solid")
    eng = celeris.Engine(p, z, form)
    s = _waves(eng.shape, nx)
    eng.set_state(s)
    for _ in range(2):
        np.testing.assert_array_equal(eng.state(), s)


def test_reads_from_several_threads(celeris):
    """Handles of their own in threads of their own share the pool of pinned blocks."""
    engines, want, got = [], [], [None] * 7
    for k in range(7):
        p, z, _, _ = cases.small_case(400 + k, 500, "solid")
        engines.append(celeris.Engine(p, z, "mixed"))
        want.append(_waves(engines[-1].shape, k))
        engines[-1].set_state(want[-1])

    def read(k):
        for _ in range(3):
            got[k] = engines[k].state()

    threads = [threading.Thread(target=read, args=(k,)) for k in range(7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)

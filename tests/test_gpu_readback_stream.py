"""Reads of an engine on the per-thread default stream: they wait for the steps that the thread has queued."""
from __future__ import annotations

import numpy as np
import pytest

from celeris_b200 import cases

pytestmark = pytest.mark.gpu

PER_THREAD = 2   # the handle of the per-thread default stream


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_reads_follow_the_steps(celeris, form):
    p, z, _, _ = cases.small_case(1100, 700, "sponge")   # 12 MB: a read of several threads
    ref, eng = celeris.Engine(p, z, form), celeris.Engine(p, z, form)
    eng.set_stream(PER_THREAD)
    for _ in range(3):
        ref.physical_steps(20)
        eng.physical_steps(20)
        np.testing.assert_array_equal(eng.state(), ref.state())

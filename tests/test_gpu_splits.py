"""Splits of the stencil's work: strip heights bound by the tuning and shortened for small batches."""
from __future__ import annotations

import numpy as np
import pytest

from celeris_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(5, 9)], [(95, 8), (94, 7)], [(189, 65), (40, 130)], [(300, 33), (2, 2), (97, 71)]])
@pytest.mark.parametrize("rows", [1, 2])
def test_strip_heights_do_not_change_results(celeris, sizes, rows):
    """Strips of 8 rows, of odd heights and of whole members give the same bits as the default."""
    members = [cases.small_case(nx, ny, k, seed=i)[:2] for i, ((nx, ny), k) in enumerate(zip(sizes, ("mixed", "sponge", "solid")))]

    def states(height):
        b = celeris.Batch(members, "mixed")
        b.set_stencil_rows(rows)
        if height:
            b.set_tuning(0, height, 0)
        b.step(12)
        return [b.state(i) for i in range(len(members))] + [b.aux(i) for i in range(len(members))]

    ref = states(0)
    for h in (8, 9, 33, 1024):
        for a, r in zip(states(h), ref):
            np.testing.assert_array_equal(a, r)

"""The plain form's solves on tall domains: a CTA per column where few columns are tall, bands of four otherwise."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import cases

pytestmark = pytest.mark.gpu


# both sides of the rule's lines (4096 rows, 296 columns), a power of two and its neighbours, the tallest domain
# there is, and four columns' levels that do not fit in shared memory
@pytest.mark.parametrize("nx, ny", [(2, 4095), (2, 4096), (5, 4097), (7, 8191), (296, 4099), (297, 4099), (3, 32768), (301, 12901)])
def test_tall_domains_bit_for_bit(celeris, nx, ny):
    p, z, bnx, bny = cases.small_case(nx, ny, "sponge", correction_steps=1)
    z = np.minimum(z, 1.0).astype(np.float32)
    ref, eng = O.Oracle(p, z, bnx, bny, "f32"), celeris.Engine(p, z, "plain")
    ref.physical_steps(3)
    eng.physical_steps(3)
    assert np.array_equal(eng.state()[..., :3].astype(np.float64), ref.state()[..., :3])

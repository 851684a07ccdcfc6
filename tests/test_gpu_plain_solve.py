"""The plain form's one-launch cyclic reduction, statistics and boundaries at the sizes where they can go wrong."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import cases

pytestmark = pytest.mark.gpu

# rows of one to several levels, ends of the warp's and the CTA's share, columns past a band of four,
# rows and columns whose levels do not fit in shared memory
SIZES = [(2, 3), (31, 17), (32, 33), (65, 34), (67, 129), (512, 63), (515, 8), (26001, 3), (5, 13001)]


@pytest.mark.parametrize("nx, ny", SIZES)
@pytest.mark.parametrize("kind", ["sponge", "solid"])
def test_plain_sizes_bit_for_bit(celeris, nx, ny, kind):
    if max(nx, ny) > 10000 and kind == "solid":
        pytest.skip("the long systems run once")
    p, z, bnx, bny = cases.small_case(nx, ny, kind, correction_steps=1)
    z = np.minimum(z, 1.0).astype(np.float32)
    ref, eng = O.Oracle(p, z, bnx, bny, "f32"), celeris.Engine(p, z, "plain")
    ref.physical_steps(6)
    eng.physical_steps(6)
    assert np.array_equal(eng.state()[..., :3].astype(np.float64), ref.state()[..., :3])
    # the totals against their definition in FP64: the volume up to the order of its sum; the mass up to
    # the rounding of a depth and of the 15 single-precision additions of a block, 16 * 2**-24 < 1e-6
    got, st, ba = eng.reset_timestep(), eng.state()[2:-2, 2:-2], eng.bottom()[2:-2, 2:-2, 2]
    depth = np.maximum(0.0, st[..., 0].astype(np.float64) - ba)
    blocks = depth[:ny // 4 * 4, :nx // 4 * 4]
    f = np.float32
    area = float(f(p.width) / f(nx - 1) * f(p.length) / f(ny - 1))
    assert got["mass_full"] == pytest.approx(depth.sum(), rel=1e-12)
    assert got["mass"] == pytest.approx(blocks.sum() * 1000 * area, rel=1e-6)
    assert got["max_depth"] == (float(np.maximum(f(0), st[:ny // 4 * 4, :nx // 4 * 4, 0] - ba[:ny // 4 * 4, :nx // 4 * 4]).max())
                                if blocks.size else 0.0)
    assert got["health"] == 0


def test_faces_of_the_state_before_a_solitary_wave(celeris):
    """The pass after addSolitaryWave takes the faces (and the record) of the state before it, however many
    waves were added; a wave before the first pass, a new state and later passes rebuild them."""
    p, z, bnx, bny = cases.small_case(67, 45, "sponge", correction_steps=1)
    ref, eng = O.Oracle(p, z, bnx, bny, "f32"), celeris.Engine(p, z, "plain")

    def both(f):
        f(ref)
        f(eng)

    def same():
        assert np.array_equal(eng.state()[..., :3].astype(np.float64), ref.state()[..., :3])
        np.testing.assert_allclose(eng.aux()[2:-2, 2:-2, 0], ref.aux()[2:-2, 2:-2, 0], rtol=1e-6, atol=1e-7)

    both(lambda e: e.add_solitary_wave(0.1, 10.0, 20.0, 10.0))     # before the first pass
    both(lambda e: e.physical_steps(4))
    same()
    both(lambda e: e.add_solitary_wave(0.2, 30.0, 25.0, 12.0))
    both(lambda e: e.add_solitary_wave(0.1, -40.0, 35.0, 20.0))
    both(lambda e: e.physical_steps(3))
    same()
    both(lambda e: e.add_solitary_wave(0.05, 0.0, 30.0, 20.0))
    s = eng.state()
    eng.set_state(s)
    ref.set_state(s.astype(np.float64))
    both(lambda e: e.physical_steps(3))
    same()

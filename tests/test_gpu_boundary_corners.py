"""Wave-makers and recorded levels that meet other sides in a corner, in the fused forms' one launch."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import abi, cases
from util import field_errors, rel_ok

pytestmark = pytest.mark.gpu

S, G, W, I, U = (abi.CEL_BC_SOLID, abi.CEL_BC_SPONGE, abi.CEL_BC_SINEWAVE, abi.CEL_BC_IRREGULAR, abi.CEL_BC_UTS)
# west, east, south, north as (type, width)
MIXES = [
    ((I, 2), (G, 9), (G, 6), (S, 2)),
    ((S, 2), (G, 150), (S, 2), (I, 3)),       # a wave-maker along a sponge of many work items
    ((G, 5), (I, 2), (U, 2), (G, 33)),
    ((U, 3), (S, 3), (I, 2), (U, 2)),
    ((W, 2), (U, 2), (S, 2), (I, 2)),
]


@pytest.mark.parametrize("sides", MIXES)
@pytest.mark.parametrize("form", ["fused", "mixed"])
def test_corners_against_the_oracle(celeris, sides, form):
    """Every strip texel after some passes against the FP64 oracle, within the parity tests' 2e-3 of the fields."""
    nx, ny = 200, 60
    p, z, bnx, bny = cases.small_case(nx, ny, "mixed")
    p.n_solitons = 0
    z = np.minimum(z, 1.0).astype(np.float32)
    rng = np.random.default_rng(5)
    t = np.arange(40) * 0.5
    table = np.stack([t, 0.1 * np.sin(t), 0.2 * np.cos(t), 0.05 * np.sin(0.7 * t)], axis=1)
    keep = []
    for name, (kind, width) in zip(("west", "east", "south", "north"), sides):
        side = getattr(p, name)
        side.type, side.width, side.sea_level = kind, width, 0.0
        side.amplitude, side.period, side.theta = 0.2, 5.0, 0.3
        if kind == I:
            comps = cases.jonswap_components(40, 0.3, 6.0, 3.3, rng)   # more components than a warp has lanes
            side.n_waves = len(comps)
            for i, c in enumerate(comps):
                for k in range(4):
                    side.waves[i][k] = float(c[k])
        if kind == U:
            keep += cases.attach_uts(p, name, table)
    ref, b = O.Oracle(p, z, bnx, bny, "f64"), celeris.Batch([(p, z)], form)
    ref.physical_steps(25)
    b.step(25)
    got, want = b.state(0).astype(np.float64), ref.state()
    assert rel_ok(field_errors(got, want), 2e-3, 1e-6)
    scale = np.abs(want[2:-2, 2:-2]).max(axis=(0, 1))
    for q in range(3):
        assert np.abs(got[..., q] - want[..., q]).max() <= 2e-3 * max(scale[q], scale[1:3].max() if q else scale[0]) + 1e-6

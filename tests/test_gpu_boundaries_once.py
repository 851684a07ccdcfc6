"""The fused forms' four sides in one launch, where sides meet and where they cannot run together."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import abi, cases
from util import field_errors, rel_ok

pytestmark = pytest.mark.gpu


def _case(nx, ny, sides, seed=0):
    """sides: west, east, south, north as (type, width)"""
    p, z, bnx, bny = cases.small_case(nx, ny, "mixed", seed=seed)
    p.n_solitons = 0
    for side, (kind, width) in zip((p.west, p.east, p.south, p.north), sides):
        side.type, side.width, side.sea_level = kind, width, 0.0
        side.amplitude, side.period, side.theta = 0.2, 5.0, 0.3
    return p, z, bnx, bny


S, G, W = abi.CEL_BC_SOLID, abi.CEL_BC_SPONGE, abi.CEL_BC_SINEWAVE
MIXES = [
    ((W, 2), (G, 7), (S, 2), (S, 2)),
    ((G, 5), (G, 40), (G, 9), (G, 3)),        # sponges meeting in every corner, one wider than a work item
    ((S, 1), (S, 3), (S, 2), (S, 3)),         # walls of the widths that read outside their own strip
    ((S, 2), (W, 2), (G, 6), (W, 3)),
    ((S, 3), (S, 4), (G, 4), (S, 2)),         # walls that read their own strip: one launch per side
    ((G, 2), (S, 2), (W, 0), (S, 2)),         # a side without texels
]


@pytest.mark.parametrize("sides", MIXES)
@pytest.mark.parametrize("nx, ny", [(75, 61), (52, 9)])
@pytest.mark.parametrize("form", ["fused", "mixed"])
def test_sides_against_the_oracle(celeris, sides, nx, ny, form):
    """Ghost texels included: every strip texel after some passes against the FP64 oracle.  The strips
    are pointwise in the interior's values, so they carry the fields' tolerance of the parity tests."""
    p, z, bnx, bny = _case(nx, ny, sides)
    ref, b = O.Oracle(p, z, bnx, bny, "f64"), celeris.Batch([(p, z)], form)
    ref.physical_steps(25)
    b.step(25)
    got, want = b.state(0).astype(np.float64), ref.state()
    assert rel_ok(field_errors(got, want), 2e-3, 1e-6)
    scale = np.abs(want[2:-2, 2:-2]).max(axis=(0, 1))
    for q in range(3):
        assert np.abs(got[..., q] - want[..., q]).max() <= 2e-3 * max(scale[q], scale[1:3].max() if q else scale[0]) + 1e-6


def test_one_batch_holds_both_kinds_of_member(celeris):
    members = [_case(60 + 9 * k, 40 + 5 * k, sides, seed=k)[:2] for k, sides in enumerate(MIXES)]
    b = celeris.Batch(members, "mixed", lanes=1)
    b.use_graph(True)
    b.step(20)
    for i, (p, z) in enumerate(members):
        e = celeris.Engine(p, z, "mixed")
        e.physical_steps(20)
        np.testing.assert_array_equal(b.state(i), e.state())

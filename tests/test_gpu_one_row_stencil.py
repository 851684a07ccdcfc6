"""The one-row stencil, selected: against the FP64 oracle and the paired-row stencil (the default)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import cases
from util import eta_rms, field_errors, rel_ok

pytestmark = pytest.mark.gpu


def _batch(celeris, members, form, rows):
    b = celeris.Batch(members, form)
    b.set_stencil_rows(rows)
    assert b.stencil_rows == rows
    return b


@pytest.mark.parametrize("form", ["fused", "mixed"])
@pytest.mark.parametrize("kind, N, adaptive", [("mixed", 0, 0), ("sponge", 1, 0), ("irregular", 2, 0), ("mixed", 1, 1), ("sponge", 0, 1)])
def test_one_row_stencil_vs_fp64_oracle(celeris, form, kind, N, adaptive):
    """The bounds of the parity tests: 1e-4 m in eta, 2e-3 of the fields."""
    p, z, bnx, bny = cases.small_case(70, 45, kind, correction_steps=N)
    p.adaptive = adaptive
    if N == 0:
        p.timestep *= 0.5   # the scheme without a corrector is stable to half the Courant number
    ref, b = O.Oracle(p, z, bnx, bny, "f64"), _batch(celeris, [(p, z)], form, 1)
    ref.physical_steps(100)
    b.step(100)
    a = b.state(0)
    assert np.isfinite(a).all()
    assert eta_rms(a, ref.state()) <= 1e-4
    assert rel_ok(field_errors(a, ref.state()), 2e-3, 1e-6)


@pytest.mark.parametrize("adaptive, N", [(0, 1), (0, 2), (1, 1)])
def test_both_stencils_agree(celeris, adaptive, N):
    """Fields to FP32 rounding, the record, and the step's statistics: totals of states that may differ by 1e-5
    within the same, the volume as in the parity tests."""
    members = []
    for i, k in enumerate(["mixed", "sponge", "irregular"]):
        p, z, _, _ = cases.small_case(150 + 10 * i, 71 + 30 * i, k, correction_steps=N)
        p.adaptive = adaptive
        members.append((p, z))
    b1, b2 = (_batch(celeris, members, "mixed", rows) for rows in (1, 2))
    b1.step(40)
    b2.step(40)
    for i in range(len(members)):
        assert rel_ok(field_errors(b2.state(i), b1.state(i)), 1e-5, 1e-9), i
        a1, a2 = b1.aux(i), b2.aux(i)
        np.testing.assert_allclose(a2[..., 0], a1[..., 0], rtol=1e-4, atol=1e-6)
        assert ((a1[..., 3] > 0) == (a2[..., 3] > 0)).mean() > 0.999
    for x, y in zip(b1.stats(), b2.stats()):
        assert y["mass_full"] == pytest.approx(x["mass_full"], rel=1e-9)
        for k in ("mass", "potential_energy", "max_depth", "kinetic_energy", "max_speed", "cfl_rate"):
            assert y[k] == pytest.approx(x[k], rel=1e-5), k
        assert y["health"] == x["health"] == 0
        assert y["total_time"] == pytest.approx(x["total_time"], rel=1e-6)

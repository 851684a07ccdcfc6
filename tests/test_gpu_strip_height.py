"""Selected stencil strip heights are the heights that run; unselected ones follow the batch's size."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from celeris_b200 import cases
from util import eta_rms, field_errors, rel_ok

pytestmark = pytest.mark.gpu

VARIANTS = [(1, 128), (2, 128), (2, 96)]   # rows a step, threads


def _select(b, rows, width, height=0):
    b.set_stencil_rows(rows)
    if rows == 2:
        b.set_stencil_width(width)
    if height:
        b.set_tuning(0, height, 0)
        assert b.strip_height == height and b.tuning[1] == height
    assert (b.stencil_rows, b.stencil_width) == (rows, width)


@pytest.mark.parametrize("rows, width", VARIANTS)
def test_selected_heights_run_and_change_nothing(celeris, rows, width):
    """Heights from less than the ring to whole members, odd ones among them: the automatic split's bits."""
    members = [cases.small_case(nx, ny, k, seed=i)[:2]
               for i, ((nx, ny), k) in enumerate(zip([(189, 150), (95, 64), (40, 131)], ("mixed", "sponge", "solid")))]

    def states(height):
        b = celeris.Batch(members, "mixed")
        _select(b, rows, width, height)
        if not height:
            assert b.tuning[1] == 64 and 4 <= b.strip_height < 64   # 445 rows of strips do not fill the GPU
        b.step(12)
        return [b.state(i) for i in range(len(members))] + [b.aux(i) for i in range(len(members))]

    ref = states(0)
    for h in (8, 9, 33, 64, 1024):
        for a, r in zip(states(h), ref):
            np.testing.assert_array_equal(a, r)


@pytest.mark.parametrize("rows, width", VARIANTS)
@pytest.mark.parametrize("form", ["fused", "mixed"])
def test_tall_strips_against_the_oracle(celeris, rows, width, form):
    """One strip from end to end, 77 row pairs through a ring of six: the parity tests' bounds."""
    p, z, bnx, bny = cases.small_case(120, 153, "sponge", correction_steps=1)
    ref, b = O.Oracle(p, z, bnx, bny, "f64"), celeris.Batch([(p, z)], form)
    _select(b, rows, width, 160)
    ref.physical_steps(60)
    b.step(60)
    assert eta_rms(b.state(0), ref.state()) <= 1e-4
    assert rel_ok(field_errors(b.state(0), ref.state()), 2e-3, 1e-6)


def test_a_height_stays_through_other_settings(celeris):
    members = [cases.small_case(150, 90, "mixed")[:2]]
    b = celeris.Batch(members, "mixed")
    auto = b.strip_height
    b.set_tuning(8, 0, 0)
    assert b.strip_height == auto and b.tuning == (8, 64)
    b.set_tuning(16, 40, 0)
    b.set_stencil_rows(1)
    b.set_tuning(8, 0, 0)
    assert b.strip_height == 40 and b.tuning == (8, 40)


def test_the_tuner_reports_what_it_left(celeris):
    b = celeris.Batch([cases.small_case(150, 90, "mixed")[:2]], "mixed")
    got = b.autotune(2)
    assert b.tuning == (got["band_width"], got["strip_height"])
    assert b.strip_height == got["strip_height"] or (got["strip_height"] == 64 and b.strip_height < 64)

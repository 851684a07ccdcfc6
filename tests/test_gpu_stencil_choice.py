"""Selecting the stencil's variant and width: what may be selected depends on what runs, not on earlier calls."""
from __future__ import annotations

import pytest

from celeris_b200 import cases

pytestmark = pytest.mark.gpu


def _batch(celeris):
    return celeris.Batch([cases.small_case(150, 90, "mixed")[:2]], "mixed")


def test_the_paired_row_stencil_takes_both_widths(celeris):
    """A fresh batch runs two rows a step, so it takes 96 threads without selecting them first."""
    b = _batch(celeris)
    assert b.stencil_rows == 2
    for width in (96, 128, 96):
        b.set_stencil_width(width)
        assert (b.stencil_rows, b.stencil_width) == (2, width)
    b.set_stencil_rows(2)                      # already running: nothing changes
    assert b.stencil_width == 96


def test_the_one_row_stencil_takes_one(celeris):
    b = _batch(celeris)
    b.set_stencil_rows(1)
    with pytest.raises(celeris.CelError, match="one-row stencil"):
        b.set_stencil_width(96)
    b.set_stencil_width(128)
    assert (b.stencil_rows, b.stencil_width) == (1, 128)
    b.set_stencil_rows(2)                      # selecting two rows starts from 128 threads
    assert (b.stencil_rows, b.stencil_width) == (2, 128)
    b.set_stencil_width(96)
    assert b.stencil_width == 96


def test_the_tuner_leaves_a_selection(celeris):
    b = _batch(celeris)
    b.autotune(2)
    before = (b.stencil_rows, b.stencil_width)
    b.set_stencil_rows(before[0])
    assert (b.stencil_rows, b.stencil_width) == before

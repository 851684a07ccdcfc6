"""Reads into memory that the caller has pinned: the same texels as into pageable memory."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from celeris_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "fused", "mixed"])
@pytest.mark.parametrize("nx, ny", [(60, 33), (300, 601)])
def test_reads_into_pinned_memory(celeris, form, nx, ny):
    p, z, _, _ = cases.small_case(nx, ny, "sponge")
    eng = celeris.Engine(p, z, form)
    eng.physical_steps(5)
    for name, want in (("cel_get_state", eng.state()), ("cel_get_aux", eng.aux())):
        pinned = torch.full(want.shape, float("nan"), dtype=torch.float32).pin_memory()
        celeris.check(getattr(celeris.lib(), name)(eng.h, C.cast(pinned.data_ptr(), C.POINTER(C.c_float))))
        np.testing.assert_array_equal(pinned.numpy(), want)

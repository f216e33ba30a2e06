"""sedi_slab_totals: pinned results are written by the kernel, pageable ones
copied; both are the plane rows' sums.  Summands are small whole numbers, so
every order of summation gives the same bits."""
import ctypes

import numpy as np
import pytest

import sedi_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3", [1, 3, 255, 256, 257, 1000])
def test_pinned_and_pageable_totals(n3):
    import torch
    vp = ctypes.c_void_p
    lib = S.load()
    lib.sedi_slab_totals.argtypes = [ctypes.c_long, vp, vp, vp, vp]
    rows = torch.randint(-1000, 1000, (n3, 3), device="cuda").double()
    scratch = torch.zeros(3, dtype=torch.float64, device="cuda")
    want = rows.sum(0).cpu().numpy()
    pinned = torch.full((3,), 0.5, dtype=torch.float64, pin_memory=True)
    pageable = np.full(3, 0.5)
    for p in (pinned.data_ptr(), pageable.ctypes.data):
        assert lib.sedi_slab_totals(n3, rows.data_ptr(), scratch.data_ptr(), p,
                                    torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(pinned.numpy(), want) and np.array_equal(pageable, want)

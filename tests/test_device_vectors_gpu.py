"""Device solves with vectors a kernel must not take as they are: on 4-byte
boundaries and in pinned host memory (both go by way of a copy, as they do on
every form that copies), in every solver with an on-chip form.  The results are
those of plain device vectors, bit for bit."""
import ctypes

import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu

DIMS = (24, 20, 18)


def _solve(c, b, x, K):
    fe, fi = ctypes.c_double(), ctypes.c_int()
    vp = ctypes.c_void_p
    rc = S.load().sedi_solve_dev(c._h, vp(b), vp(x), None, K, 0.0, ctypes.byref(fe), ctypes.byref(fi))
    return rc, fe.value, fi.value


@pytest.mark.parametrize("solver", ["cg", "pcg", "bicgstab"])
@pytest.mark.parametrize("where", ["b", "x", "both", "pinned"])
def test_vectors_that_need_a_copy(solver, where):
    import torch
    n = int(np.prod(DIMS))
    probe = torch.from_numpy(O.fill_probe(21, n))
    guess = torch.from_numpy(np.cos(np.arange(n)))

    def place(v, odd):  # v's bytes, 4 past an 8-byte boundary when odd
        raw = torch.zeros(8 * n + 16, dtype=torch.uint8, device="cuda")
        off = 4 if odd else 8
        raw[off:off + 8 * n].copy_(v.view(torch.uint8))
        return raw, off

    with S.Context(solver, DIMS) as c:
        rb, ob = place(probe, False)
        rx, ox = place(guess, False)
        torch.cuda.synchronize()
        want = _solve(c, rb.data_ptr() + ob, rx.data_ptr() + ox, 15)
        xw = rx[ox:ox + 8 * n].cpu()
        assert want[0] == 1
        if where == "pinned":
            b, x = probe.pin_memory(), guess.pin_memory()
            got = _solve(c, b.data_ptr(), x.data_ptr(), 15)
            xg = x.view(torch.uint8)
        else:
            rb, ob = place(probe, where != "x")
            rx, ox = place(guess, where != "b")
            torch.cuda.synchronize()
            got = _solve(c, rb.data_ptr() + ob, rx.data_ptr() + ox, 15)
            xg = rx[ox:ox + 8 * n].cpu()
    assert got == want and torch.equal(xg, xw)

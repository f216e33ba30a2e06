"""A context allocates when it is created: solves of any number of right-hand
sides up to its batch take no device memory and give none back, and the admission
size covers what creation takes.  The on-chip solvers' plans follow the number of
right-hand sides, and a smaller batch can need the larger buffer (CG on 256x20x20:
12 solves 11.3 MB, 16 solves 5.9 MB)."""
import ctypes

import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu


def _used():
    used, total = ctypes.c_double(), ctypes.c_double()
    assert S.load().sedi_device_memory(ctypes.byref(used), ctypes.byref(total)) == 0
    return used.value * 2 ** 20


@pytest.mark.parametrize("solver,prec,dims,batch,sizes", [
    ("cg", S.FP64, (256, 20, 20), 16, (16, 12, 1, 16, 3)),
    ("pcg", S.FP64, (48, 48, 48), 16, (16, 5, 12, 16)),
    ("bicgstab", S.FP64, (384, 148, 16), 4, (4, 1, 3)),
    ("cg", S.MIXED, (40, 36, 30), 20, (20, 19, 3, 20)),
])
def test_solves_allocate_nothing(solver, prec, dims, batch, sizes):
    import torch
    n = int(np.prod(dims))
    b = torch.from_numpy(np.stack([O.fill_probe(5 + k, n) for k in range(batch)])).cuda()
    D = torch.empty(n, dtype=torch.float64, device="cuda")
    first = {}
    for warm in (True, False):  # the first round loads the kernels
        torch.cuda.synchronize()
        before = _used()
        with S.Context(solver, dims, precision=prec, batch=batch) as c:
            created = _used()
            for k in sizes:
                r = c.estimate_dev(k, b[:k], D, maxiter=6, tol=0.0)
                got = (D.cpu().numpy().tobytes(), r["iters"].tobytes())
                assert first.setdefault(k, got) == got  # the same on a new and a used context
                if not warm:
                    assert _used() == created
        if not warm:
            assert created - before <= S.job_bytes(solver, dims, batch, prec)

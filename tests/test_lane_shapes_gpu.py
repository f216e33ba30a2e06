"""Streaming batches take their launch shapes from the number of right-hand
sides they are given.  One context solves batches of changing size (the
captured iterations of two shapes are kept, a third replaces the older one):
each against the oracle at its tolerance, and each repeated size bit for bit.

Bars as for the other batched forms: FP64 CG and pipelined CG to 1e-10 with
the oracle's iteration counts and x within 1e-9; mixed lanes meet tol on
their FP64 true residual."""
import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu

DIMS = (520, 12, 70)  # wider than a box of the on-chip solvers
SIZES = (16, 3, 16, 3, 7, 1, 7, 16)


def _probes(k):
    n = int(np.prod(DIMS))
    return np.stack([O.fill_probe(300 + j, n) for j in range(k)])


@pytest.mark.parametrize("solver,precision", [("cg", S.FP64), ("pcg", S.FP64), ("cg", S.MIXED), ("bicgstab", S.MIXED)])
def test_batches_of_changing_size(solver, precision):
    B = _probes(max(SIZES))
    want = {}
    if precision == S.FP64:
        for k in (0, 2, 6, 15):
            want[k] = O.solve({"cg": 2, "pcg": 3}[solver], DIMS, B[k], maxiter=500, tol=1e-10)
    seen = {}
    with S.Context(solver, DIMS, precision=precision, batch=max(SIZES)) as c:
        for m in SIZES:
            X = np.zeros((m, B.shape[1]))
            res, fe, fi = c.solve_batch(X, B[:m], maxiter=500, tol=1e-10)
            assert np.all(res == 0)
            for k in range(m):
                if precision == S.MIXED:
                    r = B[k] - O.stencil(DIMS, X[k])
                    assert np.sqrt((r @ r) / (B[k] @ B[k])) <= 1e-10 * 1.0000001
                elif k in want:
                    rc0, fe0, fi0, x0, _ = want[k]
                    assert (res[k], fi[k]) == (rc0, fi0)
                    assert O.relmax(X[k], x0) <= 1e-9
            if m in seen:
                assert np.array_equal(X, seen[m][0]) and np.array_equal(fi, seen[m][1])
            seen[m] = (X, np.array(fi))

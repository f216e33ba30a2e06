"""A lane slice that has finished leaves the streaming sweeps, but owes the x
step of an odd last iteration, which the next iteration's sweep takes along the
old direction.  Whatever an earlier batch left in the vectors that its own
sweeps would have written must not reach x.

Eigenvectors of the stencil converge in the first iteration (the residual after
one step is rounding); the other lanes go on.  Bars as for the other FP64
batches: the oracle's iteration counts, x within 1e-9."""
import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu

DIMS = (520, 12, 10)  # wider than a box of the on-chip solvers
LANES = 16


def _eigenvectors(k):
    n1, n2, n3 = DIMS
    s = lambda n, m: np.sin(np.pi * m * np.arange(1, n + 1) / (n + 1))
    return np.stack([(s(n3, 1 + j % 3)[:, None, None] * s(n2, 1 + j % 2)[:, None] * s(n1, 1 + j)).ravel()
                     for j in range(k)])


@pytest.mark.parametrize("solver", ["cg", "pcg"])
@pytest.mark.parametrize("maxiter", [3, 4])  # the failed batch ends on either direction buffer
def test_early_slices_after_a_batch_without_numbers(solver, maxiter):
    n = int(np.prod(DIMS))
    with S.Context(solver, DIMS, batch=LANES) as c:
        W = c.config()["slice_width"]
        assert W < LANES
        bad = np.full((LANES, n), np.nan)
        assert np.all(c.solve_batch(np.zeros_like(bad), bad, maxiter, 1e-10)[0] == 1)
        B = np.stack([O.fill_probe(700 + j, n) for j in range(LANES)])
        B[:W] = _eigenvectors(W)
        X = np.zeros_like(B)
        res, fe, fi = c.solve_batch(X, B, 500, 1e-10)
    assert np.all(res == 0)
    for k in range(W + 2):
        rc0, fe0, fi0, x0, _ = O.solve(S.SOLVER_IDS[solver], DIMS, B[k], maxiter=500, tol=1e-10)
        assert (res[k], fi[k]) == (rc0, fi0)
        assert O.relmax(X[k], x0) <= 1e-9

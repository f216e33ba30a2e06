"""The batched streaming sweeps, on grids the on-chip solvers do not take (wider
than 512 points, or more than 2^22): thin and odd widths, narrow and deep grids,
every solver and precision, all sweep forms, finished slices, tuned contexts.

Bars, as for the other batched forms: FP64 CG and pipelined CG converged to 1e-10
with the oracle's iteration counts and x within 1e-9; FP64 at a few fixed
iterations within 1e-10; mixed lanes meet tol on their FP64 true residual."""
import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu

SID = {"cg": 2, "pcg": 3, "bicgstab": 1}
THIN = [(513, 1, 1), (515, 3, 2), (520, 1, 40), (521, 7, 9), (600, 2, 2), (514, 17, 1)]


def _probes(dims, k, seed):
    n = int(np.prod(dims))
    return np.stack([O.fill_probe(seed + j, n) for j in range(k)])


def _batch(solver, dims, B, maxiter, tol, prec=S.FP64, stencil=None):
    X = np.zeros_like(B)
    with S.Context(solver, dims, stencil, precision=prec, batch=len(B)) as c:
        res, fe, fi = c.solve_batch(X, B, maxiter=maxiter, tol=tol)
        assert c.launches > fi.max()  # a sweep or more an iteration: not one launch
    return X, res, fe, fi


@pytest.mark.parametrize("dims", THIN)
@pytest.mark.parametrize("solver", ["cg", "pcg"])
def test_fp64_converged_thin_grids(dims, solver):
    B = _probes(dims, 5, 900)
    X, res, fe, fi = _batch(solver, dims, B, 500, 1e-10)
    for k in range(5):
        rc0, fe0, fi0, x0, _ = O.solve(SID[solver], dims, B[k], maxiter=500, tol=1e-10)
        assert (res[k], fi[k]) == (rc0, fi0)
        assert O.relmax(X[k], x0) <= 1e-9


@pytest.mark.parametrize("coeffs", [(6.0, 1.0, 1.0), (6.0, 1.3, 0.7)])
@pytest.mark.parametrize("dims", THIN)
def test_fp64_bicgstab_thin_grids(dims, coeffs):
    B = _probes(dims, 4, 950)
    X, res, fe, fi = _batch("bicgstab", dims, B, 8, 0.0, stencil=S.Stencil(*coeffs))
    for k in range(4):
        rc0, fe0, fi0, x0, _ = O.solve(1, dims, B[k], maxiter=8, tol=0.0, coeffs=coeffs)
        assert (res[k], fi[k]) == (rc0, fi0)
        assert O.relmax(X[k], x0) <= 1e-10


@pytest.mark.parametrize("dims", THIN)
@pytest.mark.parametrize("solver", ["cg", "pcg", "bicgstab"])
def test_mixed_thin_grids_true_residual(dims, solver):
    B = _probes(dims, 6, 970)
    X, res, fe, fi = _batch(solver, dims, B, 2000, 1e-10, S.MIXED)
    assert np.all(res == 0)
    for k in range(6):
        r = B[k] - O.stencil(dims, X[k])
        assert np.sqrt((r @ r) / (B[k] @ B[k])) <= 1e-10 * 1.0000001


@pytest.mark.parametrize("dims", [(9, 700, 700), (1, 2100, 2000), (33, 3, 43000)])
@pytest.mark.parametrize("solver", ["cg", "pcg", "bicgstab"])
def test_fp64_narrow_grids_at_fixed_iterations(dims, solver):
    B = _probes(dims, 3, 400)
    X, res, fe, fi = _batch(solver, dims, B, 7, 0.0)  # odd: CG's deferred step is pending at the end
    for k in (0, 2):
        rc0, fe0, fi0, x0, _ = O.solve(SID[solver], dims, B[k], maxiter=7, tol=0.0)
        assert (res[k], fi[k]) == (rc0, fi0)
        assert O.relmax(X[k], x0) <= 1e-10


@pytest.mark.parametrize("prec", [S.FP64, S.MIXED])
@pytest.mark.parametrize("solver", ["cg", "bicgstab"])
def test_sweep_forms_agree(solver, prec):
    """A ring of computed planes (form 1) and in place (forms 2 and 3): the same
    values summed on other tiles.  CG to 1e-10: FP64 D within 1e-12, mixed within
    1e-9; BiCGStab at 20 fixed iterations: FP64 1e-9, mixed 1e-6."""
    dims, samples = (515, 13, 11), 16
    maxiter, tol = (3000, 1e-10) if solver == "cg" else (20, 0.0)
    out = {}
    for form in (1, 2, 3):
        S.set_tuning(solver, dims, samples, precision=prec, sweep_a_form=form)
        with S.Context(solver, dims, precision=prec, batch=samples) as c:
            assert c.config()["sweep_a_form"] == form
            out[form] = c.estimate(samples, 99, maxiter, tol, ignore_errors=True)
            assert c.launches > out[form]["iters"].max()
    S.set_tuning(solver, dims, samples, precision=prec)
    bar = {("cg", S.FP64): 1e-12, ("cg", S.MIXED): 1e-9, ("bicgstab", S.FP64): 1e-9, ("bicgstab", S.MIXED): 1e-6}
    for form in (2, 3):
        assert np.array_equal(out[form]["results"], out[1]["results"])
        if (solver, prec) == ("cg", S.FP64):
            assert np.array_equal(out[form]["iters"], out[1]["iters"])
        assert O.relmax(out[form]["D"], out[1]["D"]) <= bar[solver, prec]


@pytest.mark.parametrize("prec", [S.FP64, S.MIXED])
def test_bicgstab_batches_of_changing_size(prec):
    """A slice of lanes without right-hand sides is left out; each repeated size
    gives the same bits, FP64 the oracle's x at 10 fixed iterations."""
    dims, sizes = (520, 12, 30), (16, 3, 16, 7, 1, 7)
    B = _probes(dims, max(sizes), 300)
    seen = {}
    with S.Context("bicgstab", dims, precision=prec, batch=max(sizes)) as c:
        for m in sizes:
            X = np.zeros((m, B.shape[1]))
            res, fe, fi = c.solve_batch(X, B[:m], maxiter=10, tol=0.0)
            if m in seen:
                assert np.array_equal(X, seen[m])
            seen[m] = X
    if prec == S.FP64:
        for k in (0, 6, 15):
            rc0, fe0, fi0, x0, _ = O.solve(1, dims, B[k], maxiter=10, tol=0.0)
            for m in sizes:
                if k < m:
                    assert O.relmax(seen[m][k], x0) <= 1e-10


@pytest.mark.parametrize("solver", ["cg", "pcg", "bicgstab"])
def test_slices_finish_at_their_own_iterations(solver):
    """Smooth lanes (few eigenvectors) converge in as many iterations, the others
    later: whole slices leave, in either parity of CG's deferred step."""
    dims = (520, 12, 10)
    s = lambda n, m: np.sin(np.pi * m * np.arange(1, n + 1) / (n + 1))
    lanes = 16
    B = _probes(dims, lanes, 800)
    with S.Context(solver, dims, batch=lanes) as c:
        W = c.config()["slice_width"]
        for k in range(lanes - W):  # slice j: j + 1 eigenvectors
            B[k] = sum((1.0 + 0.1 * k + m) * (s(dims[2], 1 + m)[:, None, None] * s(dims[1], 1 + 2 * m)[:, None]
                                              * s(dims[0], 1 + 40 * m)).ravel() for m in range(k // W + 1))
        X = np.zeros_like(B)
        res, fe, fi = c.solve_batch(X, B, 500, 1e-10)
    assert np.all(res == 0)
    for k in range(lanes):
        r = B[k] - O.stencil(dims, X[k])
        assert np.sqrt((r @ r) / (B[k] @ B[k])) <= 1e-9  # (recurrence residual <= 1e-10)
        if solver != "bicgstab":
            rc0, fe0, fi0, x0, _ = O.solve(SID[solver], dims, B[k], maxiter=500, tol=1e-10)
            assert (res[k], fi[k]) == (rc0, fi0)
            assert O.relmax(X[k], x0) <= 1e-9


@pytest.mark.parametrize("solver,prec", [("cg", S.FP64), ("cg", S.MIXED), ("bicgstab", S.FP64)])
def test_tuned_context_keeps_results(solver, prec):
    """The autotuner's choices change launch shapes and summation order alone."""
    dims, samples = (516, 14, 12), 16
    maxiter, tol = (20, 0.0) if solver == "bicgstab" else (3000, 1e-9)
    try:
        with S.Context(solver, dims, precision=prec, batch=samples) as c:
            ref = c.estimate(samples, 321, maxiter, tol, ignore_errors=True)
        choice = S.autotune(solver, dims, samples, precision=prec, maxiter=maxiter, tol=tol, seed=321)
        with S.Context(solver, dims, precision=prec, batch=samples) as c:
            cf = c.config()
            got = c.estimate(samples, 321, maxiter, tol, ignore_errors=True)
    finally:
        S.set_tuning(solver, dims, samples, precision=prec)
    assert choice["chunk"] and (cf["slice_width"], cf["chunk"]) == (choice["slice_width"], choice["chunk"])
    assert np.array_equal(got["results"], ref["results"])
    if prec == S.FP64:
        assert np.array_equal(got["iters"], ref["iters"])
    assert O.relmax(got["D"], ref["D"]) <= (1e-8 if prec == S.MIXED else 1e-10)

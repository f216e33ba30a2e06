"""Tuning of grids that are solved on chip: the choices of the streaming sweeps
act on nothing there and stay the built-in ones, results keep their bits, and the
mixed form's reliable-update period is the one thing measured."""
import numpy as np
import pytest

import sedi_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solve", [True, False])
@pytest.mark.parametrize("solver,prec", [("cg", S.FP64), ("cg", S.MIXED), ("pcg", S.FP64), ("bicgstab", S.FP64)])
def test_autotune_measures_what_acts(solver, prec, solve):
    dims, samples = (28, 26, 24), 12
    maxiter, tol = (15, 0.0) if solver == "bicgstab" else (500, 1e-8)

    def run():
        with S.Context(solver, dims, precision=prec, batch=samples) as c:
            r = c.estimate(samples, 77, maxiter, tol)
            return r, c.config()

    before, cb = run()
    try:
        got = S.autotune(solver, dims, samples, precision=prec, maxiter=maxiter, tol=tol, seed=77, solve=solve)
        after, ca = run()
    finally:
        S.set_tuning(solver, dims, samples, precision=prec)
    assert got["score_ms"] > 0
    assert (got["z_chunks"], got["chunk"], got["prefetch_planes"]) == (0, 0, -1)
    assert got["slice_width"] == cb["slice_width"] and got["sweep_a_form"] == cb["sweep_a_form"]
    tuned = prec == S.MIXED and solve
    assert got["period"] in ((20, 32, 50) if tuned else (0,))
    assert ca == dict(cb, period=got["period"] or cb["period"])
    if ca["period"] == cb["period"]:
        assert np.array_equal(after["D"], before["D"]) and np.array_equal(after["iters"], before["iters"])

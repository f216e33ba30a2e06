"""Whole solves in one launch with the Krylov fields on chip (grids of up to
512 points along i1 that fit the GPU's shared memory and registers).

Elementwise values round as the sweeps and march kernels round them, so the
forms differ only in the order of the dot products: 1e-10 at fixed iteration
counts, the bar of the other FP64 forms.
"""
import threading

import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu


# Boxes with remainders along i2 and i3, one block, one plane a block, a full
# block row (512), one point wide, every box shape's size range, and the first
# grid that is too wide (513).
@pytest.mark.parametrize("dims", [(33, 17, 9), (97, 65, 51), (128, 33, 70), (512, 6, 5), (513, 4, 3), (1, 40, 37),
                                  (31, 1, 64), (64, 64, 64), (300, 40, 30), (100, 110, 120), (80, 85, 88), (96, 96, 96), (61, 100, 131)])
@pytest.mark.parametrize("coeffs", [(6.0, 1.0, 1.0), (6.5, 1.2, 0.9)])
@pytest.mark.parametrize("solver,K", [("cg", 21), ("pcg", 21), ("bicgstab", 12)])
def test_single_vector_matches_oracle(dims, coeffs, solver, K):
    n = int(np.prod(dims))
    b = O.fill_probe(7, n)
    x0 = np.cos(np.arange(n))
    rc0, fe0, fi0, xo, h0 = O.solve(S.SOLVER_IDS[solver], dims, b, x0=x0, maxiter=K, tol=0.0, coeffs=coeffs)
    x = x0.copy()
    with S.Context(solver, dims, S.Stencil(*coeffs)) as c:
        rc, fe, fi = c.solve(x, b, None, K, 0.0)
        hist = c.history()
    assert (rc, fi) == (rc0, fi0)
    assert O.relmax(x, xo) <= 1e-10
    assert len(hist) == len(h0[:K + 1]) and O.relmax(hist, h0[:K + 1]) <= 1e-9


@pytest.mark.parametrize("solver,K", [("pcg", 25), ("bicgstab", 12)])
@pytest.mark.parametrize("dims,lanes", [((33, 17, 9), 5), ((40, 36, 30), 40), ((64, 20, 50), 3)])
def test_fp64_batches_match_single_vector(dims, lanes, solver, K):
    n = int(np.prod(dims))
    B = np.stack([O.fill_probe(90 + k, n) for k in range(lanes)])
    X = np.zeros_like(B)
    with S.Context(solver, dims, batch=lanes) as c:
        res, fe, fi = c.solve_batch(X, B, maxiter=K, tol=0.0)
    with S.Context(solver, dims) as c:
        for k in (0, lanes // 2, lanes - 1):
            x = np.zeros(n)
            out = c.solve(x, B[k], None, K, 0.0)
            assert (res[k], fi[k]) == (out[0], out[2]) and O.relmax(X[k], x) <= 1e-10


@pytest.mark.parametrize("prec", [S.FP64, S.MIXED])
@pytest.mark.parametrize("dims,lanes", [((33, 17, 9), 5), ((48, 48, 48), 16), ((40, 36, 30), 7), ((64, 20, 50), 33)])
def test_batch_matches_single_vector(dims, lanes, prec):
    """Several groups side by side, more solves than groups, an odd last pair."""
    n = int(np.prod(dims))
    B = np.stack([O.fill_probe(40 + k, n) for k in range(lanes)])
    X = np.zeros_like(B)
    with S.Context("cg", dims, precision=prec, batch=lanes) as c:
        res, fe, fi = c.solve_batch(X, B, maxiter=2000, tol=1e-10)
    assert np.all(res == 0)
    with S.Context("cg", dims) as c:
        for k in (0, lanes // 2, lanes - 1):
            x = np.zeros(n)
            assert c.solve(x, B[k], None, 2000, 1e-10)[0] == 0
            if prec == S.FP64:
                assert O.relmax(X[k], x) <= 1e-10
            else:  # both meet the tolerance on their FP64 true residual
                assert O.relmax(X[k], x) <= 1e-7
            r = B[k] - O.stencil(dims, X[k])
            assert np.sqrt((r @ r) / (B[k] @ B[k])) <= 1.0000001e-10


def test_device_solve_in_place_and_overlapping_vectors():
    torch = pytest.importorskip("torch")
    dims = (40, 30, 20)
    n = int(np.prod(dims))
    b = torch.from_numpy(O.fill_probe(3, n)).cuda()
    x = torch.zeros_like(b)
    same = b.clone()
    with S.Context("cg", dims) as c:
        ref = b.clone()
        r0 = c.solve(ref, b.clone(), None, 25, 0.0)  # first guess b
        r1 = c.solve(same, same, None, 25, 0.0)
        c.solve(x, b, None, 25, 0.0)
    assert r0 == r1 and torch.equal(same, ref)
    xo = O.solve(2, dims, b.cpu().numpy(), maxiter=25, tol=0.0)[3]
    assert O.relmax(x.cpu().numpy(), xo) <= 1e-10


def test_concurrent_solves_each_find_room():
    """Solves that wait for their own blocks, from several threads and streams:
    each ends, with the result it has alone."""
    shapes = [(100, 100, 100), (32, 32, 32), (96, 80, 70), (128, 100, 90)]
    probes = [O.fill_probe(11 + k, int(np.prod(d))) for k, d in enumerate(shapes)]

    def solve(k):
        x = np.zeros(probes[k].size)
        with S.Context("cg", shapes[k]) as c:
            out = c.solve(x, probes[k], None, 300, 0.0)
        return out, x

    alone = [solve(k) for k in range(len(shapes))]
    got = [[] for _ in shapes]

    def worker(k):
        for _ in range(4):
            got[k].append(solve(k))

    ts = [threading.Thread(target=worker, args=(k,)) for k in range(len(shapes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, a in enumerate(alone):
        assert len(got[k]) == 4
        for g in got[k]:
            assert g[0] == a[0] and np.array_equal(g[1], a[1])


@pytest.mark.parametrize("prec", [S.FP64, S.MIXED])
def test_streaming_forms_on_a_wide_grid(prec):
    """Grids wider than 512 points take the streaming sweeps at any size: their
    three sweep-A forms give the same values, summed on other tiles."""
    dims, samples = (520, 12, 10), 8
    out = {}
    for form in (1, 2, 3):
        S.set_tuning("cg", dims, samples, precision=prec, sweep_a_form=form)
        with S.Context("cg", dims, precision=prec, batch=samples) as c:
            out[form] = c.estimate(samples, 99, 3000, 1e-10)
    S.set_tuning("cg", dims, samples, precision=prec)
    for form in (2, 3):
        assert np.array_equal(out[form]["results"], out[1]["results"])
        assert O.relmax(out[form]["D"], out[1]["D"]) <= (1e-12 if prec == S.FP64 else 1e-9)

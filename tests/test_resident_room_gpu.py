"""On-chip solves of every room class from several threads at once: two blocks
an SM (64^3 x 8), single-block groups in several rounds (16^3 x 64) and a group
of nearly all SMs (128^3).  Each ends, with the result it has alone."""
import threading

import numpy as np
import pytest

import _oracle as O
import sedi_b200 as S

pytestmark = pytest.mark.gpu

JOBS = [((64, 64, 64), 8, 150), ((16, 16, 16), 64, 400), ((128, 128, 128), 1, 100), ((40, 30, 20), 24, 200)]


def test_launches_of_every_room_class_together():
    rhs = []
    for d, k, _ in JOBS:
        n = int(np.prod(d))
        rhs.append(np.stack([O.fill_probe(50 + j, n) for j in range(min(k, 4))])[np.arange(k) % 4])

    def solve(j):
        d, k, m = JOBS[j]
        x = np.zeros_like(rhs[j])
        with S.Context("cg", d, batch=k) as c:
            out = c.solve(x[0], rhs[j][0], None, m, 0.0) if k == 1 else c.solve_batch(x, rhs[j], m, 0.0)
        return x, out

    alone = [solve(j) for j in range(len(JOBS))]
    got = [[] for _ in JOBS]

    def worker(j):
        for _ in range(5):
            got[j].append(solve(j))

    ts = [threading.Thread(target=worker, args=(j,)) for j in range(len(JOBS))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for j in range(len(JOBS)):
        assert len(got[j]) == 5
        for x, out in got[j]:
            assert np.array_equal(x, alone[j][0])
            assert all(np.array_equal(a, b) for a, b in zip(out, alone[j][1]))

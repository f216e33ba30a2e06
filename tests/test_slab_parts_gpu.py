"""Plane sums of the slab sweeps where row chunks and their cluster parts are
uneven or empty: a plane is cut into 8 chunks of ceil(n2 / 8) rows, each shared
by a cluster of 4 blocks that add their sums in the first one's shared memory.
A part without rows has nothing to do before it hands over its zeros.

Vectors hold small whole numbers, so every order of summation gives the same
bits and the sums are compared exactly."""
import numpy as np
import pytest

from sedi_b200.domain import PCG_SETUP, SETUP, GpuSlabBackend

pytestmark = pytest.mark.gpu


def _stencil(x):
    p = np.pad(x, 1)
    y = 6.0 * x
    for d in range(3):
        for lo in (0, 2):
            s = [slice(1, -1)] * 3
            s[d] = slice(lo, lo + x.shape[d])
            y = y - p[tuple(s)]
    return y


# Rows a chunk (ceil(n2 / 8)) of 1 to 8: one to four parts with rows; chunks
# without any; rows narrower than a warp, of several warps and of several
# passes of the block.
@pytest.mark.parametrize("n2", [1, 3, 8, 9, 24, 31, 33, 40, 64])
@pytest.mark.parametrize("n1", [1, 33, 200, 300])
def test_plane_sums_with_uneven_and_empty_parts(n1, n2):
    import torch
    n3 = 5
    rng = np.random.default_rng(1000 * n1 + n2)
    x, b = (rng.integers(-3, 4, (n3, n2, n1)).astype(np.float64) for _ in range(2))
    be = GpuSlabBackend((n1, n2, n3))
    buf = {k: be.zeros(n3) for k in "xbruwqspz"}
    be.set_interior(buf["x"], x)
    be.set_interior(buf["b"], b)
    ax = _stencil(x)
    for _ in range(20):  # every launch sums the same
        G = be.plane_sums(n3)
        be.sweep(SETUP, n3, 1, n3 + 1, G, src=buf["x"], b=buf["b"], r=buf["r"])
        want = np.stack([(b * b).sum((1, 2)), ((b - ax) ** 2).sum((1, 2)), np.zeros(n3)], 1)
        torch.cuda.synchronize()
        assert np.array_equal(G.cpu().numpy(), want)
        be.sweep(PCG_SETUP, n3, 1, n3 + 1, G, src=buf["x"], u=buf["u"], w=buf["w"], q=buf["q"], s=buf["s"],
                 p=buf["p"], z=buf["z"], iM=1.0)
        want = np.stack([(x * x).sum((1, 2)), (ax * x).sum((1, 2)), (x * x).sum((1, 2))], 1)
        torch.cuda.synchronize()
        assert np.array_equal(G.cpu().numpy(), want)

"""Slender grids (few columns of nodes, many planes, and the other ways round) are not marched: products and solves against the
oracle, at sizes beside the line where the march is left out (more than 6 steps, 8 for the product, and one more for every
8,000 nodes)."""
import numpy as np
import pytest
import torch

import oracle
import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 2000), (1, 1, 2100), (2, 2, 1000), (1, 2000, 1), (2100, 1, 1), (1, 100, 100), (100, 1, 100), (4, 4, 330), (3, 5, 700), (20, 20, 20)]


def bar(dims, seed):
    """Graded, a few voxels empty, held at the ends of the long axis' first plane."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    d = rng.uniform(0.05, 1.0, (nz, ny, nx)).astype(np.float32)
    if min(dims) > 1:
        d[rng.uniform(size=d.shape) < 0.05] = 0
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    ax = int(np.argmax(dims))
    bc[(slice(None),) * (2 - ax) + (0,)] = 1
    d, _ = W.prune_floating(dims, d.ravel(), bc.reshape(-1, 3).max(axis=1))
    return d, bc.ravel()


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("shift", [False, True])
def test_products_match_the_oracle(dims, shift):
    """FP64 y = K x and the allocation-free y and x . y: sums of some hundred terms, so 1e-12 of the result."""
    d, bc = bar(dims, sum(dims))
    rng = np.random.default_rng(3)
    add = rng.uniform(0.0, 0.5, bc.size) if shift else None
    S = psfea.VoxelFEA(dims, d, 0.3, bc, 50, diag_add=add)
    P = oracle.OracleModel("port", dims, d, 0.3, bc, 50, diag_add=add)
    x = rng.standard_normal(bc.size)
    yo = P.apply(x)
    assert np.linalg.norm(S.apply(x) - yo) <= 1e-12 * np.linalg.norm(yo)
    xd, yd = torch.from_numpy(x).cuda(), torch.full((x.size,), float("nan"), dtype=torch.float64, device="cuda")
    dd = torch.zeros(1, dtype=torch.float64, device="cuda")
    for _ in range(2):
        S.apply_dot_noalloc(xd.data_ptr(), yd.data_ptr(), dd.data_ptr(), torch.cuda.current_stream().cuda_stream)
    y = yd.cpu().numpy()
    assert np.linalg.norm(y - yo) <= 1e-12 * np.linalg.norm(yo) and np.all(y[P.fixed(0) != 0] == 0)
    assert abs(float(dd[0]) - float(x @ yo)) < 1e-12 * float(np.abs(x * yo).sum())


def test_long_thin_products_take_no_march_of_many_steps():
    """1 x 1 x 4000 voxels: the product marched takes 35 us (32 steps), a node a thread 13 us."""
    dims = (1, 1, 4000)
    d, bc = bar(dims, 1)
    S = psfea.VoxelFEA(dims, d, 0.3, bc, 1100)
    x = torch.randn(bc.size, dtype=torch.float64, device="cuda")
    y, dot = torch.empty_like(x), torch.zeros(1, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def calls(n):
        for _ in range(n):
            S.apply_dot_noalloc(x.data_ptr(), y.data_ptr(), dot.data_ptr(), s)

    calls(20)
    best = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        calls(100)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 10)
    assert best < 24, best  # us a call

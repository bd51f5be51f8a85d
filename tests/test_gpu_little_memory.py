"""A solve where the device memory left does not hold a small level's stencils (1152 B a node): the level keeps the gather."""
import numpy as np
import pytest
import torch
from cuda.bindings import driver

import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def test_small_levels_keep_the_gather(monkeypatch):
    dims = (112, 80, 64)  # level 1: 77 k nodes, of which some 60 k are active: 69 MB of stencils
    nx, ny, nz = dims
    d = np.random.default_rng(5).uniform(0.2, 1.0, (nz, ny, nx)).astype(np.float32)
    d[:, ny // 2:, nx // 2:] = 0
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    f = np.zeros(bc.shape)
    f[:, :ny // 2, nx, 1] = 1.0
    d, _ = W.prune_floating(dims, d.ravel(), bc.reshape(-1, 3).max(axis=1))
    f = f.ravel()

    def make():
        return psfea.VoxelFEA(dims, d, 0.3, bc.ravel(), 300)

    # every kernel of both routes has run (and is loaded) before the memory is taken
    A = make()
    a = A.solve(f, tol=1e-8, max_iter=3000)
    monkeypatch.setenv("PSFEA_STENCIL_LEVELS", "0")
    G = make()
    g = G.solve(f, tol=1e-8, max_iter=3000)
    monkeypatch.delenv("PSFEA_STENCIL_LEVELS")
    assert a.converged and g.converged
    stencils = A.device_bytes - G.device_bytes
    assert stencils > 60 << 20
    S = make()  # (A and G stay: what they hold does not come back to the allocator's pool)
    S.time_kernel(0, 1)  # the smoothers' estimates, whose scratch is freed again
    torch.cuda.synchronize()
    taken = []
    for mb in (4096, 256, 16):  # all of the device's memory through the pool the handles allocate from, in pieces down to 16 MB
        while True:
            err, p = driver.cuMemAllocAsync(mb << 20, 0)
            if err != driver.CUresult.CUDA_SUCCESS:
                break
            taken.append(p)
    for _ in range(3):  # 48 MB back: enough for everything but the stencils of level 1
        driver.cuMemFreeAsync(taken.pop(), 0)
    torch.cuda.synchronize()
    before = S.device_bytes
    try:
        r = S.solve(f, tol=1e-8, max_iter=3000)
        held = S.device_bytes - before
    finally:
        for p in taken:
            driver.cuMemFreeAsync(p, 0)
        torch.cuda.synchronize()
    assert r.converged and np.linalg.norm(r.u - a.u) <= 1e-5 * np.linalg.norm(a.u)
    assert held < stencils - (50 << 20)  # without level 1's
    # and with memory again
    assert S.solve(f, tol=1e-8, max_iter=3000).converged

"""A model without a solid voxel (a pruned-away part, every voxel below the threshold): every DOF is held, so every call
answers with zeros, at sizes below and above the smallest marched level (8,000 nodes)."""
import numpy as np
import pytest

import psfea

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(6, 5, 4), (24, 24, 24)])
def test_every_call_answers_with_zeros(dims):
    nx, ny, nz = dims
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    S = psfea.VoxelFEA(dims, np.zeros(nx * ny * nz, np.float32), 0.3, bc.ravel(), 300)
    f = np.random.default_rng(0).standard_normal(bc.size)
    for prec in ("fp64", "mixed", "fp32", "half"):
        for x0 in (None, f):
            r = S.solve(f, tol=1e-8, max_iter=50, precision=prec, x0=x0)
            assert r.status == psfea.PS_OK and r.converged and r.iterations == 0 and np.all(r.u == 0), (prec, x0 is None)
    for r in S.solve_batch(np.stack([f, -f]), tol=1e-8, max_iter=50):
        assert r.converged and np.all(r.u == 0)
    assert np.all(S.apply(f) == 0) and np.all(S.precondition(f) == 0)
    assert S.autotune(f, tol=1e-8, max_iter=50, force=True)["trials"] > 0

"""The server admits requests by an estimate of their device memory: it has to cover what a handle holds after its solves, the
stencils of every level among them, whatever share of a level's nodes is active."""
import numpy as np
import pytest

import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def graded(dims, empty_quadrant):
    """A graded block (every coarse matrix its own, so that no shared classes hide what is missing), held at x = 0; with
    empty_quadrant a part of it is left out: a level's nodes are then far more than its active ones."""
    rng = np.random.default_rng(5)
    nx, ny, nz = dims
    d = rng.uniform(0.2, 1.0, (nz, ny, nx)).astype(np.float32)
    if empty_quadrant:
        d[:, ny // 2:, nx // 3:] = 0
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    f = np.zeros(bc.shape)
    f[:, :ny // 2, nx, 1] = 1.0
    return W.prune_floating(dims, d.ravel(), bc.reshape(-1, 3).max(axis=1))[0], bc.ravel(), f.ravel()


# level 1: 30 k nodes (stencils with eight lanes a node), 82 k nodes (one thread a node), 94 k nodes of which 60 k are active
@pytest.mark.parametrize("dims,empty", [((60, 60, 60), False), ((96, 80, 80), False), ((120, 80, 72), True)])
def test_estimate_covers_a_handle_after_its_solves(dims, empty):
    d, bc, f = graded(dims, empty)
    for prec in ("mixed", "fp32"):
        srv = psfea.Server(max_active=1, build_threads=1)
        r = srv.wait(srv.submit(dims, d, 0.3, bc, f, tol=1e-6, precision=prec, coarsest_max_dof=300))
        need = srv.stats()["peak_device_bytes"]
        srv.close()
        assert r["converged"]
        S = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
        assert S.solve(f, tol=1e-6, max_iter=5000, precision=prec).converged
        assert S.device_bytes <= need <= 1.25 * S.device_bytes + (32 << 20), (prec, S.device_bytes, need)
        S.close()

"""ps_fea_precondition gives what a fresh handle gives, whatever ran before: its V-cycle has the FP64 form's stencils from the
first call on."""
import numpy as np
import pytest

import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def models():
    yield W.l_bracket(48, 24, 24, holes=4, seed=3)  # small Galerkin levels: eight lanes a node
    yield W.simp(96, 48, 48, nrhs=1)  # graded: every coarse matrix its own


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("min_nodes", [None, "4000"])
def test_the_same_before_and_after_solves(monkeypatch, which, min_nodes):
    """min_nodes: lists of more than 4,000 nodes one thread a node (PSFEA_STENCIL_MIN_NODES), FP32 or FP16 by form."""
    if min_nodes:
        monkeypatch.setenv("PSFEA_STENCIL_MIN_NODES", min_nodes)
    m = list(models())[which]
    f = m.f if m.f.ndim == 1 else m.f[0]
    S = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    r = np.random.default_rng(4).standard_normal(S.n_dof) * (S.fixed(0) == 0)
    z = S.precondition(r)
    assert np.array_equal(S.precondition(r), z)
    for prec in ("fp32", "half", "fp64", "mixed"):
        assert S.solve(f, tol=1e-6, max_iter=2000, precision=prec).converged
        assert np.array_equal(S.precondition(r), z), prec
    T = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    assert T.solve(f, tol=1e-6, max_iter=2000, precision="fp32").converged
    assert np.array_equal(T.precondition(r), z)

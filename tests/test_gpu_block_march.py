"""The block solve's marched finest level at the sizes where its tiles end: 7 x 7 output nodes a tile in 32 bits and 7 x 5 in
64, ranges of planes, 8 right-hand sides a CTA in blocks of 8, 16 and 32, with empty voxels and a diagonal shift."""
import numpy as np
import pytest
import torch

import oracle
import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def graded(dims, seed):
    """Densities in [0.2, 1], an opening, the x = 0 face held and one node elsewhere in y only."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    d = rng.uniform(0.2, 1.0, (nz, ny, nx)).astype(np.float32)
    if min(dims) > 3:
        d[nz // 3:nz // 2 + 1, ny // 2:, nx // 3:nx // 2] = 0
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    bc[nz, ny, nx, 1] = 1
    d, _ = W.prune_floating(dims, d.ravel(), bc.reshape(-1, 3).max(axis=1))
    return d, bc.ravel()


def loads(P, n, seed):
    """n loads over the whole part (every node of an active voxel, so that no node's product goes untested)."""
    return np.random.default_rng(seed).standard_normal((n, P.n_dof)) * (P.fixed(0) == 0)


# node counts at, below and above multiples of 7 (x and y) and of 5 (y), one to three planes of voxels, columns cut into ranges
SIZES = [(5, 5, 4), (6, 6, 3), (7, 7, 5), (12, 3, 2), (13, 4, 1), (14, 5, 2), (20, 8, 3), (21, 9, 12), (6, 10, 40), (27, 13, 6)]


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("width", [8, 16, 32])
@pytest.mark.parametrize("shift", [False, True])
def test_block_solves_match_the_oracle(dims, width, shift):
    """Every right-hand side to the oracle's solution: both are solved to 1e-10, on models whose condition leaves 1e-6 of that."""
    d, bc = graded(dims, sum(dims) + width)
    add = np.random.default_rng(2).uniform(0.0, 0.3, bc.size) if shift else None
    S = psfea.VoxelFEA(dims, d, 0.3, bc, 60, diag_add=add)
    P = oracle.OracleModel("port", dims, d, 0.3, bc, 60, diag_add=add)
    F = loads(P, width - 1, 7)
    F[1] *= 1e6  # right-hand sides of their own scale
    rs = S.solve_batch(F, tol=1e-10, max_iter=2000)
    free = P.fixed(0) == 0
    for q, r in enumerate(rs):
        assert r.converged, q
        res = (F[q] - P.apply(r.u))[free]
        assert np.linalg.norm(res) <= 1e-9 * np.linalg.norm(F[q]), q
    for q in (0, 1, width - 2):
        uo, _, _, _ = P.solve(F[q], 1e-10, 2000)
        assert np.linalg.norm(rs[q].u - uo) <= 1e-6 * np.linalg.norm(uo), q


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("shift", [False, True])
def test_block_preconditioner_matches_the_oracle(dims, shift):
    """One V-cycle per vector in blocks of 8, 16 and 32 against the oracle's: FP32 sums in another order, 1e-4 as for the single
    preconditioner."""
    d, bc = graded(dims, sum(dims))
    add = np.random.default_rng(2).uniform(0.0, 0.3, bc.size) if shift else None
    P = oracle.OracleModel("port", dims, d, 0.3, bc, 60, diag_add=add)
    r = loads(P, 30, 8)
    want = [P.precondition(v) for v in r[:3]]
    for n in (3, 11, 30):
        S = psfea.VoxelFEA(dims, d, 0.3, bc, 60, diag_add=add)
        rd = torch.from_numpy(r[:n]).cuda()
        zd = torch.full_like(rd, float("nan"))
        S.precondition_block(n, rd.data_ptr(), zd.data_ptr(), torch.cuda.current_stream().cuda_stream)
        z = zd.cpu().numpy()
        assert np.all(np.isfinite(z))
        for q in range(3):
            assert np.linalg.norm(z[q] - want[q]) <= 1e-4 * np.linalg.norm(want[q]), (n, q)


def test_stencils_over_the_boundary_list_of_a_split_marched_level(monkeypatch):
    """A marched level with own matrices whose boundary nodes all go to the stencils (PSFEA_TILE_SPLIT32=-1), against its march
    without a split: solves to 1e-9 agree to 1e-5 in every form."""
    m = W.l_bracket(64, 32, 32, holes=6, seed=4)
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "0")
    monkeypatch.setenv("PSFEA_STENCIL_MIN_NODES", "0")
    A = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    monkeypatch.setenv("PSFEA_TILE_SPLIT32", "-1")
    B = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    for prec in ("fp64", "mixed", "fp32"):
        a, b = (S.solve(m.f, tol=1e-9, max_iter=3000, precision=prec) for S in (A, B))
        assert a.converged and b.converged, prec
        assert np.linalg.norm(b.u - a.u) <= 1e-5 * np.linalg.norm(a.u), prec
        assert abs(a.iterations - b.iterations) <= max(2, 0.15 * a.iterations), prec

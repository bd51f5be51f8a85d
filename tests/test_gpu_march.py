"""The marched operator (one pass over 30 x 14 node tiles along z, in reflection modes) against the oracle's
product and against the one-thread-per-node operator, at the sizes where its tiles, planes and chunks
end, forced onto every level whatever its size (PSFEA_TILE_MIN_NODES=0)."""
import numpy as np
import pytest
import torch

import oracle
import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def graded(dims, seed, empty):
    """Densities in [0.05, 1] with a share of empty voxels; the x = 0 face held, one node elsewhere held in y only."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    d = rng.uniform(0.05, 1.0, (nz, ny, nx)).astype(np.float32)
    d[rng.uniform(size=d.shape) < empty] = 0
    d[:, :, 0] = 1
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    bc[nz, ny, nx, 1] = 1
    held = bc.reshape(-1, 3).max(axis=1)
    d, _ = W.prune_floating(dims, d.ravel(), held)
    return d, bc.ravel()


# voxel counts: node counts at and beside multiples of 30 (x) and 14 (y), one and few planes, a column cut into chunks
SIZES = [(29, 13, 5), (30, 14, 1), (28, 12, 2), (59, 27, 9), (60, 28, 3), (61, 29, 4), (3, 2, 70), (31, 1, 1), (1, 15, 33), (90, 5, 7)]


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("empty", [0.0, 0.35])
def test_product_matches_the_oracle(monkeypatch, dims, empty):
    """FP64 y = K x (raw and with held DOFs 0), x and y nonzero everywhere, also with a diagonal shift: sums of some hundred
    terms, so 1e-12 of the result's norm."""
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "0")
    d, bc = graded(dims, sum(dims), empty)
    rng = np.random.default_rng(5)
    for shift in (None, rng.uniform(0.0, 0.5, bc.size)):
        S = psfea.VoxelFEA(dims, d, 0.3, bc, 50, diag_add=shift)
        P = oracle.OracleModel("port", dims, d, 0.3, bc, 50, diag_add=shift)
        x = rng.standard_normal(bc.size)
        for raw in (False, True):
            assert rel(S.apply(x, raw=raw), P.apply(x, raw=raw)) < 1e-12, (shift is None, raw)
        # the allocation-free product on the caller's dense vectors: the same y, 0 at held DOFs and off the part, and x . y
        y0 = P.apply(x)
        xd, yd, dd = torch.from_numpy(x).cuda(), torch.full((x.size,), float("nan"), dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
        for _ in range(2):
            S.apply_dot_noalloc(xd.data_ptr(), yd.data_ptr(), dd.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rel(yd.cpu().numpy(), y0) < 1e-12
        assert np.all(yd.cpu().numpy()[P.fixed(0) != 0] == 0)
        assert abs(float(dd[0]) - float(x @ y0)) < 1e-12 * float(np.abs(x * y0).sum())


def blocky(dims, seed):
    """Graded densities with two rectangular openings (no hinges)."""
    d, bc = graded(dims, seed, 0.0)
    nx, ny, nz = dims
    v = d.reshape(nz, ny, nx)
    v[:, ny // 3:ny // 2, nx // 4:nx // 2] = 0
    v[nz // 2:, :ny // 4, nx // 2:3 * nx // 4] = 0
    d, _ = W.prune_floating(dims, d, bc.reshape(-1, 3).max(axis=1))
    return d, bc


@pytest.mark.parametrize("dims", [(59, 27, 9), (61, 29, 12), (30, 44, 17)])
@pytest.mark.parametrize("inner,split", [("1", "0"), ("0", "-1")])
def test_smoother_residual_and_steps_match_the_node_kernels(monkeypatch, dims, inner, split):
    """The V-cycle (smoother and residual passes, levels with own matrices too, whose nodes go to the list kernels) and
    solves in every form, marched against one thread per node: the FP32 sums run in another order (1e-5 for a V-cycle of
    some ten passes at 1e-6 each); the solves agree to their tolerance."""
    d, bc = blocky(dims, 3)
    monkeypatch.setenv("PSFEA_TILE_INNER64", inner)
    monkeypatch.setenv("PSFEA_TILE_SPLIT32", split)
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "1000000000")
    A = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "0")
    B = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
    assert A.n_levels >= 3
    rng = np.random.default_rng(7)
    for l in range(A.n_levels):
        x = rng.standard_normal(A.level_info(l)["nDof"])
        assert rel(B.apply(x, level=l), A.apply(x, level=l)) < 1e-12, l
    # a load with a share in the softest modes, which dominate z: the relative error is then a few FP32 roundings a pass
    # (on a vector K x without them it is those roundings times the V-cycle's norm, 1e-6 to 1e-4 in either form)
    r = rng.standard_normal(A.n_dof) * (A.fixed(0) == 0)
    assert rel(B.precondition(r), A.precondition(r)) < 1e-5
    f = W._face_load(dims, d, 0, 1, (1.0, -2.0, 0.5))[0]
    for prec in ("half", "fp64", "mixed", "fp32"):
        for deg in (0, 1):
            a = A.solve(f, tol=1e-9, max_iter=3000, precision=prec, smoother_degree=deg)
            b = B.solve(f, tol=1e-9, max_iter=3000, precision=prec, smoother_degree=deg)
            assert a.converged and b.converged, (prec, deg)
            assert rel(b.u, a.u) < 1e-5, (prec, deg, rel(b.u, a.u))
            if deg == 0:  # (one smoothing step: the count jumps between 46 and 58 with a load moved by 1e-7, in either form)
                assert abs(a.iterations - b.iterations) <= max(2, 0.15 * a.iterations), (prec, deg)
    # whatever ran before on the handle, a solve gives what a fresh handle gives
    C = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
    c = C.solve(f, tol=1e-9, max_iter=3000, precision="fp32", smoother_degree=1)
    assert c.iterations == b.iterations and np.array_equal(c.u, b.u)


def test_empty_voxels_do_not_carry_infinities():
    """y = K x where x is infinite at one node: only the nodes that share a solid voxel with it see it."""
    import os
    os.environ["PSFEA_TILE_MIN_NODES"] = "0"
    try:
        dims = (33, 16, 6)
        d, bc = graded(dims, 11, 0.6)
        S = psfea.VoxelFEA(dims, d, 0.3, bc, 50)
    finally:
        del os.environ["PSFEA_TILE_MIN_NODES"]
    nx, ny, nz = dims
    s = np.asarray(d).reshape(nz, ny, nx) > 0
    i, j, k = 20, 8, 3
    x = np.random.default_rng(2).standard_normal(bc.size).reshape(nz + 1, ny + 1, nx + 1, 3)
    ref = S.apply(x.ravel(), raw=True).reshape(x.shape)
    x[k, j, i, 1] = np.inf
    y = S.apply(x.ravel(), raw=True).reshape(x.shape)
    touched = np.zeros(x.shape[:3], bool)
    for dk in (-1, 0):
        for dj in (-1, 0):
            for di in (-1, 0):
                if s[k + dk, j + dj, i + di]:
                    touched[k + dk:k + dk + 2, j + dj:j + dj + 2, i + di:i + di + 2] = True
    assert np.array_equal(~np.isfinite(y).all(axis=-1), touched)
    assert np.array_equal(y[~touched], ref[~touched])


@pytest.mark.parametrize("dims", [(13, 9, 7), (30, 44, 17), (48, 20, 24)])
@pytest.mark.parametrize("shift", [False, True])
def test_small_levels_stencils_match_the_gather(monkeypatch, dims, shift):
    """The small Galerkin levels' eight-lane stencils (level node counts that leave part of a warp, one and several blocks, with
    and without a diagonal shift) against the per-voxel gather (PSFEA_STENCIL_LEVELS=0): the V-cycle of a load to a few FP32
    roundings a pass, and solves in every form."""
    d, bc = blocky(dims, 4)
    rng = np.random.default_rng(1)
    add = rng.uniform(0.0, 0.2, bc.size) if shift else None
    monkeypatch.setenv("PSFEA_STENCIL_LEVELS", "0")
    A = psfea.VoxelFEA(dims, d, 0.3, bc, 60, diag_add=add)
    monkeypatch.delenv("PSFEA_STENCIL_LEVELS")
    B = psfea.VoxelFEA(dims, d, 0.3, bc, 60, diag_add=add)
    assert A.n_levels >= 3
    f = rng.standard_normal(A.n_dof) * (A.fixed(0) == 0)
    for prec in ("fp64", "mixed", "fp32"):
        for deg in (0, 3):
            a = A.solve(f, tol=1e-9, max_iter=3000, precision=prec, smoother_degree=deg)
            b = B.solve(f, tol=1e-9, max_iter=3000, precision=prec, smoother_degree=deg)
            assert a.converged and b.converged and rel(b.u, a.u) < 1e-5, (prec, deg)
    assert rel(B.precondition(f), A.precondition(f)) < 1e-5


@pytest.mark.parametrize("dims", [(29, 17, 13), (30, 18, 9), (61, 35, 8), (31, 36, 20)])
def test_tall_tiles_match_the_low_ones(monkeypatch, dims):
    """32-bit tiles of 18 output rows against those of 14, at node rows of one tile, one more, two tiles and one more: the
    same sums per node (1e-5 for a V-cycle as above), and solves that agree to their tolerance."""
    d, bc = blocky(dims, 5)
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "0")
    monkeypatch.setenv("PSFEA_MARCH_TALL", "0")
    A = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
    monkeypatch.setenv("PSFEA_MARCH_TALL", "1")
    B = psfea.VoxelFEA(dims, d, 0.3, bc, 300)
    r = np.random.default_rng(9).standard_normal(A.n_dof) * (A.fixed(0) == 0)
    assert rel(B.precondition(r), A.precondition(r)) < 1e-5
    f = W._face_load(dims, d, 0, 1, (1.0, -2.0, 0.5))[0]
    for prec in ("half", "mixed", "fp32"):
        a = A.solve(f, tol=1e-9, max_iter=3000, precision=prec)
        b = B.solve(f, tol=1e-9, max_iter=3000, precision=prec)
        assert a.converged and b.converged, prec
        assert rel(b.u, a.u) < 1e-5, (prec, rel(b.u, a.u))

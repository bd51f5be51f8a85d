"""What the device gets when a model is new: the tile lists made from one bit a node, and no list that nothing reads."""
import numpy as np
import pytest

import oracle
import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def islands(dims, seed):
    """Mostly empty: bars from the held face x = 0 of one to three voxels' width, some of them short, so that tiles, rows and planes
    are active, empty and cut in every combination."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    d = np.zeros((nz, ny, nx), np.float32)
    for _ in range(6):
        j, k, w = rng.integers(ny), rng.integers(nz), rng.integers(1, 4)
        d[k:k + w, j:j + w, :rng.integers(1, nx + 1)] = rng.uniform(0.1, 1.0)
    bc = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.uint8)
    bc[:, :, 0] = 1
    return d.ravel(), bc.ravel()


# node rows of one to four 64-bit words, ends at and beside a word's and a tile's (30 nodes)
@pytest.mark.parametrize("dims", [(62, 9, 5), (63, 9, 5), (64, 20, 4), (119, 12, 9), (128, 7, 3), (191, 11, 30), (240, 3, 2)])
def test_products_of_sparse_grids_match_the_oracle(monkeypatch, dims):
    monkeypatch.setenv("PSFEA_TILE_MIN_NODES", "0")
    d, bc = islands(dims, sum(dims))
    S = psfea.VoxelFEA(dims, d, 0.3, bc, 50)
    P = oracle.OracleModel("port", dims, d, 0.3, bc, 50)
    x = np.random.default_rng(1).standard_normal(bc.size)
    for raw in (False, True):
        y, yo = S.apply(x, raw=raw), P.apply(x, raw=raw)
        assert np.linalg.norm(y - yo) <= 1e-12 * np.linalg.norm(yo), raw  # (FP64 sums of some hundred terms)


def test_boundary_list_only_where_a_split_reads_it(monkeypatch):
    """The list of every node that is not uniform (4 B a node: a third of this graded model's 73,205 nodes and more) is
    made for the splits and the autotuner only; with it the solves are the same."""
    m = W.simp(60, 30, 38, nrhs=1)
    f = m.f if m.f.ndim == 1 else m.f[0]

    def make():
        return psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)

    A = make()
    monkeypatch.setenv("PSFEA_TILE_INNER64", "0")
    monkeypatch.setenv("PSFEA_TILE_SPLIT32", "-1")
    B = make()
    monkeypatch.delenv("PSFEA_TILE_INNER64")
    monkeypatch.delenv("PSFEA_TILE_SPLIT32")
    assert A.device_bytes + 4 * 20000 < B.device_bytes
    a, b = (S.solve(f, tol=1e-9, max_iter=2000) for S in (A, B))
    assert a.converged and b.converged
    assert np.linalg.norm(a.u - b.u) <= 1e-6 * np.linalg.norm(b.u)
    before = A.device_bytes
    A.autotune(f, tol=1e-8, max_iter=2000, force=True)  # tries the splits
    assert A.device_bytes >= before + 4 * 20000
    c = A.solve(f, tol=1e-9, max_iter=2000)
    assert c.converged and np.linalg.norm(c.u - b.u) <= 1e-6 * np.linalg.norm(b.u)

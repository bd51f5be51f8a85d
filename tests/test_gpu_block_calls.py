"""Calls of the block preconditioner that the GPU has not begun to run when the next one is made (they return without
waiting): each has to keep its own count of vectors."""
import numpy as np
import pytest
import torch

import psfea
import voxel_models as W

pytestmark = pytest.mark.gpu


def busy(stream):
    """Queues some 100 ms of work on the stream (1 GB read and written at a time)."""
    a = torch.zeros(1 << 28, device="cuda")
    with torch.cuda.stream(stream):
        for _ in range(300):
            a.add_(1.0)
    return a


def vectors(S, n, seed):
    """n residual-like vectors: free DOFs random, held ones 0"""
    r = np.random.default_rng(seed).standard_normal((n, S.n_dof)) * (S.fixed(0) == 0)
    return torch.from_numpy(r).cuda()


def one_by_one(S, r):
    z = torch.full_like(r, float("nan"))
    for k in range(r.shape[0]):
        S.precondition_block(1, r[k].data_ptr(), z[k].data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    return z


@pytest.mark.parametrize("nvec", [33, 40])
def test_more_vectors_than_a_block_holds(nvec):
    """A block of 32 and a remainder, behind other work on the caller's stream. Every vector's V-cycle is computed by itself
    and in a fixed order, so the result is that of one call a vector, to the bit."""
    m = W.cantilever(20, 9, 7, coarsest_max_dof=300)
    S = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    r = vectors(S, nvec, 1)
    s = torch.cuda.Stream()
    z = torch.full_like(r, float("nan"))
    S.precondition_block(nvec, r.data_ptr(), z.data_ptr(), s.cuda_stream)  # (the block is made here)
    torch.cuda.synchronize()
    z.fill_(float("nan"))
    torch.cuda.synchronize()
    keep = busy(s)
    S.precondition_block(nvec, r.data_ptr(), z.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    want = one_by_one(S, r)
    assert torch.equal(z, want) and bool((want.abs().amax(dim=1) > 0).all())
    del keep


def test_calls_one_behind_the_other():
    """Calls of 6, 2 and 5 vectors and a block solve, all made before the first has begun."""
    m = W.cantilever(20, 9, 7, coarsest_max_dof=300)
    S = psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof)
    counts = (6, 2, 5)
    rs = [vectors(S, n, n) for n in counts]
    want = [one_by_one(S, r) for r in rs]
    alone = S.solve_batch(np.stack([m.f, 2 * m.f]), tol=1e-8, max_iter=300)
    zs = [torch.full_like(r, float("nan")) for r in rs]
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    keep = busy(s)
    for n, r, z in zip(counts, rs, zs):
        S.precondition_block(n, r.data_ptr(), z.data_ptr(), s.cuda_stream)
    after = S.solve_batch(np.stack([m.f, 2 * m.f]), tol=1e-8, max_iter=300)
    torch.cuda.synchronize()
    for z, w in zip(zs, want):
        assert torch.equal(z, w)
    for a, b in zip(after, alone):
        assert a.iterations == b.iterations and np.array_equal(a.u, b.u)
    del keep


@pytest.mark.parametrize("degree", [1, 4])
def test_smoother_degree_of_the_call_not_of_the_one_before(degree):
    """A block made before a solve at another smoother degree: the block preconditioner is the reference's degree 2 again, and a
    block solve has its own degree, both as on a handle of their own."""
    m = W.l_bracket(40, 20, 20, holes=4, seed=2)
    F = np.stack([m.f, -2 * m.f])
    S, T = (psfea.VoxelFEA(m.dims, m.density, m.nu, m.bc, m.coarsest_max_dof) for _ in range(2))
    r = vectors(S, 3, 9)
    want = one_by_one(S, r)
    S.solve(m.f, tol=1e-6, max_iter=2000, smoother_degree=degree)
    assert torch.equal(one_by_one(S, r), want)
    S.solve(m.f, tol=1e-6, max_iter=2000, smoother_degree=degree)
    for a, b in zip(S.solve_batch(F, tol=1e-8, max_iter=2000), T.solve_batch(F, tol=1e-8, max_iter=2000)):
        assert a.iterations == b.iterations and np.array_equal(a.u, b.u)

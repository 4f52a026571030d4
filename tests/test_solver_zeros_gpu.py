"""FP64 solves of matrices whose pattern stores exact zeros (the solver drops them): slice remainders, sizes on
both sides of the layout's limit, and values changed in place between two solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triplets(nodes, coupled, seed):
    """SPD banded system of 6 DOFs per node; uncoupled: (0, 1, 5) and (2, 3, 4) do not couple."""
    rng = np.random.default_rng(seed)
    n = 6 * nodes
    g = np.array([0, 0, 1, 1, 1, 0])
    keep = np.ones((6, 6), bool) if coupled else g[:, None] == g[None, :]
    r, c, v = [np.arange(n)], [np.arange(n)], [np.full(n, 1.)]
    i, j = np.meshgrid(np.arange(6), np.arange(6), indexing='ij')
    for d in range(3):
        a = np.arange(max(nodes - d, 0))
        blk = rng.normal(size=(a.size, 6, 6)) * keep
        rr, cc = 6 * a[:, None, None] + i, 6 * (a[:, None, None] + d) + j
        r += [rr.ravel(), cc.ravel()]
        c += [cc.ravel(), rr.ravel()]
        v += [blk.ravel(), blk.ravel()]
    r, c, v = (np.concatenate(t) for t in (r, c, v))
    np.add.at(v, r, np.abs(v))  # diagonally dominant (the first n slots are the diagonal)
    return r, c, v


@pytest.mark.parametrize('nodes', [1, 5, 6, 11, 16, 171, 2730, 2731, 3001])
@pytest.mark.parametrize('coupled', [False, True])
def test_solve_with_stored_zeros(gpulib, nodes, coupled):
    import torch
    from scipy.sparse.linalg import spsolve
    from pyfe3d_gb300.solver import CSRPattern, Solver
    r, c, v = _triplets(nodes, coupled, nodes)
    pat = CSRPattern(r, c, 6 * nodes, None)
    assert pat.nnz == 36 * sum(min(nodes, a + 3) - max(0, a - 2) for a in range(nodes))
    vals = pat.assemble(v)
    s = Solver(pat).setup(vals)
    f = np.random.default_rng(1).normal(size=6 * nodes)
    for _ in range(2):  # the second solve sees values changed in place, one more of them non-zero
        u, st = s.solve(torch.from_numpy(f).cuda(), tol=1e-13, check_every=2)
        assert st['status'] == 'converged'
        ref = spsolve(pat.to_scipy(vals).tocsc(), f)
        assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)  # condition number below 100
        v = 3. * v
        v[((r == 0) & (c == 8)) | ((r == 8) & (c == 0))] = 0.25
        pat.assemble(v, out=vals)

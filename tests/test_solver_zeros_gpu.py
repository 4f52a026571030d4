"""FP64 solves of matrices whose pattern stores exact zeros (the solver drops them), resident and launch by launch:
remainders of blocks and slices, sizes on both sides of the layouts' limits, and values changed in place between two
solves."""
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
@pytest.mark.parametrize('flexible', [False, True])  # flexible CG runs launch by launch
def test_solve_with_stored_zeros(gpulib, nodes, coupled, flexible):
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
        u, st = s.solve(torch.from_numpy(f).cuda(), tol=1e-13, check_every=2, flexible=flexible)
        assert st['status'] == 'converged'
        ref = spsolve(pat.to_scipy(vals).tocsc(), f)
        assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)  # condition number below 100
        v = 3. * v
        v[((r == 0) & (c == 8)) | ((r == 8) & (c == 0))] = 0.25
        pat.assemble(v, out=vals)


@pytest.mark.parametrize('nodes', [40, 5000])
@pytest.mark.parametrize('order', ['shuffled', 'fixed'])
def test_numbering_and_partial_nodes(gpulib, nodes, order):
    """Nodes in random order (5000: a block's columns no longer fit shared memory) and nodes with fixed DOFs."""
    import torch
    from scipy.sparse.linalg import spsolve
    from pyfe3d_gb300.solver import CSRPattern, Solver
    rng = np.random.default_rng(7)
    r, c, v = _triplets(nodes, False, 3)
    bk = None
    if order == 'shuffled':
        perm = rng.permutation(nodes)
        r, c = 6 * perm[r // 6] + r % 6, 6 * perm[c // 6] + c % 6
    else:
        bk = rng.random(6 * nodes) < 0.3
        bk[60:90] = True
    pat = CSRPattern(r, c, 6 * nodes, bk)
    vals = pat.assemble(v)
    s = Solver(pat).setup(vals)
    f = rng.normal(size=pat.nrows)
    u, st = s.solve(torch.from_numpy(f).cuda(), tol=1e-13)
    assert st['status'] == 'converged'
    ref = spsolve(pat.to_scipy(vals).tocsc(), f)
    assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)
    # few iterations and a restart from their iterate: the same recurrence cut short
    u1, st1 = s.solve(torch.from_numpy(f).cuda(), tol=1e-300, maxiter=5, check_every=2)
    assert st1['iterations'] == 5
    u2, st2 = s.solve(torch.from_numpy(f).cuda(), u0=u1, tol=1e-13, check_every=7)
    assert st2['status'] == 'converged'
    assert np.linalg.norm(u2.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize('nodes', [2731, 2752, 9001])
@pytest.mark.parametrize('coupled', [False, True])
def test_row_wise_update(gpulib, nodes, coupled):
    """Launch-by-launch FP64 iterations (a system whose columns reach too far for resident blocks): chunks of nodes with
    fixed DOFs and of whole nodes, from zero and from a given iterate."""
    import torch
    from scipy.sparse.linalg import spsolve
    from pyfe3d_gb300.solver import CSRPattern, Solver
    rng = np.random.default_rng(nodes)
    r, c, v = _triplets(nodes, coupled, 5)
    # a weak coupling of the first and the last node widens every window beyond shared memory when n is large
    far = np.array([0, 6 * nodes - 6])
    r, c, v = np.concatenate([r, far, far[::-1]]), np.concatenate([c, far, far]), np.concatenate([v, [1., 1., .1, .1]])
    bk = rng.random(6 * nodes) < 0.15
    bk[far] = False
    bk[600:900] = True
    perm = rng.permutation(nodes)
    r, c = 6 * perm[r // 6] + r % 6, 6 * perm[c // 6] + c % 6
    pat = CSRPattern(r, c, 6 * nodes, bk)
    vals = pat.assemble(v)
    s = Solver(pat).setup(vals)
    f = rng.normal(size=pat.nrows)
    ref = spsolve(pat.to_scipy(vals).tocsc(), f)
    fd = torch.from_numpy(f).cuda()
    u, st = s.solve(fd, tol=1e-13)
    assert st['status'] == 'converged'
    assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)
    u1, _ = s.solve(fd, tol=1e-300, maxiter=4, check_every=2)
    u2, st2 = s.solve(fd, u0=u1, tol=1e-13)
    assert st2['status'] == 'converged'
    assert np.linalg.norm(u2.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)
    vals[5] = float('nan')
    _, st3 = s.solve(fd, tol=1e-13, maxiter=100)
    assert st3['status'] == 'non-finite'


@pytest.mark.parametrize('nodes', [40, 400, 5000])
def test_rows_without_entries(gpulib, nodes):
    """Nodes that no element meets: their rows are empty and their unloaded DOFs stay zero."""
    import torch
    from scipy.sparse.linalg import spsolve
    from pyfe3d_gb300.solver import CSRPattern, Solver
    r, c, v = _triplets(nodes, True, 3)
    alone = np.zeros(nodes, bool)
    alone[[nodes // 2, nodes // 2 + 1, nodes - 9, nodes - 1]] = True
    keep = ~(alone[r // 6] | alone[c // 6])
    pat = CSRPattern(r[keep], c[keep], 6 * nodes, None)
    vals = pat.assemble(v[keep])
    f = np.random.default_rng(1).normal(size=6 * nodes)
    free = np.repeat(~alone, 6)
    f[~free] = 0.
    u, st = Solver(pat).setup(vals).solve(torch.from_numpy(f).cuda(), tol=1e-13, check_every=2)
    assert st['status'] == 'converged'
    u = u.cpu().numpy()
    assert (u[~free] == 0.).all()
    ref = spsolve(pat.to_scipy(vals).tocsr()[free][:, free].tocsc(), f[free])
    assert np.linalg.norm(u[free] - ref) <= 1e-11 * np.linalg.norm(ref)  # condition number below 100


@pytest.mark.parametrize('nodes', [1, 2, 40, 700])
@pytest.mark.parametrize('exponent', [-300, 0, 300])
def test_residual_that_drops_at_once(gpulib, nodes, exponent):
    """Uncoupled nodes: the preconditioner is the inverse, the first iteration leaves rounding and the others of the
    check interval run on it."""
    import torch
    from pyfe3d_gb300.solver import CSRPattern, Solver
    r, c, v = _triplets(nodes, True, 3)
    keep = r // 6 == c // 6
    pat = CSRPattern(r[keep], c[keep], 6 * nodes, None)
    vals = pat.assemble(v[keep])
    f = torch.from_numpy(np.random.default_rng(1).normal(size=6 * nodes)).cuda() * 2. ** exponent
    for check in (2, 50, 1000):
        u, st = Solver(pat).setup(vals).solve(f, tol=1e-12, check_every=check)
        assert st['status'] == 'converged' and st['relres'] <= 1e-12
        assert torch.isfinite(u).all()

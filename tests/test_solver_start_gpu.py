"""The first residual of launch-per-kernel FP64 solves: f where the guess is zero, f - K u0 where any entry of it is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nodes', [2731, 3001, 40000])  # 16384 rows and more, the last warp partly filled
def test_one_non_zero_in_the_guess(gpulib, nodes):
    """Uncoupled nodes: the preconditioner is the inverse, one iteration from the right residual is the solution,
    which the compensated residual f - K u confirms; from a wrong one it is not."""
    import torch
    from pyfe3d_gb300.solver import CSRPattern, Solver
    rng = np.random.default_rng(nodes)
    n = 6 * nodes
    blk = rng.normal(size=(nodes, 6, 6))
    blk = blk + blk.transpose(0, 2, 1) + 20. * np.eye(6)
    d = np.arange(n).reshape(nodes, 6)
    # (next to the blocks exact zeros, which the solver leaves out)
    r = np.concatenate([np.repeat(d, 6, 1).ravel(), np.repeat(d[:-1], 6, 1).ravel()])
    c = np.concatenate([np.tile(d, (1, 6)).ravel(), np.tile(d[1:], (1, 6)).ravel()])
    pat = CSRPattern(r, c, n, None)
    vals = pat.assemble(np.concatenate([blk.ravel(), np.zeros(36 * (nodes - 1))]))
    s = Solver(pat).setup(vals)
    f = torch.from_numpy(rng.normal(size=n)).cuda()
    for at in (None, 0, 1, 31, 33, n // 2, n - 23, n - 2, n - 1):
        u0 = torch.zeros_like(f)
        if at is not None:
            u0[at] = 1e3
        _, st = s.solve(f, u0=u0, tol=1e-12, maxiter=1, check_every=2, flexible=True)
        assert st['status'] == 'converged' and st['iterations'] == 1, at

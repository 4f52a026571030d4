"""Batched solves on teams of blocks: more instances than blocks, one instance far larger than the others, iteration
caps and initial guesses, against the lockstep recurrence (which a work split of no instance selects)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(sizes, seed):
    import torch
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.meshes import BatchedPlates
    from pyfe3d_gb300.solver import ElementPattern, FusedMap
    rng = np.random.default_rng(seed)
    nx, ny = np.array(sizes).T
    P = len(sizes)
    bp = BatchedPlates.__new__(BatchedPlates)
    bp._build(nx, ny, rng.uniform(0.5, 2., P), rng.uniform(0.5, 2., P), rng.uniform(5e10, 2e11, P),
              rng.uniform(0.25, 0.35, P), rng.uniform(0.005, 0.02, P), rng.integers(0, 2, P).astype(bool))
    pat = ElementPattern([bp.cdof], bp.N, bp.bk)
    fmap = FusedMap(pat, [bp.cdof])
    vals = batch.quad4_update_KC0_csr(fmap.new_values(), fmap, bp.x, bp.props, pid=bp.pid)
    f = torch.from_numpy(bp.f).cuda()
    return bp, pat, vals, pat.reduce(f)


@pytest.mark.parametrize('sizes', [[(3, 3)], [(2, 5), (60, 40)], [(2 + i % 5, 3 + i % 4) for i in range(200)],
                                   [(50, 50)] + [(4, 4 + i % 3) for i in range(160)],
                                   [(260, 30), (30, 260), (150, 150), (140, 180), (250, 60), (200, 90)]], ids=['one', 'two', 'many', 'uneven', 'long'])
def test_teams_match_lockstep(gpulib, sizes):
    from pyfe3d_gb300.solver import BatchSolver
    bp, pat, vals, f = _batch(sizes, len(sizes))
    teams = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)
    lock = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)
    assert lock.set_split(1) == 0
    u, st = teams.solve(f, tol=1e-10)
    v, sl = lock.solve(f, tol=1e-10)
    assert (st['inst_status'] == 0).all() and (sl['inst_status'] == 0).all()
    assert (st['inst_relres'] <= 1e-10).all()
    inst = teams.inst_of_row.cpu().numpy()
    d, w = (u - v).cpu().numpy(), v.cpu().numpy()
    err = np.sqrt(np.bincount(inst, d * d) / np.bincount(inst, w * w))
    assert err.max() <= 1e-7, err.max()
    # the same recurrence: the iteration counts agree up to rounding and the check interval
    assert (abs(st['inst_iters'] - sl['inst_iters']) <= 100 + 0.05 * sl['inst_iters']).all()
    # a cap ends every unfinished instance there; its iterate continues
    u1, s1 = teams.solve(f, tol=1e-10, maxiter=30, check_every=20)
    assert s1['inst_iters'].max() <= 30 and (s1['inst_iters'][s1['inst_status'] == 1] == 30).all()
    u2, s2 = teams.solve(f, u0=u1, tol=1e-10)
    assert (s2['inst_status'] == 0).all()
    # nothing left to do
    _, s3 = teams.solve(f, u0=u2, tol=1e-9)
    assert (s3['inst_status'] == 0).all() and s3['inst_iters'].max() == 0


@pytest.mark.parametrize('size', [(2, 3), (9, 8), (40, 31)], ids=str)
@pytest.mark.parametrize('exponent', [-475, -240, 0, 240, 480])
def test_loads_of_any_scale(gpulib, size, exponent):
    """Inner products near both ends of the range of a double (their sums over lanes and blocks are made in fixed
    point, next to those ends by plain additions): the solution scales with the load."""
    from pyfe3d_gb300.solver import Solver
    _, pat, vals, f = _batch([size], 3)
    s = Solver(pat).setup(vals)
    u, st = s.solve(f, tol=1e-10)
    v, sv = s.solve(f * 2. ** exponent, tol=1e-10)
    assert st['status'] == sv['status'] == 'converged' and sv['relres'] <= 1e-10
    w = v * 2. ** -exponent
    assert ((w - u).norm() <= 1e-7 * u.norm()).item()


@pytest.mark.parametrize('size', [(3, 2), (21, 20), (75, 74), (126, 125), (133, 131), (244, 240)], ids=str)
def test_rows_in_shared_memory_and_streamed(gpulib, size):
    """Blocks that keep their rows in shared memory (up to and above a row per thread), read them from L2 and load
    them ahead: the recurrence's residual is confirmed by the compensated residual f - K u, which is evaluated by
    other kernels (a wrong product would part the two)."""
    from pyfe3d_gb300.solver import Solver
    _, pat, vals, f = _batch([size], 5)
    s = Solver(pat).setup(vals)
    _, st = s.solve(f, tol=1e-8)
    assert st['status'] == 'converged' and st['relres'] <= 1e-8

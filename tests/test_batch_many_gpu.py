"""Batches of many tiny instances: in lockstep until few enough are left, on teams of blocks from there on, against the
lockstep recurrence throughout (which a work split of no instance selects)."""
import time

import numpy as np
import pytest
from test_batch_teams_gpu import _batch

pytestmark = pytest.mark.gpu

TINY = [(2 + i % 3, 2 + i // 3 % 3) for i in range(900)]


def _solvers(bp, pat, vals):
    from pyfe3d_gb300.solver import BatchSolver
    a = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)
    b = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)
    assert b.set_split(1) == 0
    return a, b


@pytest.mark.parametrize('sizes', [TINY, TINY + [(40, 40)], [(30, 8)] + TINY[:450] + [(9, 50)] + TINY[450:] + [(20, 20)],
                                   TINY[:500], TINY[:560]], ids=['tiny', 'one large', 'three large', '500', '560'])
def test_many_match_lockstep(gpulib, sizes):
    bp, pat, vals, f = _batch(sizes, len(sizes))
    many, lock = _solvers(bp, pat, vals)
    inst = many.inst_of_row.cpu().numpy()
    for check in (50, 7):
        u, st = many.solve(f, tol=1e-10, check_every=check)
        v, sl = lock.solve(f, tol=1e-10, check_every=check)
        assert (st['inst_status'] == 0).all() and (sl['inst_status'] == 0).all()
        d, w = (u - v).cpu().numpy(), v.cpu().numpy()
        assert np.sqrt(np.bincount(inst, d * d) / np.bincount(inst, w * w)).max() <= 1e-7
        # the same recurrence: the iteration counts agree up to rounding and the check interval
        assert (abs(st['inst_iters'] - sl['inst_iters']) <= 100 + 0.05 * sl['inst_iters']).all()
    # caps before and after the change of route end every unfinished instance there; its iterate continues
    for cap in (5, 30, 150):
        u1, s1 = many.solve(f, tol=1e-10, maxiter=cap, check_every=20)
        assert s1['inst_iters'].max() <= cap and (s1['inst_iters'][s1['inst_status'] == 1] == cap).all()
        u2, s2 = many.solve(f, u0=u1, tol=1e-10)
        assert (s2['inst_status'] == 0).all()
    _, s3 = many.solve(f, u0=u2, tol=1e-9)
    assert (s3['inst_status'] == 0).all() and s3['inst_iters'].max() == 0


def test_many_take_no_longer_than_in_lockstep(gpulib):
    """5,400 plates of 9 to 25 nodes: 3.4 times the lockstep time when all are solved on teams."""
    import torch
    many, lock = _solvers(*(s := _batch(6 * TINY, 1))[:3])

    def best(b):
        ms = []
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _, st = b.solve(s[3], tol=1e-8)
            torch.cuda.synchronize()
            ms.append(time.perf_counter() - t)
        assert (st['inst_status'] == 0).all()
        return min(ms)
    assert best(many) <= 2. * best(lock)

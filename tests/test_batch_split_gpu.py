"""Where the block-resident batched solver stops."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def split(gpulib):
    """64 small plates, each on a block of its own: (solve, right-hand side)."""
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.meshes import BatchedPlates
    from pyfe3d_gb300.solver import BatchSolver, ElementPattern, FusedMap
    bp = BatchedPlates(64, 4, 12, 4)
    pat = ElementPattern([bp.cdof], bp.N, bp.bk)
    fmap = FusedMap(pat, [bp.cdof])
    vals = batch.quad4_update_KC0_csr(fmap.new_values(), fmap, bp.x, bp.props, pid=bp.pid)
    bs = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)
    assert bs.set_split(1100) == bp.P
    return bs.solve, pat.reduce(bp.f)


def test_a_looser_tolerance_takes_no_more_iterations(split):
    """Far above the rounding of the residual, the iterations for one tolerance are the first ones for a tighter one; an
    iterate that meets the tolerance is not restarted."""
    solve, f = split
    last = np.zeros(64, np.int64)
    for tol in 1e-4 * 0.97 ** np.arange(12):
        _, st = solve(f, tol=tol)
        assert (st['inst_status'] == 0).all() and (st['inst_relres'] <= tol).all()
        assert (st['inst_iters'] >= last).all(), tol
        last = st['inst_iters'].copy()


def test_tolerance_met_at_the_cap(split):
    """An iterate at the iteration cap counts as converged whenever it meets the tolerance."""
    solve, f = split
    for cap in (40, 41, 42, 43):
        _, st = solve(f, tol=1e-300, maxiter=cap)
        assert (st['inst_iters'] == cap).all()
        tol = float(np.median(st['inst_relres'])) * (1. + 1e-6)
        _, again = solve(f, tol=tol, maxiter=cap)
        met = again['inst_relres'] <= tol * (1. - 1e-5)
        assert met.any() and (again['inst_status'][met] == 0).all()

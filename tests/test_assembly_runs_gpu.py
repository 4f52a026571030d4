"""Numeric assembly by runs of entries: element blocks of 1 to 6 DOFs a node, nodes with 1 to 9 elements, fixed DOFs,
odd slot offsets, and patterns without runs, against scipy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(rng, nodes, E, nn, dof):
    conn = np.stack([rng.choice(nodes, nn, replace=False) for _ in range(E)])
    d = (dof * conn[:, :, None] + np.arange(dof)).reshape(E, -1)
    n = nn * dof
    return np.repeat(d, n, 1).ravel(), np.tile(d, (1, n)).ravel()


@pytest.mark.parametrize('nodes,E,nn,dof', [(2, 1, 2, 6), (5, 9, 4, 6), (40, 60, 3, 6), (300, 900, 4, 6),
                                            (60, 80, 2, 3), (50, 70, 4, 1), (1200, 1100, 4, 6)])
@pytest.mark.parametrize('fixed', [0., 0.3])
@pytest.mark.parametrize('lead', [0, 1])
def test_assembly_matches_scipy(gpulib, nodes, E, nn, dof, fixed, lead):
    import torch
    from scipy.sparse import coo_matrix
    from pyfe3d_gb300.solver import CSRPattern
    rng = np.random.default_rng(nodes + E)
    r, c = _blocks(rng, nodes, E, nn, dof)
    if lead:  # slots shifted by one: no 16-byte loads
        r, c = np.concatenate([[0], r]), np.concatenate([[0], c])
    v = rng.normal(size=r.size)
    N = nodes * dof
    bk = rng.random(N) < fixed
    pat = CSRPattern(r, c, N, bk)
    for view in (0, 1):  # a value array on and off a 16-byte boundary
        buf = torch.zeros(v.size + 1, dtype=torch.float64, device='cuda')
        kv = buf[view:view + v.size]
        kv.copy_(torch.from_numpy(v))
        A = pat.to_scipy(pat.assemble(kv))
        K = coo_matrix((v, (r, c)), shape=(N, N)).tocsr()[~bk][:, ~bk]
        assert A.shape == K.shape
        if K.nnz:
            assert abs(A - K).max() <= 1e-14 * abs(K).max()

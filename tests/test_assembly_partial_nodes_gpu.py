"""Numeric assembly where only some DOFs of a node are free or stored, so that neighbouring columns of different nodes
come from neighbouring slots: element triplets with single DOFs fixed, triplets of the free DOFs alone and the entries
of a sparse matrix, into an array of NaN, against scipy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(r, c, N, bk, seed=0):
    import torch
    from scipy.sparse import coo_matrix
    from pyfe3d_gb300.solver import CSRPattern
    v = np.random.default_rng(seed).normal(size=r.size)
    pat = CSRPattern(r, c, N, bk)
    out = torch.full((pat.nnz,), float('nan'), dtype=torch.float64, device='cuda')
    A = pat.to_scipy(pat.assemble(v, out=out))
    free = np.ones(N, bool) if bk is None else ~bk

    def reduced(w):
        return coo_matrix((w, (r, c)), shape=(N, N)).tocsr()[free][:, free].toarray()
    K, size, count = reduced(v), reduced(np.abs(v)), reduced(np.ones(v.size))
    A = A.toarray()  # (entries left unwritten stay NaN)
    # two sums of count terms, each within (count - 1) 2^-53 of the sum of their sizes
    assert (np.abs(A - K) <= 2 ** -52 * count * size).all()


def _plate(order, masked):
    """7 x 6 nodes numbered along y or along x, and the constrained DOFs."""
    from pyfe3d_gb300.meshes import PlateMesh
    m = PlateMesh(7, 6, 1., 0.7)
    number = np.arange(m.nnodes)
    if order == 'x':
        number = number.reshape(7, 6).T.ravel().argsort()
    x = np.empty((m.nnodes, 3))
    x[number] = m.ncoords
    edge, right = (np.empty(m.nnodes, bool) for _ in range(2))
    edge[number], right[number] = m.edge, np.isclose(m.ncoords[:, 0], m.a)
    bk = np.zeros(m.N, bool)
    for d, where in {'none': {}, 'u': {0: edge}, 'u of one edge': {0: right}, 'every u': {0: edge | True},
                     'ry and rz': {4: edge, 5: right}, 'bending': {d: edge | True for d in (0, 1, 5)}}[masked].items():
        bk[d::6] = where
    return 6 * number[m.conn], x.ravel(), m.N, bk


@pytest.mark.parametrize('kind', ['q4 m 0', 'q4 m 1', 'q4 m 2', 'q4 kg', 'beam m 0', 'beam m 1', 'beam kc0'])
@pytest.mark.parametrize('masked', ['none', 'u', 'u of one edge', 'every u', 'ry and rz', 'bending'])
@pytest.mark.parametrize('order', ['y', 'x'])
def test_single_fixed_dofs(gpulib, kind, masked, order):
    from oracle import oracle
    from pyfe3d_gb300.shellprop import BeamProp, beam_record, isotropic_plate_records
    cdof, x, N, bk = _plate(order, masked)
    E = len(cdof)
    props = isotropic_plate_records(0.004, 70e9, 0.33, rho=2700.)
    if kind.startswith('q4 m'):
        r, c, _ = oracle.q4_m_batch(cdof, 480 * np.arange(E), x, props, mtype=int(kind[-1]))
    elif kind == 'q4 kg':
        r, c, _ = oracle.q4_kg_batch(cdof, 144 * np.arange(E), x, np.ones(N), props)
    else:
        p = BeamProp()
        p.A, p.E, p.G, p.Iyy, p.Izz, p.J, p.intrho = 1e-3, 70e9, 27e9, 1e-8, 2e-8, 3e-8, 2.7
        two, ik, vxy = cdof[:, :2], 144 * np.arange(E), np.array([[0., 0., 1.]])
        if kind == 'beam kc0':
            r, c, _ = oracle.bc_kc0_batch(two, ik, x, np.repeat(vxy, E, 0), beam_record(p))
        else:
            r, c, _ = oracle.bc_m_batch(two, ik, x, vxy, beam_record(p), mtype=int(kind[-1]))
    _check(r, c, N, bk)


@pytest.mark.parametrize('nodes', [1, 4, 60])
@pytest.mark.parametrize('fixed', [(0,), (5,), (0, 1, 5), (2, 3, 4)], ids=str)
def test_free_dofs_alone(gpulib, nodes, fixed):
    """Every pair of free DOFs in row-major order: consecutive columns have consecutive slots throughout a row (300
    of them with 60 nodes and one fixed DOF)."""
    bk = np.zeros((nodes, 6), bool)
    bk[:, fixed] = True
    bk = bk.ravel()
    free = np.flatnonzero(~bk)
    _check(np.repeat(free, free.size), np.tile(free, free.size), 6 * nodes, bk)


@pytest.mark.parametrize('n,density', [(7, 1.), (600, 0.3), (601, 0.9)])
def test_entries_of_a_sparse_matrix(gpulib, n, density):
    """Triplets in the order of scipy's tocoo()."""
    from scipy.sparse import random as sparse_random
    A = sparse_random(n, n, density, random_state=1, format='csr').tocoo()
    _check(A.row.astype(np.int64), A.col.astype(np.int64), n, None)
    bk = np.random.default_rng(2).random(n) < 0.5
    _check(A.row.astype(np.int64), A.col.astype(np.int64), n, bk)


def test_many_slots_per_entry(gpulib):
    """A run of two entries with 2^23 slots each."""
    import torch
    from pyfe3d_gb300.solver import CSRPattern
    n = 1 << 24
    c = torch.arange(n, device='cuda') & 1
    pat = CSRPattern(torch.zeros_like(c), c, 6, None)
    out = torch.full((2,), float('nan'), dtype=torch.float64, device='cuda')
    pat.assemble(torch.ones(n, dtype=torch.float64, device='cuda'), out=out)
    assert out.tolist() == [n / 2, n / 2]

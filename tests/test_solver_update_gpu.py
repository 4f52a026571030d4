"""The row-wise update of launch-per-kernel FP64 solves with 1 to 6 non-zeros in a row of the block inverses, on and off
multiples of a chunk of 32 nodes; the solver's state tells that this is the path that ran."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'pyfe3d_gb300', 'csrc')

SHIM = r'''
#include "fe3d_internal.h"
extern "C" int path(fe3d_solver *s) { return s->team ? -1 : s->sell_on; }
extern "C" int longest(fe3d_solver *s, uint32_t *dinf) {
    return cudaMemcpy(dinf, s->dinf, sizeof(uint32_t) * s->n, cudaMemcpyDeviceToHost) != cudaSuccess;
}
'''


@pytest.fixture(scope='module')
def shim(gpulib, tmp_path_factory):
    from pyfe3d_gb300 import build
    d = tmp_path_factory.mktemp('shim')
    src, lib = d / 'shim.cu', d / 'shim.so'
    src.write_text(SHIM)
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ['-shared', str(src), '-o', str(lib)], check=True)
    h = ctypes.CDLL(str(lib))
    h.path.argtypes, h.longest.argtypes = [ctypes.c_void_p], [ctypes.c_void_p] * 2
    return h


@pytest.mark.parametrize('nodes', [6016, 6017, 9001])
@pytest.mark.parametrize('coupled', ['no node', 'half of the nodes', 'every node'])
@pytest.mark.parametrize('fixed', [0., 0.1])
def test_row_wise_update(gpulib, shim, nodes, coupled, fixed):
    """Nodes in random order (their columns reach over the whole system, too far for resident blocks); off the diagonal
    (0, 1, 5) and (2, 3, 4) do not couple, within the nodes named by coupled all six do."""
    import torch
    from scipy.sparse.linalg import spsolve
    from pyfe3d_gb300.solver import CSRPattern, Solver
    rng = np.random.default_rng(nodes)
    n = 6 * nodes
    g = np.array([0, 0, 1, 1, 1, 0])
    keep = g[:, None] == g[None, :]
    i, j = np.meshgrid(np.arange(6), np.arange(6), indexing='ij')
    r, c, v = [np.arange(n)], [np.arange(n)], [np.full(n, 1.)]
    for d in range(3):
        a = np.arange(nodes - d)
        blk = rng.normal(size=(a.size, 6, 6))
        whole = np.zeros(a.size, bool)
        if d == 0 and coupled != 'no node':
            whole = rng.random(a.size) < (0.5 if coupled == 'half of the nodes' else 2.)
        blk *= keep[None] | whole[:, None, None]
        rr, cc = 6 * a[:, None, None] + i, 6 * (a[:, None, None] + d) + j
        r += [rr.ravel(), cc.ravel()]
        c += [cc.ravel(), rr.ravel()]
        v += [blk.ravel(), blk.ravel()]
    r, c, v = (np.concatenate(t) for t in (r, c, v))
    np.add.at(v, r, np.abs(v))  # diagonally dominant (the first n slots are the diagonal)
    perm = rng.permutation(nodes)
    r, c = 6 * perm[r // 6] + r % 6, 6 * perm[c // 6] + c % 6
    bk = rng.random(n) < fixed
    if fixed:
        bk[600:900] = True  # whole chunks without rows
    pat = CSRPattern(r, c, n, bk)
    vals = pat.assemble(v)
    s = Solver(pat).setup(vals)
    f = rng.normal(size=pat.nrows)
    ref = spsolve(pat.to_scipy(vals).tocsc(), f)
    fd = torch.from_numpy(f).cuda()
    u1, _ = s.solve(fd, tol=1e-300, maxiter=4, check_every=2)
    assert shim.path(s._h) == 1
    dinf = np.zeros(pat.nrows, np.uint32)
    assert shim.longest(s._h, dinf.ctypes.data) == 0
    assert (dinf & 7).max() == (3 if coupled == 'no node' else 6)
    for u0 in (None, u1):
        u, st = s.solve(fd, u0=u0, tol=1e-13)
        assert st['status'] == 'converged'
        assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)  # condition number below 100

"""Solves whose resident launch cannot be used: refused by the runtime (more shared memory than a block may have, asked
for by raising the limit that the host keeps) or given up because a poll ran out (its limit set to zero).  They end as
the launch-per-kernel and the lockstep iterations do."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'pyfe3d_gb300', 'csrc')

SHIM = r'''
#include "fe3d_internal.h"
static int disturb(fe3d_team *t, int how) {
    if (!t) return 0;
    if (how == 0) t->smem_max = (size_t)1 << 20;
    else t->poll = t->poll_first = 0;
    return 1;
}
extern "C" int disturb_solver(fe3d_solver *s, int how) { return disturb(s->team, how); }
extern "C" int disturb_batch(fe3d_bsolver *b, int how) { return disturb(b->team, how); }
'''


@pytest.fixture(scope='module')
def shim(gpulib, tmp_path_factory):
    from pyfe3d_gb300 import build
    d = tmp_path_factory.mktemp('shim')
    src, lib = d / 'shim.cu', d / 'shim.so'
    src.write_text(SHIM)
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ['-shared', str(src), '-o', str(lib)], check=True)
    h = ctypes.CDLL(str(lib))
    for f in (h.disturb_solver, h.disturb_batch):
        f.argtypes = [ctypes.c_void_p, ctypes.c_int]
    return h


def _system(nodes):
    """Diagonally dominant banded system of coupled nodes: its blocks' rows take more than 227 KB on 152 blocks."""
    import torch
    rng = np.random.default_rng(nodes)
    n = 6 * nodes
    i, j = np.meshgrid(np.arange(6), np.arange(6), indexing='ij')
    r, c, v = [np.arange(n)], [np.arange(n)], [np.full(n, 1.)]
    for d in range(3):
        a = np.arange(nodes - d)
        blk = rng.normal(size=(a.size, 6, 6))
        rr, cc = 6 * a[:, None, None] + i, 6 * (a[:, None, None] + d) + j
        r += [rr.ravel(), cc.ravel()]
        c += [cc.ravel(), rr.ravel()]
        v += [blk.ravel(), blk.ravel()]
    r, c, v = (np.concatenate(t) for t in (r, c, v))
    np.add.at(v, r, np.abs(v))
    return r, c, v, torch.from_numpy(rng.normal(size=n)).cuda()


@pytest.mark.parametrize('how', ['refused', 'given up'])
def test_solver(gpulib, shim, how):
    from pyfe3d_gb300.solver import CSRPattern, Solver
    r, c, v, f = _system(20000)
    pat = CSRPattern(r, c, f.numel(), None)
    vals = pat.assemble(v)
    s = Solver(pat).setup(vals)
    u, _ = s.solve(f, tol=1e-300, maxiter=4, check_every=2)
    assert shim.disturb_solver(s._h, ['refused', 'given up'].index(how)) == 1
    for u0 in (None, u):
        w, st = s.solve(f, u0=u0, tol=1e-12)
        assert st['status'] == 'converged'
        assert ((f - pat.spmv(vals, w)).norm() <= 1e-11 * f.norm()).item()
    assert shim.disturb_solver(s._h, 0) == 0  # later solves do not try again


@pytest.mark.parametrize('how', ['refused', 'given up'])
def test_batch(gpulib, shim, how):
    from pyfe3d_gb300.solver import BatchSolver, CSRPattern
    r, c, v, f = _system(20000)
    n = f.numel()
    pat = CSRPattern(np.concatenate([r, r + n]), np.concatenate([c, c + n]), 2 * n, None)
    vals = pat.assemble(np.concatenate([v, 2. * v]))
    f = f.repeat(2)
    b = BatchSolver(pat, np.repeat([0, 1], n), 2).setup(vals)
    u, _ = b.solve(f, tol=1e-300, maxiter=4, check_every=2)
    assert shim.disturb_batch(b._h, ['refused', 'given up'].index(how)) == 1
    for u0 in (None, u):
        w, st = b.solve(f, u0=u0, tol=1e-12)
        assert (st['inst_status'] == 0).all() and (st['inst_relres'] <= 1e-12).all()
        assert ((f - pat.spmv(vals, w)).norm() <= 1e-11 * f.norm()).item()
    assert shim.disturb_batch(b._h, 0) == 0

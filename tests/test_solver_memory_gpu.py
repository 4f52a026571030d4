"""Solves under an allocator that fails: each cudaMalloc of a solve in turn is refused by a fake, and the solve ends as it
does with all of them."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# cudaMalloc as libfe3d_gb300.so calls it: the call number fail_at (from 0) since arm() returns cudaErrorMemoryAllocation
FAKE = r'''
#define _GNU_SOURCE
#include <dlfcn.h>
#include <string.h>
static int calls, fail_at = -1;
void arm(int k) { calls = 0; fail_at = k; }
int disarm(void) { fail_at = -1; return calls; }
int cudaMalloc(void **p, size_t n) {
    static int (*real)(void **, size_t);
    Dl_info who;
    if (!real) real = (int (*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
    if (dladdr(__builtin_return_address(0), &who) && who.dli_fname && strstr(who.dli_fname, "libfe3d_gb300"))
        if (calls++ == fail_at) {
            *p = 0;
            return 2;
        }
    return real(p, n);
}
'''

PROGRAM = r'''
import ctypes, sys
import numpy as np, torch
from pyfe3d_gb300.solver import BatchSolver, CSRPattern, Solver
fake = ctypes.CDLL(sys.argv[1])
nodes, order, flexible, ninst = int(sys.argv[2]), sys.argv[3], sys.argv[4] == 'True', int(sys.argv[5])
# diagonally dominant, (0, 1, 5) and (2, 3, 4) uncoupled: half of the stored entries are zeros
rng = np.random.default_rng(nodes)
n = 6 * nodes
g = np.array([0, 0, 1, 1, 1, 0])
keep = g[:, None] == g[None, :]
r, c, v = [np.arange(n)], [np.arange(n)], [np.full(n, 1.)]
i, j = np.meshgrid(np.arange(6), np.arange(6), indexing='ij')
for d in range(3):
    a = np.arange(nodes - d)
    blk = rng.normal(size=(a.size, 6, 6)) * keep
    rr, cc = 6 * a[:, None, None] + i, 6 * (a[:, None, None] + d) + j
    r += [rr.ravel(), cc.ravel()]
    c += [cc.ravel(), rr.ravel()]
    v += [blk.ravel(), blk.ravel()]
r, c, v = (np.concatenate(t) for t in (r, c, v))
np.add.at(v, r, np.abs(v))
if order == 'shuffled':
    perm = rng.permutation(nodes)
    r, c = 6 * perm[r // 6] + r % 6, 6 * perm[c // 6] + c % 6
if ninst:
    r, c, v = (np.concatenate([x + (n * k if x is not v else 0) for k in range(ninst)]) for x in (r, c, v))
    inst = np.repeat(np.arange(ninst), n)
pat = CSRPattern(r, c, n * max(ninst, 1), None)
vals = pat.assemble(v)
f = torch.from_numpy(rng.normal(size=pat.nrows)).cuda()
k, total = -1, 0
while k < total:
    s = (BatchSolver(pat, inst, ninst) if ninst else Solver(pat)).setup(vals)
    for again in range(2):  # the second solve has memory again
        fake.arm(k if again == 0 else -1)
        u, st = s.solve(f, tol=1e-12) if ninst else s.solve(f, tol=1e-12, flexible=flexible)
        calls = fake.disarm()
        if k < 0 and again == 0:
            total = calls
        assert (st['inst_status'] == 0).all() if ninst else st['status'] == 'converged', (k, again)
        assert ((f - pat.spmv(vals, u)).norm() <= 1e-11 * f.norm()).item(), (k, again)
    k += 1
print('allocations', total)
'''


@pytest.mark.parametrize('nodes,order,flexible,ninst', [(171, 'banded', False, 0), (5000, 'shuffled', False, 0),
                                                        (3001, 'banded', True, 0), (60, 'banded', False, 5)],
                         ids=['resident', 'slices', 'flexible', 'batch'])
def test_every_allocation_refused(gpulib, tmp_path, nodes, order, flexible, ninst):
    cc = shutil.which('gcc')
    if cc is None:
        pytest.skip('no gcc')
    src, lib = tmp_path / 'fake.c', tmp_path / 'fake.so'
    src.write_text(FAKE)
    subprocess.run([cc, '-shared', '-fPIC', str(src), '-o', str(lib), '-ldl'], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, '-c', PROGRAM, str(lib), str(nodes), order, str(flexible), str(ninst)],
                       env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert int(p.stdout.split()[-1]) > 0  # the fake was in place

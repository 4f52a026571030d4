"""The lists of rows and nodes that the lockstep iterations of a batch walk: nodes without free DOFs (clamped edges)
belong to no instance and are in no list."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'pyfe3d_gb300', 'csrc')

SHIM = r'''
#include "fe3d_internal.h"
extern "C" int lists(fe3d_bsolver *b, int *count, int32_t *rows, int32_t *nodes) {
    if (cudaMemcpy(count, b->lcount, 2 * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    if (cudaMemcpy(rows, b->rowlist, sizeof(int32_t) * count[0], cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    return cudaMemcpy(nodes, b->nodelist, sizeof(int32_t) * count[1], cudaMemcpyDeviceToHost) != cudaSuccess ? 3 : 0;
}
'''


@pytest.mark.parametrize('P,lo,hi', [(1, 2, 2), (37, 2, 6), (1000, 2, 5), (9728, 4, 7)])
def test_nodes_without_free_dofs(gpulib, tmp_path, P, lo, hi):
    from pyfe3d_gb300 import batch, build
    from pyfe3d_gb300.meshes import BatchedPlates
    from pyfe3d_gb300.solver import BatchSolver, ElementPattern, FusedMap
    src, lib = tmp_path / 'shim.cu', tmp_path / 'shim.so'
    src.write_text(SHIM)
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ['-shared', str(src), '-o', str(lib)], check=True)
    lists = ctypes.CDLL(str(lib)).lists
    lists.argtypes = [ctypes.c_void_p] * 4
    bp = BatchedPlates(P, lo, hi, 4)
    pat = ElementPattern([bp.cdof], bp.N, bp.bk)
    fmap = FusedMap(pat, [bp.cdof])
    vals = batch.quad4_update_KC0_csr(fmap.new_values(), fmap, bp.x, bp.props, pid=bp.pid)
    b = BatchSolver(pat, bp.inst_of_dof, bp.P).setup(vals)  # leaves the lists of all instances
    count, rows, nodes = np.zeros(2, np.int32), np.full(pat.nrows, -1, np.int32), np.full(bp.nnodes, -1, np.int32)
    assert lists(b._h, count.ctypes.data, rows.ctypes.data, nodes.ctypes.data) == 0
    free = np.flatnonzero((~bp.bk).reshape(-1, 6).any(1))
    assert count.tolist() == [pat.nrows, free.size]
    assert np.array_equal(rows, np.arange(pat.nrows)) and np.array_equal(nodes[:free.size], free)

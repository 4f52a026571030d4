"""The quotients of the resident solver (csrc/quotient.cuh) against exact ones."""
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'pyfe3d_gb300', 'csrc')

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "quotient.cuh"
__global__ void quotients(int n, const double *a, const double *b, double *c, double *d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    c[i] = fe3d::quotient(a[i], b[i]);
    d[i] = fe3d::quotient_range(b[i]) ? fe3d::quotient_by(a[i], b[i], 1. / b[i]) : fe3d::plain_quotient(a[i], b[i]);
}
int main(int, char **argv) {  // n, then n doubles a and n doubles b on stdin; both quotients to stdout
    const int n = atoi(argv[1]);
    const size_t bytes = sizeof(double) * n;
    double *h = (double *)malloc(2 * bytes), *p;
    if (fread(h, bytes, 2, stdin) != 2 || cudaMalloc((void **)&p, 4 * bytes) != cudaSuccess) return 1;
    if (cudaMemcpy(p, h, 2 * bytes, cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    quotients<<<(n + 255) / 256, 256>>>(n, p, p + n, p + 2 * n, p + 3 * n);
    if (cudaMemcpy(h, p + 2 * n, 2 * bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    return fwrite(h, bytes, 2, stdout) == 2 ? 0 : 4;
}
"""


@pytest.fixture(scope='module')
def quotients(gpulib, tmp_path_factory):
    from pyfe3d_gb300 import build
    d = tmp_path_factory.mktemp('quotient')
    src, exe = d / 'quotient.cu', d / 'quotient'
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + [str(src), '-o', str(exe)], check=True)

    def call(a, b):
        a, b = np.broadcast_arrays(np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64))
        out = subprocess.run([str(exe), str(a.size)], input=a.tobytes() + b.tobytes(), capture_output=True, check=True)
        return np.frombuffer(out.stdout).reshape(2, -1)
    return call


def test_rounding(quotients):
    """Mantissas at random and next to powers of two, exponents of b over its whole range, quotients and residuals
    normal: within 1/2 + 2^-18 units in the last place of the exact quotient."""
    rng = np.random.default_rng(0)
    n = 200000
    m = rng.uniform(1., 2., (2, n))
    edge = rng.random((2, n)) < 0.2
    m[edge] = np.where(rng.random(edge.sum()) < 0.5, 1. + rng.integers(0, 9, edge.sum()) * 2. ** -52,
                       2. - rng.integers(1, 9, edge.sum()) * 2. ** -52)
    eb = rng.integers(65 - 1023, 1984 - 1023, n)
    eq = rng.integers(-900, 900, n)
    ea = np.clip(eb + eq, -900, 1000)
    keep = (ea - eb > -960) & (ea - eb < 1000)
    sign = rng.choice([-1., 1.], (2, n))
    a, b = (np.ldexp(sign[0] * m[0], ea)[keep], np.ldexp(sign[1] * m[1], eb)[keep])
    exact = a / b  # rounded to nearest
    for c in quotients(a, b):
        off = np.flatnonzero(c != exact)
        assert (np.abs(c[off] - exact[off]) <= np.spacing(np.abs(exact[off]))).all()
        assert off.size <= 2e-4 * a.size  # 2^-18 of the quotients lie that close to a tie, on average
        for i in off[:200]:
            q = Fraction(a[i]) / Fraction(b[i])
            assert abs(Fraction(c[i]) - q) <= (Fraction(1, 2) + Fraction(1, 2 ** 18)) * Fraction(math.ulp(c[i]))


def test_ends_of_the_range(quotients):
    """Divisors on both sides of the limits of the fast path, zeros, infinities, NaN and overflowing quotients."""
    e = np.array([-1074, -1023, -1022, -960, -959, -958, -957, 0, 959, 960, 961, 962, 1023])
    b = np.concatenate([np.ldexp(1.5, e), -np.ldexp(1.25, e), [0., -0., np.inf, -np.inf, np.nan]])
    a = np.array([0., -0., 1., -3., 1e-300, 1e300, 1.7e308, np.inf, np.nan])
    a, b = (v.ravel() for v in np.meshgrid(a, b))
    with np.errstate(all='ignore'):
        exact = np.where(b == 0., 0., a / b)
    for c in quotients(a, b):
        assert (np.isnan(c) == np.isnan(exact)).all() and (np.isinf(c) == np.isinf(exact)).all()
        ok = np.isfinite(exact)
        # (denormal quotients: rounded twice)
        assert (np.abs(c[ok] - exact[ok]) <= np.spacing(np.abs(exact[ok]))).all()

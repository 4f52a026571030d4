"""The fixed-point sums of the resident solver (csrc/fixed_sum.h, compiled for the host) against exact sums."""
import ctypes
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'pyfe3d_gb300', 'csrc')

SHIM = r'''
#include "fixed_sum.h"
#include <string.h>
extern "C" int fixed_sum(const int64_t *b, int n, int64_t *out) {
    int emax = 0;
    for (int i = 0; i < n; i++) {
        const int e = (int)(b[i] >> 52) & 0x7ff;
        if (e > emax) emax = e;
    }
    fe3d::FixedLimbs f{0u, 0u, 0};
    for (int i = 0; i < n; i++) fe3d::fixed_add(f, b[i], emax);
    *out = fe3d::fixed_round(f, emax);
    return fe3d::FS_TERMS;
}
extern "C" int fixed_range(int emax) { return fe3d::fixed_range(emax); }
'''


@pytest.fixture(scope='module')
def fixed_sum(tmp_path_factory):
    cxx = shutil.which('g++')
    if cxx is None:
        pytest.skip('no g++')
    d = tmp_path_factory.mktemp('fixed_sum')
    src, lib = d / 'shim.cpp', d / 'shim.so'
    src.write_text(SHIM)
    subprocess.run([cxx, '-O1', '-std=c++17', '-shared', '-fPIC', '-I' + CSRC, str(src), '-o', str(lib)], check=True)
    h = ctypes.CDLL(str(lib))
    f = h.fixed_sum

    def call(v):
        v = np.ascontiguousarray(v, dtype=np.float64)
        out = np.zeros(1)
        assert v.size <= f(v.ctypes.data_as(ctypes.c_void_p), v.size, out.ctypes.data_as(ctypes.c_void_p))
        return out[0]
    call.range = h.fixed_range
    return call


def _check(fixed_sum, v):
    v = np.asarray(v, dtype=np.float64)
    exact = sum((Fraction(x) for x in v.tolist()), Fraction(0))
    top = Fraction(2) ** (math.frexp(np.abs(v).max())[1] - 1) if np.any(v) else Fraction(0)
    got = fixed_sum(v)
    # half a unit in the last place of the exact sum's neighbourhood, and 2^-62 of the largest term per term that
    # has bits below that
    cut = sum(1 for x in v.tolist() if x and Fraction(x) % (top / 2 ** 62))
    err, bound = abs(Fraction(got) - exact), Fraction(math.ulp(got)) / 2 + cut * top / 2 ** 62
    assert err <= bound, (v, got, float(exact), float(err / bound))


def test_single_terms_and_cancellation(fixed_sum):
    one = 1. + 2. ** -52
    for v in ([one] + 31 * [0.], [one, -1.], [-one, 1.], [one, one], [1., 2. ** -53], [1., 2. ** -53, 2. ** -62],
              [1., -2. ** -54], [-1., 2. ** -62], [1.9999999999999998, 2. ** -52], 256 * [one], 160 * [-one],
              [2. ** 1000, -2. ** 950], [1.] + 31 * [0.], [1., -0., 5e-324], [1., -1.]):
        _check(fixed_sum, v)
    assert fixed_sum([one] + 31 * [0.]) == one


@pytest.mark.parametrize('n', [1, 2, 3, 5, 17, 32, 160, 256])
@pytest.mark.parametrize('decades', [0, 1, 6, 20, 40])
@pytest.mark.parametrize('signs', ['plus', 'minus', 'mixed', 'cancel'])
def test_against_exact_sums(fixed_sum, n, decades, signs):
    rng = np.random.default_rng(1000 * n + decades)
    for scale in (0, -750, 900):
        for _ in range(4):
            v = rng.uniform(1., 2., n) * 10. ** rng.uniform(-decades / 2, decades / 2, n) * 2. ** scale
            if signs == 'minus':
                v = -v
            elif signs == 'mixed':
                v *= rng.choice([-1., 1.], n)
            elif signs == 'cancel':
                v[n // 2:] = -v[:n - n // 2] * (1. + 2. ** -40)
            _check(fixed_sum, v)


def test_ends_of_the_range(fixed_sum):
    """Where the fixed-point sum is taken it neither overflows (256 terms of the largest size) nor ends below the
    normal numbers (all but the last bit cancelled); infinities, NaN and the rest are left to plain additions."""
    big = 2. - 2. ** -52
    for e in range(2048):
        if not fixed_sum.range(e):
            continue
        for v in (256 * [math.ldexp(big, e - 1023)], 256 * [math.ldexp(-big, e - 1023)],
                  [math.ldexp(big, e - 1023), math.ldexp(-(2. - 2. ** -51), e - 1023)]):
            got = fixed_sum(v)
            assert math.isfinite(got) and got == math.fsum(v) and abs(got) >= 2. ** -1022
    assert fixed_sum.range(1023 - 800) and fixed_sum.range(1023) and fixed_sum.range(1023 + 1000)
    assert not any(fixed_sum.range(e) for e in (0, 1, 2040, 2046, 2047))

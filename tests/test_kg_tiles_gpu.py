"""Quad4 KG at the edges of its tiles: part-filled and several tiles, flat elements next to others in one warp, the
sections that its phases tell apart, cleared and filled values, odd offsets, against the oracle."""
import numpy as np
import pytest

from conftest import REL_TOL, blockwise_rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('E', [1, 7, 31, 32, 33, 200])
@pytest.mark.parametrize('section', ['iso', 'a16', 'b'])
@pytest.mark.parametrize('shape', ['flat', 'mixed'])
@pytest.mark.parametrize('shift', [0, 1])
def test_kg_tiles_match_oracle(gpulib, oracle, E, section, shape, shift):
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.shellprop import isotropic_plate_records
    rng = np.random.default_rng(E)
    i, j = np.meshgrid(np.arange(E + 1), np.arange(2), indexing='ij')
    x = np.stack([i + rng.uniform(-.2, .2, i.shape), j + rng.uniform(-.2, .2, i.shape), 0. * i], -1)
    if shape == 'mixed':
        x[::3, 0, 2] += rng.uniform(0.1, 0.3, x[::3, 0, 2].shape)  # two elements of three are not flat
    x = x.reshape(-1)
    a = 2 * np.arange(E)
    cdof = 6 * np.stack([a, a + 2, a + 3, a + 1], 1).astype(np.int64)
    props = isotropic_plate_records(rng.uniform(0.002, 0.02, E), 70e9, 0.3, rho=2700.)
    if section == 'a16':
        props[::2, 2] = 1e6  # A16 of every other element
    if section == 'b':
        props[::2, 6:12] = rng.normal(size=props[::2, 6:12].shape) * 1e3
    u = rng.normal(size=12 * (E + 1)) * 1e-3
    init_k = shift + 144 * np.arange(E, dtype=np.int64)
    r0, c0, v0 = oracle.q4_kg_batch(cdof, init_k - shift, x, u, props)
    for fill in (0., 1.):
        n = 144 * E + shift
        r = np.zeros(n, np.int64); c = np.zeros(n, np.int64)
        start = fill * rng.normal(size=n)
        v = start.copy()
        batch.quad4_update_KG(r, c, v, x, u, cdof, init_k, props)
        assert (r[shift:] == r0).all() and (c[shift:] == c0).all()
        assert (v[:shift] == start[:shift]).all()
        assert blockwise_rel_err(v[shift:], start[shift:] + v0, 144) < REL_TOL

"""Quad4 KC0 at the edges of its tiles (4 elements a CTA, 14 and 28 a tile, one full wave of tiles) over every kind of
element and section at once, onto cleared, partly cleared and arbitrary values, against the oracle."""
import numpy as np
import pytest

from conftest import REL_TOL, blockwise_rel_err

pytestmark = pytest.mark.gpu


def _elements(E, seed):
    """Separate quads: flat with either normal, warped about a diagonal, tilted; and a section record each."""
    from pyfe3d_gb300.shellprop import shell_record
    from pyfe3d_gb300.shellprop_utils import isotropic_plate, laminated_plate
    rng = np.random.default_rng(seed)
    lam = (142.5e9, 8.7e9, 0.28, 5.1e9, 5.1e9, 5.1e9)
    recs = np.stack([shell_record(p) for p in (
        isotropic_plate(0.004, 70e9, 0.33), isotropic_plate(1.7, 70e9, 0.3),
        laminated_plate([0, 45, -45, 90, 90, -45, 45, 0], 0.000125, lam),
        laminated_plate([0, 30, 60], 0.0002, lam, offset=0.003))])
    base = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float)
    xy = base + rng.uniform(-0.2, 0.2, (E, 4, 2))
    x = np.concatenate([xy, np.zeros((E, 4, 1))], 2)
    kind = rng.integers(0, 4, E)
    flip = kind == 1
    x[flip] = x[flip][:, ::-1]
    x[kind == 2, 1::2, 2] = 0.1  # both diagonals level: flat by the element's frame
    for e in np.where(kind == 3)[0]:
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        x[e] = x[e] @ q + rng.normal(size=3)
    cdof = 6 * np.arange(4 * E, dtype=np.int64).reshape(E, 4)
    return x.ravel(), cdof, recs, rng.integers(0, 4, E).astype(np.int32), rng


@pytest.mark.parametrize('E', [1, 2, 3, 5, 13, 29, 607, 1215, 1217, 4257, 8513])
@pytest.mark.parametrize('start', ['clear', 'mixed', 'random'])
def test_tiles_sections_and_current_values(gpulib, oracle, E, start):
    import torch
    from pyfe3d_gb300 import batch
    x, cdof, recs, pid, rng = _elements(E, E)
    ik = 576 * np.arange(E, dtype=np.int64) + (1 if E % 2 else 0)  # odd: the 8-byte path
    n = 576 * E + 2
    v0 = np.zeros(n)
    if start != 'clear':
        v0[:] = rng.normal(size=n)
    if start == 'mixed':
        v0.reshape(-1)[:576 * (E // 2)] = 0.
        v0[rng.random(n) < 0.5] = 0.
    r = torch.zeros(n, dtype=torch.int64, device='cuda')
    c, v = torch.zeros_like(r), torch.from_numpy(v0).cuda()
    batch.quad4_update_KC0(r, c, v, x, cdof, ik, recs, pid=pid)
    r0, c0, k0 = oracle.q4_kc0_batch(cdof, 576 * np.arange(E, dtype=np.int64), x, recs, pid=pid)
    s = int(ik[0])
    assert (r.cpu().numpy()[s:s + 576 * E] == r0).all() and (c.cpu().numpy()[s:s + 576 * E] == c0).all()
    got = v.cpu().numpy()
    assert blockwise_rel_err(got[s:s + 576 * E] - v0[s:s + 576 * E], k0, 576) < REL_TOL
    out = np.concatenate([got[:s], got[s + 576 * E:]])
    assert (out == np.concatenate([v0[:s], v0[s + 576 * E:]])).all()


@pytest.mark.parametrize('nx,ny', [(2, 2), (2, 9), (6, 7), (30, 41), (71, 70)])
@pytest.mark.parametrize('section', [0, 2, 3])
def test_csr_matches_triplets(gpulib, nx, ny, section):
    """Assigned, added and atomic blocks of plates with perturbed nodes and mixed fixed DOFs."""
    import torch
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.meshes import PlateMesh
    from pyfe3d_gb300.solver import CSRPattern, ElementPattern, FusedMap
    recs = _elements(1, 0)[2]
    m = PlateMesh(nx, ny, 1.0, 0.8, perturb=0.1, seed=nx)
    bk = np.random.default_rng(ny).random(m.N) < 0.2
    n = 576 * m.E
    r = torch.zeros(n, dtype=torch.int64, device='cuda')
    c, v = torch.zeros_like(r), torch.zeros(n, dtype=torch.float64, device='cuda')
    rec = recs[section:section + 1]
    batch.quad4_update_KC0(r, c, v, m.x, m.cdof, m.init_k(576), rec)
    want = CSRPattern(r, c, m.N, bk).assemble(v)
    pat = ElementPattern([m.cdof], m.N, bk)
    fmap = FusedMap(pat, [m.cdof])
    scale = float(want.abs().max())
    for mode, start in (('assign', float('nan')), ('add', 0.), ('add', 3.), ('atomic', 0.)):
        vals = torch.full_like(want, start)
        batch.quad4_update_KC0_csr(vals, fmap, m.x, rec, mode=mode)
        got = vals - start if mode == 'add' else vals
        assert float((got - want).abs().max()) <= 1e-14 * scale, (mode, start)


@pytest.mark.parametrize('E', [1, 5, 7, 29, 31, 1823, 1825, 9121])
@pytest.mark.parametrize('start', ['clear', 'mixed', 'random'])
def test_tria_tiles_sections_and_current_values(gpulib, oracle, E, start):
    """Tria3R at the edges of its tiles (6 elements a CTA, 5 a warp, 30 a tile, one full wave)."""
    import torch
    from pyfe3d_gb300 import batch
    x4, _, recs, pid, rng = _elements(E, 3 * E)
    x = x4.reshape(E, 4, 3)[:, :3].copy()
    x[rng.random(E) < 0.6, :, 2] = 0.
    x = x.ravel()
    cdof = 6 * np.arange(3 * E, dtype=np.int64).reshape(E, 3)
    k6, alpha = rng.uniform(10., 200., E), rng.uniform(0.2, 1., E)
    off = 1 if E % 2 else 0  # odd: the 8-byte path
    n = 324 * E + 2
    v0 = np.zeros(n)
    if start != 'clear':
        v0[:] = rng.normal(size=n)
    if start == 'mixed':
        v0[:324 * (E // 2)] = 0.
        v0[rng.random(n) < 0.5] = 0.
    r = torch.zeros(n, dtype=torch.int64, device='cuda')
    c, v = torch.zeros_like(r), torch.from_numpy(v0).cuda()
    ik = 324 * np.arange(E, dtype=np.int64)
    batch.tria3r_update_KC0(r, c, v, x, cdof, ik + off, recs, pid=pid, k6rot=k6, alpha=alpha)
    r0, c0, k0 = oracle.t3_kc0_batch(cdof, ik, x, recs, pid=pid, k6rot=k6, alpha=alpha)
    s = slice(off, off + 324 * E)
    assert (r.cpu().numpy()[s] == r0).all() and (c.cpu().numpy()[s] == c0).all()
    got = v.cpu().numpy()
    assert blockwise_rel_err(got[s] - v0[s], k0, 324) < REL_TOL
    out = np.ones(n, bool)
    out[s] = False
    assert (got[out] == v0[out]).all()

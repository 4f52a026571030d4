"""The work that programs built on pyfe3d_gb300 spend their time in, as cases that can be timed and checked.

Every case is one pass through the public entry points with everything on the GPU that a user keeps
there (mesh, property records, pattern, solver).  Families (the ``kind`` of a case):

  triplets   Quad4 update_KC0 of a flat plate into the caller's row, column and value arrays
  shell      the same on a laminated cylinder with a material direction, values only
  csr        update_KC0 straight into the reduced CSR matrix
  panel      the stiffened panel: laminated skin and BeamC stringers into one reduced CSR matrix
  tria       Tria3R update_KC0
  kgm        geometric stiffness of a displacement field and the mass matrix (prestressed vibration, buckling)
  assemble   triplet values to the reduced CSR values through a pattern built once
  steps      a fixed number of block-Jacobi PCG iterations (the eigensolver's inner preconditioner)
  solve      a static analysis step: update_KC0 into the CSR matrix, preconditioner set-up, solve
  batch      the same for many uneven plates at once

``exact`` restates the element matrices and the solves with plain torch operations in 64 bits.
"""
import math

import numpy as np
import torch

from pyfe3d_gb300 import batch
from pyfe3d_gb300.shellprop import BeamProp, beam_record, isotropic_plate_records_device, shell_record
from pyfe3d_gb300.shellprop_utils import laminated_plate
from pyfe3d_gb300.solver import BatchSolver, CSRPattern, ElementPattern, FusedMap, Solver

DEV = 'cuda'
F64 = torch.float64
I64 = torch.int64
E_MOD, NU, RHO = 70e9, 0.33, 2700.
PLIES = (0, 45, -45, 90, 90, -45, 45, 0)
PLY_T = 0.000125
LAMINA = (142.5e9, 8.7e9, 0.28, 5.1e9, 5.1e9, 5.1e9)
TOL = 1e-10


def listed():
    return [
        # the first plate of the reference's tutorial: every launch and check counts
        {'name': 'kc0_first_plate', 'kind': 'triplets', 'nx': 21, 'ny': 21, 'uniform': True},
        # the benchmark plate: a million elements with a thickness each
        {'name': 'kc0_scale_plate', 'kind': 'triplets', 'nx': 1001, 'ny': 1001, 'uniform': False},
        # a composite shell whose values are updated in an optimisation loop (no flat elements, B^T ABD B in full)
        {'name': 'kc0_cylinder', 'kind': 'shell', 'nx': 121, 'ny': 241, 'direction': True},
        # matrix update of a plate model without triplets
        {'name': 'kc0_csr_plate', 'kind': 'csr', 'nx': 301, 'ny': 301},
        # matrix update of a stiffened composite panel: two element types in one matrix
        {'name': 'kc0_csr_panel', 'kind': 'panel', 'nel': 200},
        # unstructured-style triangles of uneven shape
        {'name': 'tria_plate', 'kind': 'tria', 'nx': 201, 'ny': 301},
        # what buckling and prestressed vibration add to a static step
        {'name': 'kg_mass_plate', 'kind': 'kgm', 'nx': 301, 'ny': 301, 'mtype': 0},
        # the reference's coo -> csc -> K[bu][:, bu] with the pattern kept
        {'name': 'assemble_plate', 'kind': 'assemble', 'nx': 301, 'ny': 301},
        # large system, matrix far above the L2 cache
        {'name': 'pcg_steps_large', 'kind': 'steps', 'nx': 501, 'ny': 501, 'iters': 50},
        # static step of the tutorial plate
        {'name': 'solve_first_plate', 'kind': 'solve', 'nx': 21, 'ny': 21, 'clamped': False},
        # static step of an ordinary model
        {'name': 'solve_plate', 'kind': 'solve', 'nx': 101, 'ny': 101, 'clamped': True},
        # a design study: many small uneven plates
        {'name': 'solve_batch', 'kind': 'batch', 'plates': 48, 'nmin': 8, 'nmax': 40},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['triplets', 'triplets', 'shell', 'csr', 'panel', 'tria', 'kgm', 'assemble', 'steps', 'solve',
                       'solve', 'batch'])
    if kind == 'triplets':
        return {'kind': kind, 'nx': _log(rng, 6, 1001), 'ny': _log(rng, 6, 1001), 'uniform': rng.random() < 0.4}
    if kind == 'shell':
        return {'kind': kind, 'nx': _log(rng, 6, 121), 'ny': _log(rng, 12, 241), 'direction': rng.random() < 0.6}
    if kind == 'panel':
        return {'kind': kind, 'nel': 10 * rng.randint(2, 20)}
    if kind == 'kgm':
        return {'kind': kind, 'nx': _log(rng, 8, 301), 'ny': _log(rng, 8, 301), 'mtype': rng.randint(0, 2)}
    if kind == 'steps':
        return {'kind': kind, 'nx': _log(rng, 60, 501), 'ny': _log(rng, 60, 501), 'iters': rng.randint(20, 50)}
    if kind == 'solve':
        return {'kind': kind, 'nx': _log(rng, 9, 101), 'ny': _log(rng, 9, 101), 'clamped': rng.random() < 0.5}
    if kind == 'batch':
        lo = rng.randint(4, 12)
        return {'kind': kind, 'plates': _log(rng, 6, 48), 'nmin': lo, 'nmax': lo + rng.randint(4, 28)}
    return {'kind': kind, 'nx': _log(rng, 8, 301), 'ny': _log(rng, 8, 301)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=F64)


def _randn(g, n):
    return torch.randn(n, generator=g, device=DEV, dtype=F64)


def _quads(nx, ny, wrap=False):
    """Node ids (E, 4) of a structured nx x ny node grid, x slow; wrap closes the ny direction."""
    ids = torch.arange(nx * ny, device=DEV, dtype=I64).reshape(nx, ny)
    up = torch.roll(ids, -1, 1) if wrap else ids[:, 1:]
    lo = ids if wrap else ids[:, :-1]
    return torch.stack([lo[:-1].reshape(-1), lo[1:].reshape(-1), up[1:].reshape(-1), up[:-1].reshape(-1)], 1)


def _plate(case, g, a=2.0, b=2.0, perturb=0.1):
    """Coordinates (nodes, 3), quads (E, 4) and edge mask of a flat plate with moved interior nodes."""
    nx, ny = case['nx'], case['ny']
    X = torch.linspace(0, a, nx, device=DEV, dtype=F64)[:, None].expand(nx, ny).clone()
    Y = torch.linspace(0, b, ny, device=DEV, dtype=F64)[None, :].expand(nx, ny).clone()
    edge = torch.ones(nx, ny, dtype=torch.bool, device=DEV)
    edge[1:-1, 1:-1] = False
    dx, dy = perturb * a / (nx - 1), perturb * b / (ny - 1)
    X += torch.where(edge, 0., 1.) * _rand(g, (nx, ny), -dx, dx)
    Y += torch.where(edge, 0., 1.) * _rand(g, (nx, ny), -dy, dy)
    x = torch.stack([X, Y, torch.zeros_like(X)], 2).reshape(-1, 3).contiguous()
    return x, _quads(nx, ny), edge.reshape(-1)


def _thickness(g, n):
    return 0.005 * torch.exp(0.3 * _randn(g, n))


def _pid(n):
    return torch.arange(n, device=DEV, dtype=torch.int32)


def _offsets(n, size):
    return size * torch.arange(n, device=DEV, dtype=I64)


def _mask(edge, dofs, nodes):
    bk = torch.zeros(nodes, 6, dtype=torch.bool, device=DEV)
    for d in dofs:
        bk[:, d] = edge
    return bk.reshape(-1)


def _coo(n):
    return (torch.zeros(n, dtype=I64, device=DEV), torch.zeros(n, dtype=I64, device=DEV),
            torch.zeros(n, dtype=F64, device=DEV))


def _laminate():
    return laminated_plate(list(PLIES), plyt=PLY_T, laminaprop=LAMINA, calc_scf=False)


def _stringer():
    p = BeamProp()
    p.A, p.E, p.G = 0.02 * 0.004, E_MOD, E_MOD / (2 * (1 + NU))
    p.Iyy, p.Izz = 0.004 * 0.02 ** 3 / 12, 0.02 * 0.004 ** 3 / 12
    p.J = p.Iyy + p.Izz
    return p


def _inputs(case, seed):
    """Mesh, thickness and loads of a case: plain tensors, the same for prepare and exact."""
    g, k = _gen(seed), case['kind']
    m = {}
    if k == 'shell':
        nx, ny = case['nx'], case['ny']
        r, length = 0.4, 1.2
        ax = torch.linspace(0, length, nx, device=DEV, dtype=F64)[:, None].expand(nx, ny)
        th = (2 * math.pi / ny) * torch.arange(ny, device=DEV, dtype=F64)[None, :].expand(nx, ny)
        rr = r * (1 + 0.002 * _randn(g, (nx, ny)))  # measured imperfections
        m['x'] = torch.stack([rr * torch.cos(th), rr * torch.sin(th), ax + 0.0], 2).reshape(-1, 3).contiguous()
        m['conn'] = _quads(nx, ny, wrap=True)
        m['xmat'] = torch.tensor([0.02, 0.01, 1.], dtype=F64, device=DEV) if case['direction'] else None
        return m
    if k == 'panel':
        n = case['nel'] + 1
        m['x'], m['conn'], m['edge'] = _plate({'nx': n, 'ny': n}, g, 1.0, 1.0, 0.05)
        ids = torch.arange(n * n, device=DEV, dtype=I64).reshape(n, n)
        rows = [case['nel'] // 10 * j for j in range(1, 10)]
        m['beam'] = torch.cat([torch.stack([ids[:-1, r], ids[1:, r]], 1) for r in rows])
        m['bk'] = _mask(m['edge'], (2,), n * n)
        e = torch.zeros(n, n, dtype=torch.bool, device=DEV)
        e[0] = True
        m['bk'] |= _mask(e.reshape(-1), (0,), n * n)
        e = torch.zeros(n, n, dtype=torch.bool, device=DEV)
        e[:, 0] = True
        m['bk'] |= _mask(e.reshape(-1), (1,), n * n)
        return m
    if k == 'batch':
        P = case['plates']
        rng = np.random.default_rng((P, case['nmin'], case['nmax']))
        nx, ny = rng.integers(case['nmin'], case['nmax'] + 1, (2, P)) + 1
        clamped = rng.integers(0, 2, P)
        rng = np.random.default_rng(seed)
        a, b = rng.uniform(0.5, 2.0, (2, P))
        m['shape'] = list(zip(nx.tolist(), ny.tolist()))
        m['E'], m['nu'], m['h'] = rng.uniform(50e9, 210e9, P), rng.uniform(0.25, 0.35, P), rng.uniform(0.005, 0.02, P)
        xs, cs, bs, fs, inst, pid, n0 = [], [], [], [], [], [], 0
        for i, (p, q) in enumerate(m['shape']):
            x, c, edge = _plate({'nx': p, 'ny': q}, g, a[i], b[i], 0.0)
            f = torch.zeros(p * q, 6, dtype=F64, device=DEV)
            f[(p // 2) * q + q // 2, 2] = -1000.
            bk = _mask(edge, range(6) if clamped[i] else (0, 1, 2), p * q)
            xs.append(x), cs.append(c + n0), bs.append(bk), fs.append(f.reshape(-1))
            inst.append(torch.full((6 * p * q,), i, dtype=torch.int32, device=DEV))
            pid.append(torch.full((c.shape[0],), i, dtype=torch.int32, device=DEV))
            n0 += p * q
        m['x'], m['conn'], m['bk'], m['f'] = (torch.cat(v) for v in (xs, cs, bs, fs))
        m['inst'], m['pid'] = torch.cat(inst), torch.cat(pid)
        m['f'][m['bk']] = 0.
        return m
    m['x'], m['conn'], m['edge'] = _plate(case, g)
    E, nn = m['conn'].shape[0], case['nx'] * case['ny']
    m['h'] = _thickness(g, 1 if case.get('uniform') else E)
    m['bk'] = _mask(m['edge'], (0, 1, 2) if case.get('clamped') is False else range(6), nn)
    if k == 'tria':
        c = m['conn']
        m['conn'] = torch.stack([c[:, [0, 1, 2]], c[:, [0, 2, 3]]], 1).reshape(-1, 3).contiguous()
        m['h'] = m['h'].repeat_interleave(2)
    if k == 'kgm':
        X, Y = m['x'][:, 0], m['x'][:, 1]
        u = torch.zeros(nn, 6, dtype=F64, device=DEV)
        u[:, 0] = -1e-4 * X + 2e-5 * torch.sin(3 * Y)
        u[:, 1] = 3e-5 * Y + 1e-5 * torch.cos(2 * X)
        u[:, 2] = 1e-3 * torch.sin(math.pi * X / 2) * torch.sin(math.pi * Y / 2)
        u += 1e-7 * _randn(g, (nn, 6))
        m['u'] = u.reshape(-1)
    if k in ('steps', 'solve'):
        f = torch.zeros(nn, 6, dtype=F64, device=DEV)
        if case.get('clamped') is False:
            f[(case['nx'] // 2) * case['ny'] + case['ny'] // 2, 2] = -1000.  # centre point load
        else:
            f[:, 2] = -1. - 0.1 * _rand(g, nn, 0., 1.)
        m['f'] = f.reshape(-1)
        m['f'][m['bk']] = 0.
    return m


class State:
    pass


def prepare(case, seed):
    s, m, k = State(), _inputs(case, seed), case['kind']
    s.kind, s.case = k, case
    s.x = m['x'].reshape(-1)
    s.cdof = 6 * m['conn']
    E, N = s.cdof.shape[0], 2 * s.x.numel()
    s.pid = None
    if k in ('shell', 'panel'):
        s.props = torch.from_numpy(shell_record(_laminate())[None, :]).to(DEV)
    elif k == 'batch':
        s.props = isotropic_plate_records_device(m['h'], m['E'], m['nu'])
        s.pid = m['pid']
    else:
        s.props = isotropic_plate_records_device(m['h'], E_MOD, NU, RHO)
        s.pid = _pid(E) if m['h'].numel() > 1 else None
    if k in ('triplets', 'assemble'):
        s.init_k = _offsets(E, 576)
        s.r, s.c, s.v = _coo(576 * E)
        if k == 'assemble':
            batch.quad4_update_KC0(s.r, s.c, s.v, s.x, s.cdof, s.init_k, s.props, pid=s.pid)
            s.pat = CSRPattern(s.r, s.c, N, m['bk'])
            s.out = torch.empty(s.pat.nnz, dtype=F64, device=DEV)
            s.r = s.c = None
    elif k == 'shell':
        s.init_k = _offsets(E, 576)
        s.v = torch.zeros(576 * E, dtype=F64, device=DEV)
        s.xmat = m['xmat']
    elif k == 'tria':
        s.init_k = _offsets(E, 324)
        s.r, s.c, s.v = _coo(324 * E)
    elif k == 'kgm':
        s.u = m['u']
        s.ik_g, s.ik_m = _offsets(E, 144), _offsets(E, 288 if case['mtype'] == 2 else 480)
        s.kg, s.m = _coo(144 * E), _coo((288 if case['mtype'] == 2 else 480) * E)
    else:
        groups = [s.cdof]
        if k == 'panel':
            s.beam = 6 * m['beam']
            s.beam_ik = _offsets(s.beam.shape[0], 144)
            s.beam_v = torch.zeros(144 * s.beam.shape[0], dtype=F64, device=DEV)
            s.beam_props = torch.from_numpy(beam_record(_stringer())[None, :]).to(DEV)
            s.vxy = torch.tensor([0., 1., 0.], dtype=F64, device=DEV)
            groups.append(s.beam)
        s.pat = ElementPattern(groups, N, m['bk'])
        s.fmap = FusedMap(s.pat, groups)
        s.vals = s.fmap.new_values()
        if k in ('steps', 'solve', 'batch'):
            s.f = s.pat.reduce(m['f'])
            s.solver = (BatchSolver(s.pat, m['inst'], case['plates']) if k == 'batch' else Solver(s.pat))
        if k == 'steps':
            batch.quad4_update_KC0_csr(s.vals, s.fmap, s.x, s.props, pid=s.pid)
            s.solver.setup(s.vals)
    return s


def run(s):
    k = s.kind
    if k == 'triplets':
        s.v.zero_()
        batch.quad4_update_KC0(s.r, s.c, s.v, s.x, s.cdof, s.init_k, s.props, pid=s.pid)
        return {'r': s.r, 'c': s.c, 'v': s.v}
    if k == 'shell':
        s.v.zero_()
        batch.quad4_update_KC0(None, None, s.v, s.x, s.cdof, s.init_k, s.props, xmat=s.xmat, update_KC0v_only=1)
        return {'v': s.v}
    if k == 'tria':
        s.v.zero_()
        batch.tria3r_update_KC0(s.r, s.c, s.v, s.x, s.cdof, s.init_k, s.props, pid=s.pid)
        return {'r': s.r, 'c': s.c, 'v': s.v}
    if k == 'kgm':
        s.kg[2].zero_()
        s.m[2].zero_()
        batch.quad4_update_KG(*s.kg, s.x, s.u, s.cdof, s.ik_g, s.props, pid=s.pid)
        batch.quad4_update_M(*s.m, s.x, s.cdof, s.ik_m, s.props, pid=s.pid, mtype=s.case['mtype'])
        return {'kgr': s.kg[0], 'kgc': s.kg[1], 'kgv': s.kg[2], 'mr': s.m[0], 'mc': s.m[1], 'mv': s.m[2]}
    if k == 'assemble':
        return {'vals': s.pat.assemble(s.v, out=s.out)}
    if k == 'steps':
        n = s.case['iters']
        u, _ = s.solver.solve(s.f, tol=1e-300, maxiter=n, check_every=n + (n & 1))
        return {'u': u}
    batch.quad4_update_KC0_csr(s.vals, s.fmap, s.x, s.props, pid=s.pid)
    if k == 'panel':
        s.beam_v.zero_()
        batch.beamc_update_KC0(None, None, s.beam_v, s.x, s.beam, s.beam_ik, s.vxy, s.beam_props,
                               update_KC0v_only=1)
        s.fmap.scatter(s.vals, 1, s.beam_ik, s.beam_v)
        return {'vals': s.vals}
    if k == 'csr':
        return {'vals': s.vals}
    u, _ = s.solver.setup(s.vals).solve(s.f, tol=TOL)
    return {'u': u, 'vals': s.vals}


def work(case):
    k = case['kind']
    if k == 'panel':
        nel = case['nel']
        nnz = 54. * 6 * (nel + 1) ** 2
        return {'bytes': 8 * nnz + nel * nel * 60 + 9 * nel * 40, 'flops': 6000. * nel * nel}
    if k == 'batch':
        n = (case['nmin'] + case['nmax']) / 2.
        nodes = case['plates'] * (n + 1) ** 2
        nnz = 54. * 6 * nodes
        return {'bytes': 8 * nnz + nodes * 120., 'flops': 2 * nnz * 150. * n + 3000. * nodes}
    nx, ny = case['nx'], case['ny']
    nodes, quads = nx * ny, (nx - 1) * (ny - 1)
    nnz = 54. * 6 * nodes
    geo = 44. + 24.                       # DOF offsets, first slot, property id, coordinates
    rec = 8. if case.get('uniform') else 224.  # property record
    if k == 'triplets':
        return {'bytes': quads * (576. * 24 + geo + rec), 'flops': 3000. * quads}
    if k == 'shell':
        return {'bytes': (nx - 1) * ny * (576. * 8 + geo), 'flops': 9000. * (nx - 1) * ny}
    if k == 'tria':
        return {'bytes': 2 * quads * (324. * 24 + geo + rec), 'flops': 2 * 1500. * quads}
    if k == 'kgm':
        slots = 288 if case['mtype'] == 2 else 480
        return {'bytes': quads * ((144. + slots) * 24 + 2 * (geo + rec) + 48), 'flops': 2000. * quads}
    if k == 'assemble':
        return {'bytes': quads * 576. * 8 + nnz * 8, 'flops': 576. * quads}
    if k == 'csr':
        return {'bytes': 8 * nnz + quads * (geo + rec), 'flops': 3000. * quads}
    iters = case['iters'] if k == 'steps' else 160. * max(nx, ny)
    flops = iters * (2 * nnz + nodes * 6 * 24.)
    if k == 'steps':
        return {'bytes': iters * (8 * nnz + nodes * 6 * 8 * 14.), 'flops': flops}
    return {'bytes': 8 * nnz + nodes * 6 * 16. + quads * (geo + rec), 'flops': flops + 3000. * quads}


# ------------------------------------------------------- 64-bit references

def _section(case, m, e0, e1):
    """(ABD (., 6, 6), E44, E45, E55, h, rho-integral I0, I2) of elements e0..e1 (or one for all)."""
    k = case['kind']
    if k in ('shell', 'panel'):
        e1m, e2m, nu12, g12, g13, g23 = LAMINA
        d = 1 - nu12 * nu12 * e2m / e1m
        q11, q12, q22 = e1m / d, nu12 * e2m / d, e2m / d
        C = np.zeros((6, 6))
        S = np.zeros((2, 2))
        z = -PLY_T * len(PLIES) / 2
        for deg in PLIES:
            t = math.radians(deg)
            c, s = math.cos(t), math.sin(t)
            T = np.array([[c * c, s * s, -2 * s * c], [s * s, c * c, 2 * s * c], [s * c, -s * c, c * c - s * s]])
            Q = T @ np.array([[q11, q12, 0], [q12, q22, 0], [0, 0, g12]]) @ T.T
            G = np.array([[g23 * c * c + g13 * s * s, (g13 - g23) * s * c],
                          [(g13 - g23) * s * c, g13 * c * c + g23 * s * s]])
            z1 = z + PLY_T
            C[:3, :3] += Q * (z1 - z)
            C[:3, 3:] += Q * (z1 ** 2 - z ** 2) / 2
            C[3:, 3:] += Q * (z1 ** 3 - z ** 3) / 3
            S += G * (z1 - z)
            z = z1
        C[3:, :3] = C[:3, 3:].T
        t = lambda v: torch.tensor([v], dtype=F64, device=DEV)  # noqa: E731
        return (torch.from_numpy(C).to(DEV)[None], t(S[0, 0] * 5 / 6), t(S[0, 1] * 5 / 6), t(S[1, 1] * 5 / 6),
                t(PLY_T * len(PLIES)), t(0.), t(0.))
    if k == 'batch':
        p = m['pid'][e0:e1].to(I64)
        h, Em, nu = (torch.from_numpy(np.asarray(m[q])).to(DEV)[p] for q in ('h', 'E', 'nu'))
    else:
        h = m['h'] if m['h'].numel() == 1 else m['h'][e0:e1]
        Em, nu = torch.full_like(h, E_MOD), torch.full_like(h, NU)
    ABD = torch.zeros(h.numel(), 6, 6, dtype=F64, device=DEV)
    q, G = Em / (1 - nu * nu), Em / (2 * (1 + nu))
    for o, f in ((0, h), (3, h ** 3 / 12)):
        ABD[:, o, o] = ABD[:, o + 1, o + 1] = q * f
        ABD[:, o, o + 1] = ABD[:, o + 1, o] = nu * q * f
        ABD[:, o + 2, o + 2] = G * f
    return ABD, G * h * 5 / 6, torch.zeros_like(h), G * h * 5 / 6, h, RHO * h, RHO * h ** 3 / 12


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _quad_frame(X):
    """R (E, 3, 3) with columns x, y, z and node coordinates (E, 4, 2) in the element axes (from node 1)."""
    v13, v42 = X[:, 2] - X[:, 0], X[:, 1] - X[:, 3]
    z = _unit(torch.linalg.cross(v42, v13))
    xa = _unit(v13 + v42)
    y = _unit(torch.linalg.cross(z, xa))
    R = torch.stack([xa, y, z], 2)
    return R, ((X - X[:, :1]) @ R)[:, :, :2]


def _shape(xy, xi, eta):
    dev = dict(dtype=F64, device=DEV)
    sx, sy = torch.tensor([-1., 1., 1., -1.], **dev), torch.tensor([-1., -1., 1., 1.], **dev)
    N = (1 + sx * xi) * (1 + sy * eta) / 4
    d = torch.stack([sx * (1 + sy * eta) / 4, sy * (1 + sx * xi) / 4])
    J = d @ xy
    det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
    D = torch.stack([J[:, 1, 1, None] * d[0] - J[:, 0, 1, None] * d[1],
                     J[:, 0, 0, None] * d[1] - J[:, 1, 0, None] * d[0]], 1) / det[:, None, None]
    return N.expand(xy.shape[0], 4), D[:, 0], D[:, 1], det


def _strain_rows(N, Nx, Ny, nn):
    """Membrane-bending rows (E, 6, 6 nn), shear rows (y, x) without and with N, drilling row."""
    E = Nx.shape[0]
    B = torch.zeros(E, 6, 6 * nn, dtype=F64, device=DEV)
    g = torch.zeros(4, E, 6 * nn, dtype=F64, device=DEV)
    dr = torch.zeros(E, 6 * nn, dtype=F64, device=DEV)
    B[:, 0, 0::6], B[:, 1, 1::6] = Nx, Ny
    B[:, 2, 0::6], B[:, 2, 1::6] = Ny, Nx
    B[:, 3, 4::6], B[:, 4, 3::6] = Nx, -Ny
    B[:, 5, 3::6], B[:, 5, 4::6] = -Nx, Ny
    g[0, :, 2::6], g[1, :, 3::6] = Ny, -N
    g[2, :, 2::6], g[3, :, 4::6] = Nx, N
    dr[:, 0::6], dr[:, 1::6], dr[:, 5::6] = Ny / 2, -Nx / 2, N
    return B, g, dr


def _outer(a, b, w):
    return (w[:, None] * a)[:, :, None] * b[:, None, :]


def _turn(K, R, nn):
    T = torch.zeros(R.shape[0], 6 * nn, 6 * nn, dtype=F64, device=DEV)
    for i in range(2 * nn):
        T[:, 3 * i:3 * i + 3, 3 * i:3 * i + 3] = R
    return T @ K @ T.transpose(1, 2)


def _quad_kc0(X, sec, xmat=None):
    """Global 24 x 24 matrices of Quad4 elements with node coordinates X (E, 4, 3)."""
    ABD, E44, E45, E55, h = (s.expand(X.shape[0], *s.shape[1:]) for s in sec[:5])
    R, xy = _quad_frame(X)
    if xmat is not None:
        z = R[:, :, 2]
        xm = _unit(xmat[None].expand(X.shape[0], 3))
        xm = _unit(torch.linalg.cross(_unit(torch.linalg.cross(z, xm)), z))
        c = (xm * R[:, :, 0]).sum(1)
        s = torch.sqrt(1 - c * c)
        s = torch.where((xm * R[:, :, 1]).sum(1) > 0, -s, s)
        T = torch.zeros(X.shape[0], 6, 6, dtype=F64, device=DEV)
        rows = ((c * c, s * s, 2 * c * s), (s * s, c * c, -2 * c * s), (-c * s, c * s, c * c - s * s))
        for o in (0, 3):
            for i in range(3):
                for j in range(3):
                    T[:, o + i, o + j] = rows[i][j]
        ABD = T @ ABD @ T.transpose(1, 2)
    d13, d24 = xy[:, 2] - xy[:, 0], xy[:, 3] - xy[:, 1]
    area = 0.5 * (d13[:, 0] * d24[:, 1] - d13[:, 1] * d24[:, 0]).abs()
    thick = (h / torch.sqrt(area) >= 1).to(F64)
    K = torch.zeros(X.shape[0], 24, 24, dtype=F64, device=DEV)
    p = 1 / math.sqrt(3.)
    for xi in (-p, p):
        for eta in (-p, p):
            N, Nx, Ny, det = _shape(xy, xi, eta)
            B, g, dr = _strain_rows(N, Nx, Ny, 4)
            K += B.transpose(1, 2) @ (det[:, None, None] * (ABD @ B))
            K += _outer(dr, dr, det)
            w = det * thick
            K += _outer(g[0], g[0], w * E44) + _outer(g[0], g[2], w * E45) + _outer(g[2], g[0], w * E45) + \
                _outer(g[2], g[2], w * E55)
    N, Nx, Ny, det = _shape(xy, 0., 0.)
    _, g, _ = _strain_rows(N, Nx, Ny, 4)
    w = 4 * det
    gy, gx = g[0] + g[1], g[2] + g[3]
    K += _outer(gy, gy, w * E44) + _outer(gy, gx, w * E45) + _outer(gx, gy, w * E45) + _outer(gx, gx, w * E55)
    w = w * thick
    K -= _outer(g[0], g[0], w * E44) + _outer(g[0], g[2], w * E45) + _outer(g[2], g[0], w * E45) + \
        _outer(g[2], g[2], w * E55)
    return _turn(K, R, 4)


def _tria_kc0(X, sec, k6rot=100., alpha=0.7):
    ABD, E44, E45, E55, h = (s.expand(X.shape[0], *s.shape[1:]) for s in sec[:5])
    v12, v13 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
    z, xa = _unit(torch.linalg.cross(v12, v13)), _unit(v12)
    R = torch.stack([xa, _unit(torch.linalg.cross(z, xa)), z], 2)
    xy = ((X - X[:, :1]) @ R)[:, :, :2]
    x, y = xy[:, :, 0], xy[:, :, 1]
    area = 0.5 * (x[:, 1] * y[:, 2] - x[:, 2] * y[:, 1]).abs()
    Nx = torch.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], 1) / (2 * area[:, None])
    Ny = torch.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], 1) / (2 * area[:, None])
    lmax = torch.stack([(xy[:, i] - xy[:, j]).norm(dim=1) for i, j in ((0, 1), (1, 2), (2, 0))], 1).max(1).values
    f = 1 / (1 + alpha * lmax ** 2 / h ** 2)
    B, g, _ = _strain_rows(torch.full_like(Nx, 1 / 3.), Nx, Ny, 3)
    K = B.transpose(1, 2) @ (area[:, None, None] * (ABD @ B))
    gy, gx, w = g[0] + g[1], g[2] + g[3], area * f
    K += _outer(gy, gy, w * E44) + _outer(gy, gx, w * E45) + _outer(gx, gy, w * E45) + _outer(gx, gx, w * E55)
    kd = 1e-6 * k6rot * ABD[:, 2, 2]
    Kd = torch.zeros_like(K)
    for a, b in ((2 / 3., 1 / 6.), (1 / 6., 1 / 6.), (1 / 6., 2 / 3.)):
        N = torch.tensor([a, b, 1 - a - b], dtype=F64, device=DEV).expand_as(Nx)
        dr = _strain_rows(N, Nx, Ny, 3)[2]
        Kd += _outer(dr, dr, kd * area / 3)
    K += Kd
    rz = torch.zeros(18, dtype=torch.bool, device=DEV)
    rz[5::6] = True
    drop = (rz[:, None] | rz[None, :]) & ~torch.eye(18, dtype=torch.bool, device=DEV)
    K[:, drop] = 0.  # update_KC0 keeps only the diagonal of the drilling rotations
    return _turn(K, R, 3)


def _beam_kc0(X, p, vxy):
    """Global 12 x 12 matrices of BeamC elements (consistent Timoshenko, no offsets)."""
    d = X[:, 1] - X[:, 0]
    L = d.norm(dim=1)
    xa = d / L[:, None]
    z = _unit(torch.linalg.cross(xa, vxy[None].expand_as(xa)))
    R = torch.stack([xa, _unit(torch.linalg.cross(z, xa)), z], 2)
    K = torch.zeros(X.shape[0], 12, 12, dtype=F64, device=DEV)

    def put(i, j, v):
        K[:, i, j] = v
        K[:, j, i] = v
    for i, v in ((0, p.A * p.E / L), (3, p.G * p.J / L)):
        put(i, i, v), put(i + 6, i + 6, v), put(i, i + 6, -v)
    for I, (v1, t1), s in ((p.Izz, (1, 5), 1.), (p.Iyy, (2, 4), -1.)):
        al = 12 * p.E * I / (p.G * p.A * L * L)
        be2 = 1 / (1 - al) ** 2
        EI = p.E * I
        w = p.A * p.G * L * L * al * al
        kv = be2 * (w + 12 * EI) / L ** 3
        kr = s * be2 * (w + 12 * EI) / (2 * L ** 2)
        k1 = be2 * (w / 4 + EI * al * al - 2 * EI * al + 4 * EI) / L
        k2 = be2 * (w / 4 - EI * al * al + 2 * EI * al + 2 * EI) / L
        v2, t2 = v1 + 6, t1 + 6
        put(v1, v1, kv), put(v2, v2, kv), put(v1, v2, -kv)
        put(v1, t1, kr), put(v1, t2, kr), put(t1, v2, -kr), put(v2, t2, -kr)
        put(t1, t1, k1), put(t2, t2, k1), put(t1, t2, k2)
    return _turn(K, R, 2)


def _kc0_all(case, m, chunk=100000):
    """KC0 of all shell elements (E, n, n)."""
    E, nn = m['conn'].shape
    n = 6 * nn
    K = torch.empty(E, n, n, dtype=F64, device=DEV)
    for e0 in range(0, E, chunk):
        e1 = min(E, e0 + chunk)
        X = m['x'][m['conn'][e0:e1]]
        sec = _section(case, m, e0, e1)
        K[e0:e1] = _tria_kc0(X, sec) if nn == 3 else _quad_kc0(X, sec, m.get('xmat'))
    return K


def _kg_m(case, m, chunk=100000):
    KG, M = [], []
    p = 1 / math.sqrt(3.)
    for e0 in range(0, m['conn'].shape[0], chunk):
        c = m['conn'][e0:e0 + chunk]
        X, E = m['x'][c], c.shape[0]
        ABD, _, _, _, _, I0, I2 = (s.expand(E, *s.shape[1:]) for s in _section(case, m, e0, e0 + E))
        R, xy = _quad_frame(X)
        u = m['u'].reshape(-1, 2, 3)[c]                       # (E, 4, 2, 3)
        ue = (u.reshape(E, 8, 3) @ R).reshape(E, 24)
        G = torch.zeros(E, 4, 4, dtype=F64, device=DEV)
        H = torch.zeros(E, 4, 4, dtype=F64, device=DEV)
        for xi in (-1., 1.):
            for eta in (-1., 1.):
                N, Nx, Ny, det = _shape(xy, p * xi, p * eta)
                S = (ABD @ (_strain_rows(N, Nx, Ny, 4)[0] @ ue[:, :, None]))[:, :3, 0]
                G += _outer(Nx, Nx, det * S[:, 0]) + _outer(Ny, Ny, det * S[:, 1]) + \
                    _outer(Nx, Ny, det * S[:, 2]) + _outer(Ny, Nx, det * S[:, 2])
                if case['mtype'] == 2:
                    N, _, _, det = _shape(xy, xi, eta)
                H += _outer(N, N, det)
        if case['mtype'] == 1:
            d13, d24 = xy[:, 2] - xy[:, 0], xy[:, 3] - xy[:, 1]
            area = 0.5 * (d13[:, 0] * d24[:, 1] - d13[:, 1] * d24[:, 0]).abs()
            H = (area / 16)[:, None, None].expand(E, 4, 4)
        n = R[:, :, 2]
        KG.append(torch.einsum('ei,ej,eab->eaibj', n, n, G).reshape(E, 144))
        U = torch.zeros(E, 6, 6, dtype=F64, device=DEV)       # unit mass in global axes
        U[:, :3, :3] = torch.eye(3, dtype=F64, device=DEV) * I0[:, None, None]
        U[:, 3:, 3:] = I2[:, None, None] * (R[:, :, :2] @ R[:, :, :2].transpose(1, 2))
        i = torch.arange(6, device=DEV)
        keep = ((i[:, None] < 3) == (i[None, :] < 3)) if case['mtype'] == 2 else ((i[:, None] - i[None, :]).abs() != 3)
        full = torch.einsum('emn,eab->eambn', U, H)
        M.append(full.permute(0, 1, 2, 3, 4).reshape(E, -1)[:, keep[None, :, None, :].expand(4, 6, 4, 6).reshape(-1)]
                 .reshape(-1))
    return torch.cat(KG).reshape(-1), torch.cat(M)


def _reduced(groups, bk):
    """Sorted unique (row, column) keys and summed values of [(dofs (E, n), K (E, n, n))] over the free DOFs."""
    free = ~bk
    num = torch.cumsum(free.to(I64), 0) - 1
    nf = int(free.sum())
    keys, vals = [], []
    for dofs, K in groups:
        E, n = dofs.shape
        r, c = dofs[:, :, None].expand(E, n, n).reshape(-1), dofs[:, None, :].expand(E, n, n).reshape(-1)
        ok = free[r] & free[c]
        keys.append((num[r] * nf + num[c])[ok])
        vals.append(K.reshape(-1)[ok])
    keys, vals = torch.cat(keys), torch.cat(vals)
    uniq, at = torch.unique(keys, return_inverse=True)
    return uniq, torch.zeros(uniq.numel(), dtype=F64, device=DEV).index_add_(0, at, vals), nf


def _dofs(conn):
    return (6 * conn[:, :, None] + torch.arange(6, device=DEV)).reshape(conn.shape[0], -1)


def _line_solve(nx, ny, conn, K, bk, f):
    """Direct solve of a structured plate, block tridiagonal over its nx node lines, with refinement."""
    b = 6 * ny
    d = _dofs(conn)
    n = d.shape[1]
    r, c = d[:, :, None].expand(-1, n, n).reshape(-1), d[:, None, :].expand(-1, n, n).reshape(-1)
    ok = ~(bk[r] | bk[c])
    r, c, v = r[ok], c[ok], K.reshape(-1)[ok]
    D = torch.zeros(nx, b, b, dtype=F64, device=DEV)
    U = torch.zeros(nx - 1, b, b, dtype=F64, device=DEV)
    lr, lc = r // b, c // b
    for blk, sel in ((D, lr == lc), (U, lc == lr + 1)):
        blk.view(-1).index_add_(0, (lr[sel] * b + r[sel] % b) * b + c[sel] % b, v[sel])
    D.diagonal(dim1=1, dim2=2).add_(bk.to(F64).reshape(nx, b))
    ch, W = [], []
    for i in range(nx):
        S = D[i] if i == 0 else D[i] - U[i - 1].T @ W[-1]
        ch.append(torch.linalg.cholesky(S))
        if i < nx - 1:
            W.append(torch.cholesky_solve(U[i], ch[-1]))

    def solve(g):
        y = []
        for i in range(nx):
            y.append(torch.cholesky_solve(g[i] if i == 0 else g[i] - U[i - 1].T @ y[-1], ch[i]))
        for i in range(nx - 2, -1, -1):
            y[i] = y[i] - W[i] @ y[i + 1]
        return torch.stack(y)
    g = f.reshape(nx, b, 1)
    x = solve(g)
    for _ in range(2):
        res = g - D @ x
        res[:-1] -= U @ x[1:]
        res[1:] -= U.transpose(1, 2) @ x[:-1]
        x = x + solve(res)
    return x.reshape(-1)[~bk]


def _pcg(keys, vals, nf, f, iters):
    """Plain block-Jacobi PCG from zero (all six DOFs of a node free or none)."""
    r, c = keys // nf, keys % nf
    ptr = torch.searchsorted(r, torch.arange(nf + 1, device=DEV))
    A = torch.sparse_csr_tensor(ptr, c, vals, (nf, nf))
    own = r // 6 == c // 6
    B = torch.zeros(nf // 6, 6, 6, dtype=F64, device=DEV)
    B[r[own] // 6, r[own] % 6, c[own] % 6] = vals[own]
    Bi = torch.linalg.inv(B)
    pre = lambda v: (Bi @ v.reshape(-1, 6, 1)).reshape(-1)  # noqa: E731
    u, res = torch.zeros_like(f), f.clone()
    z = pre(res)
    p, rz = z.clone(), res @ z
    for _ in range(iters):
        q = A @ p
        al = rz / (p @ q)
        u, res = u + al * p, res - al * q
        z = pre(res)
        rz, old = res @ z, rz
        p = z + (rz / old) * p
    return u


def exact(case, seed):
    m, k = _inputs(case, seed), case['kind']
    if k == 'kgm':
        kg, mass = _kg_m(case, m)
        return {'kgr': None, 'kgc': None, 'kgv': kg, 'mr': None, 'mc': None, 'mv': mass}
    K = _kc0_all(case, m)
    if k in ('triplets', 'tria'):
        return {'r': None, 'c': None, 'v': K.reshape(-1)}
    if k == 'shell':
        return {'v': K.reshape(-1)}
    groups = [(_dofs(m['conn']), K)]
    if k == 'panel':
        vxy = torch.tensor([0., 1., 0.], dtype=F64, device=DEV)
        groups.append((_dofs(m['beam']), _beam_kc0(m['x'][m['beam']], _stringer(), vxy)))
    keys, vals, nf = _reduced(groups, m['bk'])
    if k in ('csr', 'panel', 'assemble'):
        return {'vals': vals}
    if k == 'steps':
        return {'u': _pcg(keys, vals, nf, m['f'][~m['bk']], case['iters'])}
    if k == 'solve':
        return {'u': _line_solve(case['nx'], case['ny'], m['conn'], K, m['bk'], m['f']), 'vals': vals}
    us, n0, e0 = [], 0, 0
    for nx, ny in m['shape']:
        e1, d = e0 + (nx - 1) * (ny - 1), slice(6 * n0, 6 * (n0 + nx * ny))
        us.append(_line_solve(nx, ny, m['conn'][e0:e1] - n0, K[e0:e1], m['bk'][d], m['f'][d]))
        n0, e0 = n0 + nx * ny, e1
    return {'u': torch.cat(us), 'vals': vals}

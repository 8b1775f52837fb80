"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case is a set of em2d runs driven through the Python binding (``zpic_b200``): a simulation with its
species is what the program has in hand, one pass advances it by the steps between two dumps and takes
the dump (fields and charge densities; energies where a program reads them every step).  The inputs --
particle momenta, laser phases and amplitudes -- are made from the seed.

``exact`` restates the em2d step (Boris push, charge-conserving deposit, Yee solver, boundaries, filters,
moving window) on one global grid in 64-bit torch, without the framework.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.path.abspath('.'), 'zpic-parallel_b200'))
import zpic_b200 as zb  # noqa: E402

BC = {'periodic': (1, 1, 1, 1), 'window': (0, 0, 1, 1), 'walls': (2, 2, 1, 1)}

# Defaults of a case: 0.1 cells, dt 0.07, periodic, one species of electrons.
BASE = {'kind': 'advance', 'ntx': 8, 'nty': 8, 'nxx': 16, 'nxy': 16, 'dx': 0.1, 'dy': 0.1, 'dt': 0.07,
        'species': 1, 'ppcx': 4, 'ppcy': 4, 'uth': 0.1, 'uz': 0.0, 'steps': 20, 'bounds': 'periodic',
        'euler': 0, 'filter': 'none', 'filter_dir': 0, 'filter_order': 1, 'laser': 0, 'edge': -1.0,
        'runs': 1, 'mix': 0}


def _case(**kw):
    c = dict(BASE)
    assert set(kw) <= set(c) | {'name'}
    c.update(kw)
    return c


def listed():
    return [
        # A notebook on a small box: one step at a time, the energies read after each (latency).
        _case(name='notebook_64', kind='notebook', ntx=4, nty=4, species=2, ppcx=2, ppcy=2, uz=0.6, steps=10),
        # A user's own loop over the objects' advance() calls, on a two-stream box of odd tiles.
        _case(name='own_loop_120x112', kind='loop', ntx=5, nty=8, nxx=24, nxy=14, species=2, ppcx=3, ppcy=3, uz=0.4,
              uth=0.05, steps=10),
        # The Weibel test of the reference's driver: 128x128 cells, two species of 4x4 per cell.
        _case(name='weibel_128', ntx=8, nty=8, species=2, uz=0.6, steps=100),
        # The same instability at the size and tiles of the reference's CUDA driver (32x32 tiles, 8x8 per cell).
        _case(name='weibel_512_tiles32', ntx=16, nty=16, nxx=32, nxy=32, species=2, ppcx=8, ppcy=8, uz=0.6, steps=50),
        # Uniform warm plasma, 16x16 tiles, 8x8 per cell: the throughput workload (at a quarter of its area).
        _case(name='plasma_1024', ntx=64, nty=64, ppcx=8, ppcy=8, uth=0.05, steps=50),
        # A medium production run with few particles per cell: fields and sort weigh as much as the push.
        _case(name='plasma_1024_ppc4', ntx=64, nty=64, ppcx=2, ppcy=2, uth=0.2, steps=100),
        # Laser wakefield in a moving window: 4096x512 cells, 4x2 per cell behind a density step.
        _case(name='lwfa_4096x512', kind='window', bounds='window', ntx=256, nty=32, dx=0.025, dy=0.1, dt=0.022, ppcx=4,
              ppcy=2, uth=0.0, laser=1, edge=20.0, steps=100),
        # The same on a small box with the compensated current filter along the laser's axis.
        _case(name='lwfa_256x64_filter', kind='window', bounds='window', ntx=16, nty=4, dx=0.025, dy=0.1, dt=0.022, ppcx=4,
              ppcy=2, uth=0.0, laser=1, edge=2.0, filter='compensated', filter_order=2, steps=50),
        # A plasma between conducting, reflecting walls with the exact-rotation pusher and a filtered
        # current; odd, oblong tiles.
        _case(name='walls_euler_385x210', bounds='walls', ntx=11, nty=10, nxx=35, nxy=21, species=2, ppcx=3, ppcy=5, uth=0.15,
              euler=1, filter='binomial', filter_dir=1, filter_order=1, steps=50),
        # A parameter sweep: runs of uneven sizes advanced together.
        _case(name='sweep_16_runs', kind='batch', runs=16, mix=1, species=2, steps=50),
        # A laser pulse crossing vacuum: the field solver alone.
        _case(name='vacuum_2048x1024', ntx=128, nty=64, dx=0.05, dy=0.1, dt=0.04, species=0, laser=1, steps=200),
        # One full dump: every field component, charge density, 1D and 2D phase spaces.
        _case(name='dump_512', kind='dump', ntx=32, nty=32, species=2, ppcx=3, ppcy=3, uz=0.3, steps=5),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(['plasma', 'plasma', 'plasma', 'small', 'small', 'loop', 'window', 'window', 'walls', 'batch',
                       'vacuum', 'dump'])
    # tiles: 16x16 in most runs, else anything from 8 to 40 cells a side
    nxx, nxy = (16, 16) if rng.random() < 0.5 else (rng.randint(8, 40), rng.randint(8, 40))
    species = rng.choice([1, 1, 2])
    uth, uz = rng.uniform(0.02, 0.25), (rng.uniform(0.2, 0.8) if species == 2 else 0.0)

    def tiles(cells):
        """Tiles for about `cells` cells, up to 2:1 oblong."""
        nt, r = max(4.0, cells / (nxx * nxy)), _log(rng, 0.5, 2.0)
        return max(2, round(math.sqrt(nt * r))), max(2, round(math.sqrt(nt / r)))

    if kind == 'plasma':
        ppcx, ppcy = rng.randint(2, 8), rng.randint(2, 8)
        ntx, nty = tiles(_log(rng, 6e4, 1.5e7 / (species * ppcx * ppcy)))
        return _case(ntx=ntx, nty=nty, nxx=nxx, nxy=nxy, species=species, ppcx=ppcx, ppcy=ppcy, uth=uth, uz=uz,
                     euler=int(rng.random() < 0.15), steps=rng.choice([25, 50, 100]))
    if kind in ('small', 'loop'):
        ntx, nty = tiles(_log(rng, 2e3, 6e4))
        return _case(kind='loop' if kind == 'loop' else rng.choice(['advance', 'notebook']), ntx=ntx, nty=nty, nxx=nxx,
                     nxy=nxy, species=species, ppcx=rng.randint(1, 5), ppcy=rng.randint(1, 5), uth=uth, uz=uz,
                     steps=rng.randint(8, 40))
    if kind == 'window':
        ntx, nty = max(6, round(_log(rng, 200, 4000) / nxx)), max(2, round(_log(rng, 48, 512) / nxy))
        f = rng.choice(['none', 'none', 'binomial', 'compensated'])
        return _case(kind='window', bounds='window', ntx=ntx, nty=nty, nxx=nxx, nxy=nxy, dx=0.025, dy=0.1, dt=0.022,
                     ppcx=rng.randint(1, 4), ppcy=rng.randint(1, 4), uth=0.0, laser=1, edge=0.2 * ntx * nxx * 0.025,
                     filter=f, filter_order=rng.randint(1, 3), steps=rng.randint(25, 100))
    if kind == 'walls':
        ntx, nty = tiles(_log(rng, 1e4, 3e5))
        f = rng.choice(['none', 'binomial', 'compensated'])
        return _case(bounds='walls', ntx=ntx, nty=nty, nxx=nxx, nxy=nxy, species=species, ppcx=rng.randint(2, 5),
                     ppcy=rng.randint(2, 5), uth=uth, uz=uz, euler=rng.randint(0, 1), filter=f, filter_dir=rng.randint(0, 1),
                     filter_order=rng.randint(1, 2), steps=rng.randint(25, 60))
    if kind == 'batch':
        return _case(kind='batch', runs=rng.randint(6, 20), mix=rng.randint(2, 10000), species=2, steps=rng.choice([25, 50]))
    if kind == 'vacuum':
        ntx, nty = tiles(_log(rng, 2e5, 2e6))
        return _case(ntx=ntx, nty=nty, nxx=nxx, nxy=nxy, dx=0.05, dy=0.1, dt=0.04, species=0, laser=1, steps=rng.randint(50, 200))
    ntx, nty = tiles(_log(rng, 2e4, 4e5))
    return _case(kind='dump', ntx=ntx, nty=nty, nxx=nxx, nxy=nxy, species=species, ppcx=rng.randint(2, 4), ppcy=rng.randint(2, 4),
                 uth=uth, uz=uz, steps=rng.randint(2, 10))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _members(case):
    """The simulations of a case: itself, or the runs of a sweep (sizes, particles per cell and momenta
    as in the ensemble workload, at most 256 cells a side)."""
    if case['kind'] != 'batch':
        return [case]
    r, got = random.Random(case['mix']), []
    for _ in range(case['runs']):
        n, p = r.choice([64, 96, 128, 192, 256]) // 16, r.choice([2, 4, 4, 8])
        got.append(dict(case, ntx=n, nty=n, ppcx=p, ppcy=p, uz=r.uniform(0.2, 0.8), uth=r.uniform(0.02, 0.15)))
    return got


def _cells(c):
    return c['ntx'] * c['nxx'] * c['nty'] * c['nxy']


def _particles(c):
    n = c['species'] * c['ppcx'] * c['ppcy'] * _cells(c)
    if c['edge'] >= 0:
        n = int(n * (1 - c['edge'] / (c['ntx'] * c['nxx'] * c['dx'])))
    return n


def _momenta(c, seed, member, sp):
    """u of one species in tile order: thermal, drifting along z (opposite ways for two species).  Drawn in
    32 bits on the host's or the card's generator, whichever the run has."""
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    g = torch.Generator(device=dev).manual_seed((seed * 64 + member) * 8 + sp + 1)
    n = c['ppcx'] * c['ppcy'] * _cells(c)
    u = torch.randn((n, 3), generator=g, device=dev, dtype=torch.float32).mul_(c['uth'])
    u[:, 2] += c['uz'] * (1 - 2 * sp)
    return u


def _lattice(c):
    """Cells and positions of one tile's particles, in injection order: for every place in the cell, every cell."""
    px = ((np.arange(c['ppcx']) + 0.5) / c['ppcx'] - 0.5).astype(np.float32)
    py = ((np.arange(c['ppcy']) + 0.5) / c['ppcy'] - 0.5).astype(np.float32)
    cy, cx = [a.ravel() for a in np.meshgrid(np.arange(c['nxy']), np.arange(c['nxx']), indexing='ij')]
    np_cell, places = cx.size, c['ppcx'] * c['ppcy']
    ix = np.empty((places, np_cell, 2), np.int32)
    x = np.empty((places, np_cell, 2), np.float32)
    ix[:, :, 0], ix[:, :, 1] = cx, cy
    x[:, :, 0] = np.tile(px, c['ppcy'])[:, None]
    x[:, :, 1] = np.repeat(py, c['ppcx'])[:, None]
    return ix.reshape(-1, 2), x.reshape(-1, 2)


def _laser(c, seed):
    """E, B [3, NY, NX + 3] (x guard columns 1 and 2) of a Gaussian pulse moving along +x, from a vector
    potential A_z, so that B has no divergence on the staggered grid; in 32 bits."""
    r = random.Random(seed)
    nx, ny, dx, dy = c['ntx'] * c['nxx'], c['nty'] * c['nxy'], c['dx'], c['dy']
    lx = nx * dx
    a0, phase = 2.0 * r.uniform(0.9, 1.1), r.uniform(0, 2 * math.pi)
    half = min(2.0, 0.1 * lx)                         # half width of the cos^2 envelope
    x0 = c['edge'] + 1.2 * half if c['edge'] >= 0 else 0.3 * lx
    axis, w0 = 0.5 * ny * dy * r.uniform(0.95, 1.05), min(4.0, 0.15 * ny * dy)
    k = 10.0 if dx < 0.03 else 5.0
    x, y = (np.arange(nx + 4) - 1) * dx - x0, (np.arange(ny + 1) * dy - axis)[:, None]
    env = np.where(np.abs(x) < half, np.cos(0.5 * math.pi * x / half) ** 2, 0.0)
    denv = np.where(np.abs(x) < half, -0.5 * math.pi / half * np.sin(math.pi * x / half), 0.0)
    g = np.exp(-(y / w0) ** 2)
    az = a0 * g * (env * np.sin(k * x + phase))
    ez = a0 * g * (denv * np.sin(k * x + phase) + k * env * np.cos(k * x + phase))
    E, B = np.zeros((2, 3, ny, nx + 3), np.float32)
    E[2] = ez[:ny, :nx + 3]
    B[0] = (az[1:, :nx + 3] - az[:ny, :nx + 3]) / dy
    B[1] = -(az[:ny, 1:] - az[:ny, :nx + 3]) / dx
    return E, B


def _tiled(c, g):
    """[ntiles, tile_vol, 3] blocks with guard cells {1, 2} of g [3, NY, NX + 3] (numpy or torch)."""
    lib = torch if isinstance(g, torch.Tensor) else np
    ntx, nty, nxx, nxy = c['ntx'], c['nty'], c['nxx'], c['nxy']
    rows = (np.arange(nty)[:, None] * nxy + np.arange(-1, nxy + 2)).ravel() % (nty * nxy)
    cols = (np.arange(ntx)[:, None] * nxx + np.arange(nxx + 3)).ravel()
    if lib is torch:
        rows, cols = torch.as_tensor(rows, device=g.device), torch.as_tensor(cols, device=g.device)
    b = g[:, rows][:, :, cols].reshape(3, nty, nxy + 3, ntx, nxx + 3)
    b = b.permute(1, 3, 2, 4, 0) if lib is torch else b.transpose(1, 3, 2, 4, 0)
    b = b.reshape(ntx * nty, (nxx + 3) * (nxy + 3), 3)
    pad = -b.shape[1] % 4
    out = torch.nn.functional.pad(b, (0, 0, 0, pad)) if lib is torch else np.pad(b, ((0, 0), (0, pad), (0, 0)))
    return out


def _wrap_x(g):
    """Periodic x guard columns of [.., NX + 3] arrays, in place."""
    n = g.shape[-1] - 3
    g[..., 0] = g[..., n]
    g[..., n + 1:n + 3] = g[..., 1:3]
    return g


def _build(c, seed, member):
    s = zb.Simulation((c['ntx'], c['nty']), (c['nxx'], c['nxy']),
                      (c['ntx'] * c['nxx'] * c['dx'], c['nty'] * c['nxy'] * c['dy']), c['dt'])
    bc = BC[c['bounds']]
    for sp in range(c['species']):
        m_q = -1.0 if sp == 0 else 1.0
        sbc = bc if c['bounds'] != 'window' else (1, 1, 1, 1)          # set_moving_window opens the x ends
        dens = ('uniform', 1.0) if c['edge'] < 0 else ('step', 1.0, c['edge'], 0)
        s.add_species(m_q, (c['ppcx'], c['ppcy']), density=dens, push_type=c['euler'], bc=sbc)
        if c['edge'] < 0:
            ix, x = _lattice(c)
            nt = c['ntx'] * c['nty']
            s.set_particles(sp, np.full(nt, len(ix), np.int32), np.tile(ix, (nt, 1)), np.tile(x, (nt, 1)),
                            _momenta(c, seed, member, sp).cpu().numpy())
    if c['bounds'] == 'walls':
        s.emf_set_bc(bc)
        s.current_set_bc(bc)
    if c['filter'] != 'none':
        s.current_set_filter(c['filter'], c['filter_dir'], c['filter_order'])
    if c['laser']:
        E, B = _laser(c, seed)
        if c['bounds'] == 'periodic':
            E, B = _wrap_x(E), _wrap_x(B)
        s.set_grid('E', _tiled(c, E))
        s.set_grid('B', _tiled(c, B))
    if c['bounds'] == 'window':
        s.set_moving_window()
    return s


def prepare(case, seed):
    sims = [_build(c, seed, k) for k, c in enumerate(_members(case))]
    if case['kind'] == 'dump':
        sims[0].advance(case['steps'])
    for s in sims:
        s.synchronize()
    return {'case': case, 'sims': sims, 'batch': zb.Batch(sims) if case['kind'] == 'batch' else None}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
PHASE = {'bins': 256, 'range': (-1.5, 1.5)}


def _dump(s, species):
    out = {'E': s.grid('E'), 'B': s.grid('B')}
    for sp in range(species):
        out['rho%d' % sp] = s.charge(sp)
    return out


def run(state):
    c, sims = state['case'], state['sims']
    s, n = sims[0], c['steps']
    if c['kind'] == 'batch':
        state['batch'].advance(n)
        return [_dump(m, 1) for m in sims]
    if c['kind'] == 'dump':
        box = (c['ntx'] * c['nxx'] * c['dx'], c['nty'] * c['nxy'] * c['dy'])
        out = {w + f: s.grid_gather(w, k) for w in 'EBJ' for k, f in enumerate('xyz')}
        for sp in range(c['species']):
            out['rho%d' % sp] = s.charge(sp)
            out['uz%d' % sp] = s.phasespace(sp, 'uz', PHASE['range'], PHASE['bins'])
            out['xuz%d' % sp] = s.phasespace(sp, 'x', (0.0, box[0]), PHASE['bins'], 'uz', PHASE['range'], PHASE['bins'] // 2)
        return out
    energies = []
    if c['kind'] == 'window':
        s.advance_mov_window(n)
    elif c['kind'] == 'advance':
        s.advance(n)
    elif c['kind'] == 'notebook':
        for _ in range(n):
            s.advance(1)
            e, b = s.emf_energy()
            energies.append([*e, *b] + [s.species_energy(sp) for sp in range(c['species'])])
    else:
        for _ in range(n):
            s.current_zero()
            for sp in range(c['species']):
                s.species_advance(sp)
            s.current_advance()
            s.emf_advance()
    out = _dump(s, c['species'])
    if energies:
        out['energies'] = np.array(energies)
    return out


def work(case):
    """Per step: the particle state (24 bytes a particle) read and written, E, B, J read or written by push,
    deposit and field solve (96 bytes a cell); then the dump, each value written once."""
    b = f = 0.0
    for c in _members(case):
        n, cells = _particles(c), _cells(c)
        if c['kind'] == 'dump':
            b += 24.0 * n + 4 * cells * (9 + c['species'])
            f += 30.0 * n
            continue
        b += c['steps'] * (48.0 * n + 96.0 * cells) + cells * (24 + 4 * c['species'])
        f += c['steps'] * (250.0 * n + 60.0 * cells)
    return {'bytes': b, 'flops': f}


def tolerance(case):
    # 32-bit fields, currents and offsets, and currents summed in another order.  Measured over these
    # ranges: up to 3.7e-5 between two runs on the same inputs (magnetic field of a growing Weibel
    # instability, 2.4e-4 in single values), up to 2.7e-5 from the 64-bit step; times about four.
    return {'rel': 1e-4, 'max': 2e-3}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """em2d in float64 on global arrays [3, NY, NX + 3]: y wraps, x has guard columns 1 (left) and 2 (right)."""

    def __init__(self, c, seed, member):
        self.c, self.dev = c, 'cuda' if torch.cuda.is_available() else 'cpu'
        self.nx, self.ny = c['ntx'] * c['nxx'], c['nty'] * c['nxy']
        f32 = np.float32
        self.dx = float(f32(self.nx * c['dx']) / f32(self.nx))
        self.dy = float(f32(self.ny * c['dy']) / f32(self.ny))
        self.dt, self.moved, self.iter, self.periodic = c['dt'], [0, 0], 0, c['bounds'] == 'periodic'
        # self.moved: window moves of the (only) species and of the fields
        self.E, self.B, self.J = (torch.zeros((3, self.ny, self.nx + 3), dtype=torch.float64, device=self.dev) for _ in range(3))
        if c['laser']:
            E, B = _laser(c, seed)
            self.E, self.B = (torch.as_tensor(a, device=self.dev).double() for a in (E, B))
            if self.periodic:
                _wrap_x(self.E), _wrap_x(self.B)
        self.sp = []
        ix, x = _lattice(c)
        t = np.arange(c['ntx'] * c['nty'])
        for k in range(c['species']):
            m_q = -1.0 if k == 0 else 1.0
            px = torch.as_tensor(ix[:, 0] + x[:, 0].astype(np.float64) + 0.5, device=self.dev)
            py = torch.as_tensor(ix[:, 1] + x[:, 1].astype(np.float64) + 0.5, device=self.dev)
            px = (torch.as_tensor((t % c['ntx']) * c['nxx'], device=self.dev)[:, None] + px).reshape(-1)
            py = (torch.as_tensor((t // c['ntx']) * c['nxy'], device=self.dev)[:, None] + py).reshape(-1)
            if c['edge'] >= 0:
                keep = px > float(f32(c['edge']) / f32(self.dx))
                px, py = px[keep], py[keep]
                u = torch.zeros((px.numel(), 3), dtype=torch.float64, device=self.dev)
            else:
                u = _momenta(c, seed, member, k).to(self.dev).double()
            self.sp.append({'m_q': m_q, 'q': math.copysign(1.0, m_q) / (c['ppcx'] * c['ppcy']),
                            'x': px, 'y': py, 'u': u, 'energy': 0.0})

    # fields at the particles, boris rotation
    def _push(self, s, a, b):
        x, y, u = s['x'][a:b], s['y'][a:b], s['u'][a:b]
        w = self.nx + 3

        def at(f, hx, hy):
            fx, fy = torch.floor(x - 0.5 * hx), torch.floor(y - 0.5 * hy)
            wx, wy = x - 0.5 * hx - fx, y - 0.5 * hy - fy
            i, j = fx.long() + 1, fy.long()
            j0, j1 = (j % self.ny) * w + i, ((j + 1) % self.ny) * w + i
            f = f.reshape(-1)
            return (f[j0] * (1 - wx) + f[j0 + 1] * wx) * (1 - wy) + (f[j1] * (1 - wx) + f[j1 + 1] * wx) * wy

        alpha = 0.5 * self.dt / s['m_q']
        e = torch.stack([at(self.E[0], 1, 0), at(self.E[1], 0, 1), at(self.E[2], 0, 0)], 1) * alpha
        m = torch.stack([at(self.B[0], 0, 1), at(self.B[1], 1, 0), at(self.B[2], 1, 1)], 1)
        ut = u + e
        usq = (ut * ut).sum(1)
        gamma = torch.sqrt(1 + usq)
        s['energy'] += float((usq / (gamma + 1)).sum())
        if not self.c['euler']:
            m = m * (alpha / gamma)[:, None]
            v = ut + torch.linalg.cross(ut, m)
            m = m * (2 / (1 + (m * m).sum(1)))[:, None]
            ut = ut + torch.linalg.cross(v, m)
        else:
            # Euler-Rodrigues rotation with the matrix the reference uses
            m = m * (2 * alpha / gamma)[:, None]
            n = m.norm(dim=1)
            sn = torch.where(n > 0, -torch.sin(n / 2) / n, torch.full_like(n, -1.0))
            ra = torch.cos(n / 2)
            rb, rc, rd = (m * sn[:, None]).unbind(1)
            r11, r22 = ra * ra + rb * rb - rc * rc - rd * rd, ra * ra + rc * rc - rb * rb - rd * rd
            r33 = ra * ra + rd * rd - rb * rb + rc * rc
            r12, r13, r21 = 2 * (rb * rc + ra * rd), 2 * (rb * rd - ra * rc), 2 * (rb * rc - ra * rd)
            r23, r31, r32 = 2 * (rc * rd + ra * rb), 2 * (rb * rd + ra * rc), 2 * (rc * rd - ra * rb)
            ux, uy, uz = ut.unbind(1)
            ut = torch.stack([r11 * ux + r21 * uy + r31 * uz, r12 * ux + r22 * uy + r32 * uz, r13 * ux + r23 * uy + r33 * uz], 1)
        s['u'][a:b] = ut + e

    def _segment(self, s, x0, y0, x1, y1, qvz):
        """Current of straight pieces, each inside one cell (the one its middle is in)."""
        i, j = torch.floor(0.5 * (x0 + x1)), torch.floor(0.5 * (y0 + y1))
        ax, bx, ay, by = x0 - i, x1 - i, y0 - j, y1 - j
        w = self.nx + 3
        k0 = (j.long() % self.ny) * w + i.long() + 1
        k1 = ((j.long() + 1) % self.ny) * w + i.long() + 1
        wx, wy = s['q'] * self.dx / self.dt * (x1 - x0), s['q'] * self.dy / self.dt * (y1 - y0)
        my, mx = 0.5 * (ay + by), 0.5 * (ax + bx)
        J = self.J.reshape(3, -1)
        J[0].index_add_(0, k0, wx * (1 - my))
        J[0].index_add_(0, k1, wx * my)
        J[1].index_add_(0, k0, wy * (1 - mx))
        J[1].index_add_(0, k0 + 1, wy * mx)
        for sx0, sx1, kx in ((1 - ax, 1 - bx, 0), (ax, bx, 1)):
            for sy0, sy1, k in ((1 - ay, 1 - by, k0), (ay, by, k1)):
                J[2].index_add_(0, k + kx, 0.5 * qvz * (sx0 * sy0 + sx1 * sy1 + 0.5 * (sx0 * sy1 - sx1 * sy0)))

    def _move(self, s, a, b):
        x0, y0, u = s['x'][a:b], s['y'][a:b], s['u'][a:b]
        rg = 1 / torch.sqrt(1 + (u * u).sum(1))
        dx, dy = self.dt / self.dx * rg * u[:, 0], self.dt / self.dy * rg * u[:, 1]
        x1, y1, qvz = x0 + dx, y0 + dy, s['q'] * u[:, 2] * rg
        cx, cy = torch.floor(x0) != torch.floor(x1), torch.floor(y0) != torch.floor(y1)
        one = ~(cx | cy)
        self._segment(s, x0[one], y0[one], x1[one], y1[one], qvz[one])
        k = (~one).nonzero()[:, 0]
        if k.numel():
            # the fractions of the step at which a cell edge is crossed, in order
            def cut(p, d, c):
                edge = torch.where(d > 0, torch.floor(p) + 1, torch.floor(p))
                return torch.where(c, (edge - p) / torch.where(c, d, torch.ones_like(d)), torch.ones_like(d))
            px, py, ddx, ddy, q = x0[k], y0[k], dx[k], dy[k], qvz[k]
            tx, ty = cut(px, ddx, cx[k]), cut(py, ddy, cy[k])
            t = [torch.zeros_like(tx), torch.minimum(tx, ty), torch.maximum(tx, ty), torch.ones_like(tx)]
            for p in range(3):
                self._segment(s, px + ddx * t[p], py + ddy * t[p], px + ddx * t[p + 1], py + ddy * t[p + 1], q * (t[p + 1] - t[p]))
        s['x'][a:b], s['y'][a:b] = x1, y1

    def _advance_species(self, s):
        s['energy'] = 0.0
        for a in range(0, s['x'].numel(), 1 << 23):
            b = min(s['x'].numel(), a + (1 << 23))
            self._push(s, a, b)
            self._move(s, a, b)
        s['y'] %= self.ny
        # a species' clock runs in 32 bits (steps at which the window is due to the last bit are common)
        moving = self.c['bounds'] == 'window' and float(np.float32(self.iter + 1) * np.float32(self.dt)) > self.dx * (self.moved[0] + 1)
        if self.periodic:
            s['x'] %= self.nx
        elif self.c['bounds'] == 'walls':
            lo, hi = s['x'] < 0, s['x'] >= self.nx
            s['x'] = torch.where(lo, -s['x'], torch.where(hi, 2 * self.nx - s['x'], s['x']))
            flip = lo | hi
            s['u'][:, 0] = torch.where(flip, -s['u'][:, 0], s['u'][:, 0])
        else:
            if moving:
                s['x'] -= 1
            keep = (s['x'] >= 0) & (s['x'] < self.nx)
            s['x'], s['y'], s['u'] = s['x'][keep], s['y'][keep], s['u'][keep]
            if moving:
                c = self.c
                px = torch.arange(c['ppcx'], device=self.dev, dtype=torch.float64).add(0.5) / c['ppcx'] + self.nx - 1
                py = torch.arange(self.ny * c['ppcy'], device=self.dev, dtype=torch.float64).add(0.5) / c['ppcy']
                px = px[px > (c['edge'] - self.moved[0] * self.dx) / self.dx]
                gx, gy = (g.reshape(-1) for g in torch.meshgrid(px, py, indexing='ij'))
                s['x'], s['y'] = torch.cat([s['x'], gx]), torch.cat([s['y'], gy])
                s['u'] = torch.cat([s['u'], torch.zeros((gx.numel(), 3), dtype=torch.float64, device=self.dev)])
                self.moved[0] += 1

    def _current(self):
        J, n, c = self.J, self.nx, self.c
        if self.periodic:
            J[..., 1:3] += J[..., n + 1:n + 3]
            J[..., n] += J[..., 0]
            _wrap_x(J)
        elif c['bounds'] == 'walls':
            lo = [-J[0, :, 0] + J[0, :, 1], J[1, :, 0] + J[1, :, 2], J[2, :, 0] + J[2, :, 2]]
            hi = [J[0, :, n] - J[0, :, n + 1], J[1, :, n] + J[1, :, n + 2], J[2, :, n] + J[2, :, n + 2]]
            for k, inner, outer in ((0, 1, n + 1), (1, 2, n + 2), (2, 2, n + 2)):
                J[k, :, 0], J[k, :, inner] = lo[k], lo[k]
                J[k, :, n], J[k, :, outer] = hi[k], hi[k]

        def smooth(a, b):
            if c['filter_dir']:
                self.J = b * self.J + a * (torch.roll(self.J, 1, 1) + torch.roll(self.J, -1, 1))
            else:
                self.J[..., 1:n + 1] = b * self.J[..., 1:n + 1] + a * (self.J[..., 0:n] + self.J[..., 2:n + 2])
                if self.periodic:
                    _wrap_x(self.J)

        if c['filter'] != 'none':
            order = c['filter_order']
            for _ in range(order):
                smooth(0.25, 0.5)
            if c['filter'] == 'compensated':
                b = (4.0 + 2.0 * order) / order
                smooth(-1 / (b - 2), b / (b - 2))

    def _fields(self):
        E, B, J, n, dt = self.E, self.B, self.J, self.nx, self.dt
        dtx, dty = dt / self.dx, dt / self.dy

        def half_b():
            e, up = E[..., 0:n + 3], torch.roll(E, -1, 1)
            B[0, :, :n + 2] -= 0.5 * dty * (up[2] - e[2])[:, :n + 2]
            B[1, :, :n + 2] += 0.5 * dtx * (e[2, :, 1:] - e[2, :, :-1])
            B[2, :, :n + 2] += -0.5 * dtx * (e[1, :, 1:] - e[1, :, :-1]) + 0.5 * dty * (up[0] - e[0])[:, :n + 2]

        half_b()
        dn = torch.roll(B, 1, 1)
        E[0, :, 1:] += dty * (B[2] - dn[2])[:, 1:] - dt * J[0, :, 1:]
        E[1, :, 1:] += -dtx * (B[2, :, 1:] - B[2, :, :-1]) - dt * J[1, :, 1:]
        E[2, :, 1:] += dtx * (B[1, :, 1:] - B[1, :, :-1]) - dty * (B[0] - dn[0])[:, 1:] - dt * J[2, :, 1:]
        half_b()
        if self.periodic:
            _wrap_x(E), _wrap_x(B)
        elif self.c['bounds'] == 'walls':
            o = n + 1                                 # the upper wall's column
            e, b = E.clone(), B.clone()
            E[0, :, 0], E[1, :, 0], E[2, :, 0] = e[0, :, 1], -e[1, :, 2], -e[2, :, 2]
            E[1:, :, 1] = 0
            B[0, :, 0], B[1, :, 0], B[2, :, 0] = -b[0, :, 2], b[1, :, 1], b[2, :, 1]
            B[0, :, 1] = 0
            E[0, :, o], E[1, :, o], E[2, :, o] = e[0, :, o - 1], 0, 0
            E[0, :, o + 1], E[1, :, o + 1], E[2, :, o + 1] = e[0, :, o - 2], -e[1, :, o - 1], -e[2, :, o - 1]
            B[0, :, o], B[1, :, o], B[2, :, o] = 0, b[1, :, o - 1], b[2, :, o - 1]
            B[0, :, o + 1], B[1, :, o + 1], B[2, :, o + 1] = -b[0, :, o - 1], b[1, :, o - 2], b[2, :, o - 2]
        if self.c['bounds'] == 'window' and (self.iter + 1) * dt > self.dx * (self.moved[1] + 1):
            for f in (E, B):
                f[..., :-1] = f[..., 1:].clone()
                f[..., -1] = 0
            self.moved[1] += 1

    def step(self):
        self.J.zero_()
        for s in self.sp:
            self._advance_species(s)
        self._current()
        self._fields()
        self.iter += 1

    # diagnostics
    def charge(self, s):
        out = torch.zeros(self.ny * self.nx, dtype=torch.float64, device=self.dev)
        i, j = torch.floor(s['x']), torch.floor(s['y'])
        wx, wy = s['x'] - i, s['y'] - j
        i, j = i.long(), j.long()
        for a, fx in ((0, 1 - wx), (1, wx)):
            for b, fy in ((0, 1 - wy), (1, wy)):
                out.index_add_(0, ((j + b) % self.ny) * self.nx + (i + a) % self.nx, s['q'] * fx * fy)
        return out.reshape(self.ny, self.nx)

    def phase(self, s, axes):
        """Linear deposit of the particles' weight; the last bin of each axis stays empty."""
        size, norm, idx = 1, abs(s['q']) * self.dx * self.dy, []
        for v, (lo, hi), n in axes:
            p = (v - lo) * (n / (hi - lo)) - 0.5
            k = torch.trunc(p + 1) - 1
            idx.append([(k.long(), 1 - (p - k), n), (k.long() + 1, p - k, n)])
            norm *= n / (hi - lo)
            size *= n
        out = torch.zeros(size, dtype=torch.float64, device=self.dev)
        pairs = [[a] for a in idx[0]] if len(idx) == 1 else [[a, b] for a in idx[0] for b in idx[1]]
        for p in pairs:
            at, w, ok, stride = 0, norm, True, 1
            for k, f, n in p:
                ok = ok & (k >= 0) & (k < n - 1)
                at, w, stride = at + k * stride, w * f, stride * n
            out.index_add_(0, at[ok], w[ok])
        return out.reshape([n for _, _, n in reversed(axes)])

    def dump(self, species):
        out = {'E': _tiled(self.c, self.E), 'B': _tiled(self.c, self.B)}
        for sp in range(species):
            out['rho%d' % sp] = self.charge(self.sp[sp])
        return out

    def energies(self):
        # sums of squares over the interior; along x as many cells of a tile as it has along y (and as its block holds)
        c, f = self.c, []
        n = 1 + min(c['nxy'], c['nxx'] + 2)
        for g in (self.E, self.B):
            t = _tiled(c, g)[:, :(c['nxx'] + 3) * (c['nxy'] + 3)].reshape(-1, c['nxy'] + 3, c['nxx'] + 3, 3)
            f += [float(v) for v in (t[:, 1:c['nxy'] + 1, 1:n] ** 2).sum((0, 1, 2))]
        return f + [s['energy'] * s['q'] * s['m_q'] * self.dx * self.dy for s in self.sp]


def exact(case, seed):
    if not torch.cuda.is_available() and work(case)['flops'] > 2e10:
        return None
    got = []
    for k, c in enumerate(_members(case)):
        m, energies = _Exact(c, seed, k), []
        for _ in range(c['steps']):
            m.step()
            if c['kind'] == 'notebook':
                energies.append(m.energies())
        if c['kind'] == 'dump':
            box = (0.0, c['ntx'] * c['nxx'] * c['dx'])
            out = {w + f: getattr(m, w)[i, :, 1:m.nx + 1] for w in 'EBJ' for i, f in enumerate('xyz')}
            for sp, s in enumerate(m.sp):
                x, uz, n = s['x'] * m.dx, s['u'][:, 2], PHASE['bins']
                out['rho%d' % sp] = m.charge(s)
                out['uz%d' % sp] = m.phase(s, [(uz, PHASE['range'], n)])
                out['xuz%d' % sp] = m.phase(s, [(x, box, n), (uz, PHASE['range'], n // 2)])
            return out
        out = m.dump(1 if case['kind'] == 'batch' else c['species'])
        if energies:
            out['energies'] = np.array(energies)
        got.append(out)
    return got if case['kind'] == 'batch' else got[0]

"""The particle kernel's pair arithmetic against the oracle, over the ranges where its paths part: momenta and
fields from denormal to beyond the range of the pair operations (the general operations take over), time step
over mass that the pair quotient does not take, tiles of every remainder of a warp's 64 particles, and sums of the
tile current that wrap a 32-bit word thousands of times."""
import time

import numpy as np
import pytest

import zpic_b200 as zb
from em2d_oracle import OracleSim
from helpers import interior_mask, random_fields, rel_err, same_multisets

pytestmark = pytest.mark.gpu

# particles per tile: none, remainders of a pair, of a warp's 64 particles and of a CTA's blocks
COUNTS = [0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 127, 128, 129, 255, 256, 257, 511, 513, 640, 1000, 1027]


def _ppc(tiles):
    """Particles per cell with room for the counts above."""
    return (6, 6) if tiles[1][0] < 48 else (1, 1)


def _particles(geom, u_range, seed):
    (ntx, nty), (nx, ny) = geom[0], geom[1]
    rng = np.random.default_rng(seed)
    npt = np.array([COUNTS[k % len(COUNTS)] for k in range(ntx * nty)], np.int32)
    n = int(npt.sum())
    ix = np.stack([rng.integers(0, nx, n), rng.integers(0, ny, n)], 1).astype(np.int32)
    x = (rng.random((n, 2)) - 0.5).astype(np.float32)
    x[x >= 0.5] = 0.0
    u = np.exp(rng.uniform(*np.log(u_range), (n, 3))) * rng.choice([-1.0, 1.0], (n, 3))
    u[rng.random(n) < 0.05] = 0.0
    return npt, ix, x, u.astype(np.float32)


# square tiles of 8, 16 and 32 cells (their own instances, 32 in CTAs of 384 threads), generic ones in CTAs of 128
# and 256 threads (9x7 and 35x21 cells), tiles that fill an SM with CTAs of 384, 224, 192 and 128 threads
GEOMS = [((5, 5), (16, 16)), ((7, 3), (9, 7)), ((3, 7), (35, 21)), ((7, 3), (32, 32)), ((7, 6), (8, 8))]
IDS = ['16x16', '9x7', '35x21', '32x32', '8x8']
LARGE = [((5, 5), (48, 50)), ((7, 3), (64, 64)), ((7, 3), (61, 68)), ((7, 3), (65, 64))]
LARGE_IDS = ['48x50', '64x64', '61x68', '65x64']


@pytest.mark.parametrize('tiles', GEOMS + LARGE, ids=IDS + LARGE_IDS)
@pytest.mark.parametrize('m_q,u_range,b', [(-1.0, (1e-3, 1e2), 2.0), (1.0, (1e-42, 1e-3), 1e-20), (-1.0, (1e2, 1e18), 1e3),
                                           (-1.0, (1e-3, 1e2), 1e17), (1e21, (1e-2, 1e1), 1.0), (-1e-19, (1e-2, 1e1), 1e-3)])
def test_push_bit_exact(tiles, m_q, u_range, b):
    geom = tiles + ((0.1 * tiles[0][0] * tiles[1][0], 0.1 * tiles[0][1] * tiles[1][1]), 0.05)
    sims = []
    for cls in (OracleSim, zb.Simulation):
        s = cls(*geom)
        s.add_species(m_q, _ppc(tiles))
        s.set_grid('E', random_fields(s, 3, min(b, 10.0)))
        s.set_grid('B', random_fields(s, 4, b))
        s.set_particles(0, *_particles(geom, u_range, 7))
        s.species_push(0)
        sims.append(s.particles(0) + (s.species_energy(0),))
    o, g = sims
    assert np.array_equal(o[0], g[0])
    # no tolerance: every operation is correctly rounded in both
    assert np.array_equal(o[3], g[3], equal_nan=True)
    # the same non-negative terms, each one FP32 value, summed in FP64 in another order
    if np.isfinite(o[4]):
        assert abs(g[4] - o[4]) <= 2 * (int(o[0].sum()) + 8) * 2.0 ** -53 * abs(o[4])


@pytest.mark.parametrize('tiles', GEOMS + LARGE, ids=IDS + LARGE_IDS)
@pytest.mark.parametrize('jacc', [2, 0, 1])
@pytest.mark.parametrize('u_range', [(1e-3, 1e-1), (0.5, 50.0)])
def test_move_and_current(tiles, jacc, u_range):
    """Slow particles (few crossings) and fast ones (most particles cross, often two edges: the crossing queue
    fills in every iteration)."""
    geom = tiles + ((0.1 * tiles[0][0] * tiles[1][0], 0.1 * tiles[0][1] * tiles[1][1]), 0.07)
    sims = [cls(*geom) for cls in (OracleSim, zb.Simulation)]
    sims[1].set_option('jacc', jacc)
    for s in sims:
        s.add_species(-1.0, _ppc(tiles))
        s.set_particles(0, *_particles(geom, u_range, 11))
        s.current_zero()
        s.species_move(0)
    o, g = sims
    a, b = o.particles(0), g.particles(0)
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    m = interior_mask(o)
    # the parity tests' bar for sums in another order
    assert rel_err(g.grid('J')[:, m], o.grid('J')[:, m]) <= 1e-6


@pytest.mark.parametrize('tiles', GEOMS + LARGE, ids=IDS + LARGE_IDS)
@pytest.mark.parametrize('jacc', [2, 0, 1])
def test_whole_step(tiles, jacc):
    geom = tiles + ((0.1 * tiles[0][0] * tiles[1][0], 0.1 * tiles[0][1] * tiles[1][1]), 0.05)
    sims = [cls(*geom) for cls in (OracleSim, zb.Simulation)]
    sims[1].set_option('jacc', jacc)
    for s in sims:
        s.add_species(-1.0, _ppc(tiles))
        s.set_grid('E', random_fields(s, 3, 1.0))
        s.set_grid('B', random_fields(s, 4, 1.0))
        s.set_particles(0, *_particles(geom, (1e-3, 1e1), 13))
        s.advance(1)
    o, g = sims
    assert same_multisets(o.particles(0), g.particles(0))
    m = interior_mask(o)
    assert rel_err(g.grid('J')[:, m], o.grid('J')[:, m]) <= 1e-6


def test_other_tile_currents_are_not_far_behind():
    """32x32-cell tiles: the FP32 and FP64 tile currents' compare-and-swap loops cost half as much again as the
    fixed-point one (1.49 and 1.54 measured; 2.3 and 2.5 with a third of the warps)."""
    ms = []
    for jacc in (2, 0, 1):
        s = zb.Simulation((16, 16), (32, 32), (51.2, 51.2), 0.07)
        s.set_option('jacc', jacc)
        s.add_species(-1.0, (4, 4), udist=('thermal', (0.1, 0.1, 0.1), (0, 0, 0.3)))
        s.advance(10)
        s.synchronize()
        t = time.perf_counter()
        s.advance(100)
        s.synchronize()
        ms.append(time.perf_counter() - t)
        s.close()
    assert max(ms[1:]) <= 1.9 * ms[0]


@pytest.mark.parametrize('chunks', [1, 3])
def test_current_of_a_crowded_cell(chunks):
    """60,000 particles in one cell, all along +z near the speed of light: every node's sum wraps its word
    ten thousand times.  Expected: N q vz times the mean weight, in float64; the contributions are rounded to
    2^-24 of their value each, the sum once more to FP32."""
    n = 60000
    s = zb.Simulation((2, 2), (16, 16), (3.2, 3.2), 0.05)
    s.set_option('chunks', chunks)
    s.add_species(-1.0, (1, 1))
    rng = np.random.default_rng(5)
    x = (0.9 * (rng.random((n, 2)) - 0.5)).astype(np.float32)
    u = np.zeros((n, 3), np.float32)
    u[:, 2] = 20.0
    s.set_particles(0, np.array([n, 0, 0, 0], np.int32), np.full((n, 2), 7, np.int32), x, u)
    s.current_zero()
    s.species_move(0)
    j = s.grid('J')[0, :361].reshape(19, 19, 3)[..., 2]
    vz = 20.0 / np.sqrt(401.0)
    w = x.astype(np.float64)
    for dy in (0, 1):
        for dx in (0, 1):
            wx = 0.5 + w[:, 0] if dx else 0.5 - w[:, 0]
            wy = 0.5 + w[:, 1] if dy else 0.5 - w[:, 1]
            want = -vz * (wx * wy).sum()
            assert abs(j[8 + dy, 8 + dx] - want) <= 3 * 2.0 ** -24 * abs(want)
    j[8:10, 8:10] = 0
    assert not j.any()

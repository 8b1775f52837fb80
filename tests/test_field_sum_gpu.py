"""The field solve that sums the deposits of the tiles itself, and the current filter in one kernel (whole steps),
against the separate sum, filter passes and solve (the same step issued object by object): J, E and B, guard cells
included, bit for bit.  One species with one CTA per tile: its fixed-point deposits do not depend on the order of
the sums, so there is no rounding to allow."""
import numpy as np
import pytest

import zpic_b200 as zb

pytestmark = pytest.mark.gpu


# 16x16 tiles (their own instance), tiles at the limit of the sum in the solver (3 cells) and below it, oblong and
# odd ones, one tile per axis (its own neighbour), and open ends of the current
@pytest.mark.parametrize('ntiles,nx,current_bc', [
    ((4, 3), (16, 16), (1, 1, 1, 1)), ((1, 1), (16, 16), (1, 1, 1, 1)), ((1, 4), (16, 16), (1, 1, 1, 1)),
    ((5, 6), (3, 3), (1, 1, 1, 1)), ((6, 5), (2, 5), (1, 1, 1, 1)), ((5, 6), (4, 2), (1, 1, 1, 1)),
    ((3, 4), (24, 14), (1, 1, 1, 1)), ((2, 1), (33, 17), (1, 1, 1, 1)), ((4, 3), (16, 16), (0, 0, 1, 1)),
    ((4, 3), (16, 16), (1, 1, 0, 0)), ((3, 3), (5, 7), (0, 0, 0, 0)), ((3, 3), (16, 16), (2, 2, 1, 1))])
def test_step_equals_separate_objects(ntiles, nx, current_bc):
    def make():
        s = zb.Simulation(ntiles, nx, (0.1 * ntiles[0] * nx[0], 0.1 * ntiles[1] * nx[1]), 0.05)
        s.set_option('chunks', 1)
        s.current_set_bc(current_bc)
        s.add_species(-1.0, (3, 2), udist=('thermal', (0.3, 0.2, 0.1), (0.1, 0, 0.3)))
        return s

    a, b = make(), make()
    for _ in range(3):
        a.advance(1)
        b.current_zero()
        b.species_advance(0)
        b.current_advance()
        b.emf_advance()
        for w in 'JEB':
            assert np.array_equal(a.grid(w), b.grid(w)), w


# passes within the neighbours' interiors (their number at most the tile's cells - 2, and 8) and beyond; both
# axes, one tile per axis, open and reflecting ends along and across the filter
@pytest.mark.parametrize('ntiles,nx,bc,kind,direction,order', [
    ((4, 3), (16, 16), (1, 1, 1, 1), 'binomial', 0, 1), ((4, 3), (16, 16), (1, 1, 1, 1), 'compensated', 0, 2),
    ((4, 3), (16, 16), (1, 1, 1, 1), 'compensated', 1, 3), ((1, 1), (16, 16), (1, 1, 1, 1), 'compensated', 0, 7),
    ((4, 3), (16, 16), (1, 1, 1, 1), 'compensated', 0, 8), ((5, 4), (5, 7), (1, 1, 1, 1), 'compensated', 0, 2),
    ((5, 4), (5, 7), (1, 1, 1, 1), 'compensated', 0, 3), ((4, 5), (7, 4), (1, 1, 1, 1), 'binomial', 1, 2),
    ((4, 5), (7, 4), (1, 1, 1, 1), 'binomial', 1, 3), ((3, 4), (24, 14), (0, 0, 1, 1), 'compensated', 0, 4),
    ((3, 4), (24, 14), (0, 0, 1, 1), 'compensated', 1, 2), ((3, 4), (24, 14), (2, 2, 1, 1), 'binomial', 0, 2),
    ((3, 2), (33, 40), (1, 1, 2, 2), 'compensated', 1, 3), ((4, 4), (3, 3), (1, 1, 1, 1), 'binomial', 0, 1)])
def test_filtered_step_equals_separate_objects(ntiles, nx, bc, kind, direction, order):
    def make():
        s = zb.Simulation(ntiles, nx, (0.1 * ntiles[0] * nx[0], 0.1 * ntiles[1] * nx[1]), 0.05)
        s.set_option('chunks', 1)
        s.current_set_bc(bc)
        s.current_set_filter(kind, direction, order)
        s.add_species(-1.0, (3, 2), udist=('thermal', (0.3, 0.2, 0.1), (0.1, 0, 0.3)))
        return s

    a, b = make(), make()
    for _ in range(3):
        a.advance(1)
        b.current_zero()
        b.species_advance(0)
        b.current_advance()
        b.emf_advance()
        for w in 'JEB':
            assert np.array_equal(a.grid(w), b.grid(w)), w

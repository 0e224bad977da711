"""The walk over the cells, which serves every particle where there is no table and the particles whose rows
are too short where there is one: the same sums as the table's, bit for bit."""
import math

import numpy as np
import pytest

from test_gpu_pairs import C0, RHO0, cloud, pairSums, sameBits, sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('threads', [1, 2, 8])
@pytest.mark.parametrize('mixed', [False, True])
def test_the_walk_across_the_seam(mixed, threads):
    # other lanes than the four of the comparison beside: under four a row's entries are found one by one
    x, v, rho, m, fluid, h = cloud(3, 700, 701, ratio=1.7)
    lengths = np.where(np.random.default_rng(5).uniform(size=len(x)) < 0.5, h, 0.5 * h) if mixed else None
    sameBits(*(sums(pairSums(3, h, table, threads, period=1.0), x, v, rho, m, fluid, lengths)
               for table in (False, True)))


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('threads', [1, 2, 4, 8])
def test_runs_of_one_kind_and_of_both(dim, threads):
    # a layer of boundary particles under fluid, so that runs hold one kind, the other, or both, and of every
    # length against the lanes that test them together
    rng = np.random.default_rng(3)
    for n, ratio in ((150, 1.2), (700, 2.6)):
        x, v, rho, m, _, h = cloud(dim, n, n, ratio=ratio)
        fluid = (x[:, -1] > 0.4) ^ (rng.uniform(size=n) < 0.02)
        sameBits(*(sums(pairSums(dim, h, table, threads), x, v, rho, m, fluid) for table in (False, True)))


def stepped(s, state, h, dim):
    from pysurf_b200.state import ContainerBoundary
    g = np.zeros(dim)
    g[-1] = -9.81
    s.setPhysics(RHO0, C0, 0.1, 0.5, g, 0.5 if s.classicScheme else 0.0, 0.0)
    s.push(state)
    s.setBoundary(ContainerBoundary(np.zeros(dim), np.ones(dim), h), state)
    s.advance(0.0, 0, math.inf, 2, float(h if state.lengths is None else state.lengths.min()), 0.2, 1.0, 2)
    return s.pullState()


@pytest.mark.parametrize('scheme', ['paired', 'classic', 'mixed'])
@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('threads', [1, 4, 8])
def test_rows_too_short_for_their_counts(dim, threads, scheme):
    # A push of as many particles keeps the rows' length: sized for a sparse cloud, they are too short for the
    # packed part of the next, whose two ends of a row would meet, and long enough for the rest.
    from pysurf_b200.state import ParticleState
    n = 900
    x, v, rho, m, fluid, h = cloud(dim, n, 41 + dim, walls=0.4, ratio=1.3)
    lengths = np.where(np.random.default_rng(8).uniform(size=n) < 0.5, h, 0.75 * h) if scheme == 'mixed' else None
    packed = x.copy()
    near = x[:, 0] < 0.6
    packed[near] = 0.5 * x[near]
    options = dict(diffusion='none', corrected=False, limited=False) if scheme == 'classic' else {}
    runs, over = [], None
    for table in (False, True):
        s = pairSums(dim, h, table, threads, kernel='cubicSpline' if scheme == 'classic' else 'wendlandC2', **options)
        s.classicScheme = scheme == 'classic'
        state = ParticleState(x, 0.01 * v, np.zeros_like(x), rho, np.zeros(n), m, fluid, lengths)
        stepped(s, state, h, dim)
        state.positions = packed
        out = stepped(s, state, h, dim)
        p = C0 ** 2 * (rho - RHO0)
        g = np.zeros(dim)
        out['acceleration'] = s.pairAccelerations(v, rho, p, C0, 0.05, 0.5, g)
        out['rate'] = s.continuityRate(v, rho)
        out['shepard'] = s.shepardDensity(rho)
        if table:
            # the fluid's own neighbours, of which a row holds both kinds
            counts = np.diff(s.neighborList()[0])[fluid]
            over = counts > s.neighborTableCapacity()
            assert s.neighborTableCapacity() > 0
        runs.append(out)
    if lengths is None:
        assert over.any() and not over.all()
    sameBits(*runs)

"""The sweeps over pairs of neighbours, their table's rows and the packed frame, at the sizes where they
can go wrong.

Table and walk hand the same neighbours to the same arithmetic, so every sum is the same bits with the
table on and off: a row mis-parted, a neighbour lost at a row's odd end or one counted twice shows as a
difference of bits.  Clouds of a few particles give rows of 0, 1, 2, ... entries of either kind; larger
ones cross the sizes at which the table kernel takes other lanes or batches.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO0, C0 = 1000.0, 30.0


def cloud(dim, n, seed, walls=0.3, ratio=2.0):
    """n particles jittered about a lattice of unit spacing / n^(1/dim), a share of them boundary, in no order."""
    rng = np.random.default_rng(seed)
    side = max(1, math.ceil(n ** (1.0 / dim)))
    spacing = 1.0 / side
    grid = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing='ij'), -1).reshape(-1, dim)
    x = (rng.permutation(grid)[:n] + 0.5 + rng.uniform(-0.2, 0.2, (n, dim))) * spacing
    v = rng.uniform(-1.0, 1.0, (n, dim))
    rho = RHO0 * (1.0 + rng.uniform(0.0, 0.01, n))
    return x, v, rho, np.full(n, RHO0 * spacing ** dim), rng.uniform(size=n) >= walls, ratio * spacing


def pairSums(dim, h, table, threads=4, period=0.0, kernel='wendlandC2', precision='float64', **switches):
    from pysurf_b200.sphGpu import PairSums
    s = PairSums(dim, h, np.zeros(dim), np.ones(dim), period, kernelType=kernel, separationPrecision=precision)
    s.setSweepOptions(table, threads)
    s.setDiffusion(switches.get('diffusion', 'hydrostatic'), 0.1, C0, RHO0, 9.81)
    s.setContinuityCorrection(switches.get('corrected', True))
    s.setViscosityLimiter(switches.get('limited', True))
    return s


def sums(s, x, v, rho, m, fluid, lengths=None):
    """Every host-step sum the switches allow."""
    s.update(x, m, fluid, lengths)
    p = C0 ** 2 * (rho - RHO0)
    g = np.zeros(x.shape[1])
    g[-1] = -9.81
    out = {'acceleration': s.pairAccelerations(v, rho, p, C0, 0.05, 0.5, g), 'rate': s.continuityRate(v, rho),
           'wall': s.wallPressure(rho, p, g, RHO0, C0), 'shepard': s.shepardDensity(rho),
           'xsph': s.xsphVelocity(v, rho, 0.5)}
    if s.needsVelocityGradients:
        out['gradients'] = s.velocityGradients(v, rho)
    if s.needsCorrections:
        out['corrections'] = s.correctionMatrices(rho)
    return out


def sameBits(a, b):
    assert a.keys() == b.keys()
    for name in a:
        assert np.array_equal(a[name], b[name], equal_nan=True), name


@pytest.mark.parametrize('threads', [1, 2, 4, 8])
@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('n', [1, 2, 3, 5, 9, 17, 40, 333])
def test_a_rows_ends(n, dim, threads):
    # rows from empty up, of every remainder a lane can be left with, at long and short supports
    for ratio in (0.8, 1.3, 3.0):
        x, v, rho, m, fluid, h = cloud(dim, n, n + dim, ratio=ratio)
        sameBits(*(sums(pairSums(dim, h, table, threads), x, v, rho, m, fluid) for table in (False, True)))


@pytest.mark.parametrize('options', [dict(kernel='cubicSpline'), dict(precision='float32'), dict(diffusion='antuono'),
                                     dict(diffusion='none', corrected=False, limited=False), dict(period=1.0)])
@pytest.mark.parametrize('walls', [0.0, 0.5, 1.0])
def test_the_sweeps_forms(options, walls):
    # the walk at its own width of cells, and the forms the pipelined rows do not take
    dim = 3
    x, v, rho, m, fluid, h = cloud(dim, 1500, 7, walls=walls, ratio=1.6)
    sameBits(*(sums(pairSums(dim, h, table, **options), x, v, rho, m, fluid) for table in (False, True)))


@pytest.mark.parametrize('dim', [2, 3])
def test_mixed_lengths(dim):
    x, v, rho, m, fluid, h = cloud(dim, 1200, 11, ratio=2.0)
    lengths = np.where(np.random.default_rng(3).uniform(size=len(x)) < 0.5, h, 0.5 * h)
    sameBits(*(sums(pairSums(dim, h, table), x, v, rho, m, fluid, lengths) for table in (False, True)))


@pytest.mark.parametrize('precision', ['float64', 'float32'])
@pytest.mark.parametrize('mixed', [False, True])
@pytest.mark.parametrize('n', [700, 1201])
def test_the_table_across_the_seam(n, mixed, precision):
    # the table moves a batch's points across the seam (one length) or each distance (mixed): both searches
    # of a periodic axis, on one grid level and on two, find the walk's neighbours
    x, v, rho, m, fluid, h = cloud(3, n, n, ratio=1.7)
    lengths = np.where(np.random.default_rng(5).uniform(size=n) < 0.5, h, 0.5 * h) if mixed else None
    sameBits(*(sums(pairSums(3, h, table, period=1.0, precision=precision), x, v, rho, m, fluid, lengths)
               for table in (False, True)))


@pytest.mark.parametrize('dim, n', [(2, 24575), (2, 24576), (3, 65535), (3, 65536)])
def test_the_tables_lanes_and_batches(dim, n):
    # either side of the sizes at which the table kernel takes other lanes (2D) or batches (3D)
    x, v, rho, m, fluid, h = cloud(dim, n, 5, ratio=1.3)
    sameBits(*(sums(pairSums(dim, h, table), x, v, rho, m, fluid) for table in (False, True)))


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('threads', [1, 4, 8])
def test_the_classic_schemes_rows(dim, threads):
    # XSPH over the plain sums keeps one row of both kinds: table and walk alike, its steps and its sums,
    # and rows built before a switch turned the scheme over are not read as the other kind's
    from pysurf_b200.state import ContainerBoundary, ParticleState
    x, v, rho, m, fluid, h = cloud(dim, 600, 21, ratio=1.3)
    g = np.zeros(dim)
    g[-1] = -9.81
    runs = []
    for table in (False, True):
        s = pairSums(dim, h, table, threads, kernel='cubicSpline', diffusion='none', corrected=False, limited=False)
        s.setPhysics(RHO0, C0, 0.1, 0.0, g, 0.5, 0.0)
        out = sums(s, x, v, rho, m, fluid)
        s.setViscosityLimiter(True)
        out['limited'] = s.pairAccelerations(v, rho, C0 ** 2 * (rho - RHO0), C0, 0.05, 0.5, g)
        out['turned gradients'] = s.velocityGradients(v, rho)
        s.setViscosityLimiter(False)
        state = ParticleState(x.copy(), 0.01 * v, np.zeros_like(x), rho.copy(), np.zeros(len(x)), m, fluid)
        s.push(state)
        s.setBoundary(ContainerBoundary(np.zeros(dim), np.ones(dim), h), state)
        s.advance(0.0, 0, math.inf, 8, h, 0.2, 1.0, 3)
        s.pull(state)
        out.update(positions=state.positions, velocities=state.velocities, densities=state.densities)
        runs.append(out)
    sameBits(*runs)
    fresh = pairSums(dim, h, True, threads, kernel='cubicSpline', diffusion='none', corrected=False, limited=True)
    fresh.setPhysics(RHO0, C0, 0.1, 0.0, g, 0.5, 0.0)
    fresh.update(x, m, fluid)
    again = fresh.pairAccelerations(v, rho, C0 ** 2 * (rho - RHO0), C0, 0.05, 0.5, g)
    assert np.array_equal(again, runs[1]['limited'])


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('n, walls', [(1, 0.0), (1, 1.0), (31, 0.5), (1023, 0.4), (1024, 0.4), (1025, 0.4), (2048, 1.0),
                                      (2049, 0.0), (70001, 0.3)])
def test_a_frame_is_the_fluids_rows(n, walls, dim):
    # the device packs the fluid's rows in the caller's order: the pulled state's rows, rounded
    from pysurf_b200.state import ParticleState
    x, v, rho, m, fluid, h = cloud(dim, n, 2, walls=walls)
    s = pairSums(dim, h, True)
    s.push(ParticleState(x, v, np.zeros_like(x), rho, np.zeros(n), m, fluid))
    positions, speeds = s.frame()
    assert positions.dtype == np.float32 and speeds.dtype == np.float32
    assert np.array_equal(positions, x[fluid].astype(np.float32))
    assert np.array_equal(speeds, np.linalg.norm(v[fluid], axis=1).astype(np.float32))


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('epsilon, filterInterval', [(0.0, 0), (0.5, 0), (0.0, 1)])
def test_the_stages_of_a_step_follow_one_another(dim, epsilon, filterInterval):
    # the stamps are of one clock and in order, a stage without a kernel takes no time, and the stages of a
    # step fit in the time the host waits for it
    import time
    from pysurf_b200.state import ContainerBoundary, ParticleState
    x, v, rho, m, fluid, h = cloud(dim, 2000, 4, ratio=1.3)
    s = pairSums(dim, h, True)
    g = np.zeros(dim)
    g[-1] = -9.81
    s.setPhysics(RHO0, C0, 0.1, 0.0, g, epsilon, 0.0)
    state = ParticleState(x, 0.01 * v, np.zeros_like(x), rho, np.zeros(len(x)), m, fluid)
    s.push(state)
    s.setBoundary(ContainerBoundary(np.zeros(dim), np.ones(dim), h), state)
    s.beginSteps(0.0, 0, math.inf, 1 << 30, h, 0.2, 1.0, filterInterval)
    s.enqueueSteps(3)
    s.finishSteps()
    for _ in range(3):
        start = time.perf_counter()
        s.enqueueSteps(1)
        s.finishSteps()
        span = 1e3 * (time.perf_counter() - start)
        stages = dict(zip(s.stageNames(), s.stageTimes()))
        assert all(ms >= 0.0 for ms in stages.values()) and 0.0 < sum(stages.values()) <= span
        assert stages['cells'] > 0.0 and stages['momentum'] > 0.0 and stages['continuity'] > 0.0
        assert (stages['filter'] > 0.0) == (filterInterval > 0)

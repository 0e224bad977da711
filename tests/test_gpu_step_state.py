"""What a handle holds after the calls that set a step up without running it, and after those that drive
steps from the host: the neighbour table's order, the frame and the stage stamps stay those of work done."""
import math

import numpy as np
import pytest

from test_gpu_pairs import C0, RHO0, cloud, pairSums

pytestmark = pytest.mark.gpu


def steppedHandle(dim, table, limited, threads=4):
    """A handle with half its cloud boundary and XSPH on, at rest but for a small noise, pushed; its state."""
    from pysurf_b200.state import ContainerBoundary, ParticleState
    x, v, rho, m, fluid, h = cloud(dim, 500, 17 + dim, walls=0.5, ratio=1.6)
    s = pairSums(dim, h, table, threads, kernel='cubicSpline', diffusion='none', corrected=False, limited=limited)
    g = np.zeros(dim)
    g[-1] = -9.81
    s.setPhysics(RHO0, C0, 0.1, 0.0, g, 0.5, 0.0)
    state = ParticleState(x.copy(), 0.01 * v, np.zeros_like(x), rho.copy(), np.zeros(len(x)), m, fluid)
    s.push(state)
    s.setBoundary(ContainerBoundary(np.zeros(dim), np.ones(dim), h), state)
    return s, state, h


def hostSum(s, state, dim, name):
    g = np.zeros(dim)
    g[-1] = -9.81
    v, rho = state.velocities, state.densities
    p = C0 ** 2 * (rho - RHO0)
    return {'acceleration': lambda: s.pairAccelerations(v, rho, p, C0, 0.05, 0.5, g),
            'rate': lambda: s.continuityRate(v, rho), 'wall': lambda: s.wallPressure(rho, p, g, RHO0, C0),
            'shepard': lambda: s.shepardDensity(rho), 'xsph': lambda: s.xsphVelocity(v, rho, 0.5)}[name]()


def hostSums(s, state, dim):
    return {name: hostSum(s, state, dim, name) for name in ('acceleration', 'rate', 'wall', 'shepard', 'xsph')}


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('limited', [False, True])
@pytest.mark.parametrize('stepless', ['advance', 'beginSteps', 'none'])
def test_a_step_that_is_only_set_up_leaves_the_rows_as_they_are(dim, limited, stepless):
    # rows built in one scheme's order, the scheme turned over, a run that is already over: the host sums
    # after it read the rows in the order they were built in, whatever the captured step would build
    runs = []
    for table in (False, True):
        s, state, h = steppedHandle(dim, table, limited)
        s.residentRates(False)
        s.setViscosityLimiter(not limited)
        if stepless == 'advance':
            assert s.advance(1.0, 7, 1.0, 1 << 40, h, 0.2, 1.0)[:2] == (1.0, 7)
        elif stepless == 'beginSteps':
            s.beginSteps(1.0, 7, 1.0, 1 << 40, h, 0.2, 1.0)
        runs.append(hostSums(s, state, dim))
    for name in runs[0]:
        assert np.array_equal(runs[0][name], runs[1][name]), name


@pytest.mark.parametrize('dim', [2, 3])
def test_every_span_leaves_the_pressures_of_its_last_step(dim):
    # the frame a step leaves is in the master's order whether or not the span captured its graph: the
    # second span of a handle pulls the pressures that the host-driven step has too
    pulled = []
    for drive in ('device', 'host'):
        s, state, h = steppedHandle(dim, True, True)
        for _ in range(2):
            s.push(state)
            if drive == 'device':
                _, _, dt = s.advance(0.0, 0, math.inf, 1, h, 0.2, 1.0)
            else:
                s.residentRates(False)
                s.residentIntegrate(dt)
            out = state.copy()
            s.pull(out)
            pulled.append(out)
    for other in pulled[1:]:
        for name in ('positions', 'velocities', 'densities', 'pressures', 'accelerations'):
            assert np.array_equal(getattr(pulled[0], name), getattr(other, name)), name


@pytest.mark.parametrize('filterInterval', [0, 1])
@pytest.mark.parametrize('halves', [1, 2])
def test_stage_times_are_of_one_step(filterInterval, halves):
    # stage times are the device loop's last step's: the halves of a step that the host drives after it
    # change none of them
    s, state, h = steppedHandle(2, True, True)
    time, step, dt = s.advance(0.0, 0, math.inf, 2, h, 0.2, 1.0, filterInterval)
    before = s.stageTimes()
    assert all(0.0 <= ms < 1e3 for ms in before) and sum(before) > 0.0
    s.residentRates(filterInterval > 0)
    if halves == 2:
        s.residentIntegrate(dt)
    assert s.stageTimes() == before
    s.advance(time, step, math.inf, step + 1, h, 0.2, 1.0, filterInterval, dt)
    assert all(0.0 <= ms < 1e3 for ms in s.stageTimes())


@pytest.mark.parametrize('limited', [False, True])
@pytest.mark.parametrize('dim', [2, 3])
def test_host_sums_in_any_order_read_their_own_rows(dim, limited):
    # the classic scheme's own sums and the others read the table's rows in different orders: whichever is
    # asked for next, after a step too, each gives a table-free handle's bits
    asked = ['acceleration', 'wall', 'wall', 'rate', 'shepard', 'wall', 'xsph', 'acceleration', 'rates', 'wall', 'rate']
    runs = []
    for table in (False, True):
        s, state, h = steppedHandle(dim, table, limited)
        s.residentRates(False)
        out = []
        for name in asked:
            if name == 'rates':
                s.residentRates(True)
            else:
                out.append(hostSum(s, state, dim, name))
        runs.append(out)
    assert all(np.array_equal(a, b) for a, b in zip(*runs))

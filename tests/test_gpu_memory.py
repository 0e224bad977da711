"""What a handle holds on the device for each particle, and what shares it."""
import math

import numpy as np
import pytest

from test_gpu_pairs import C0, RHO0, cloud, pairSums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dim', [2, 3])
def test_a_particles_bytes(dim):
    # without the table: two masters, the frame, the sort's scratch and the staging took 623 bytes before the
    # sweeps' rows were laid out anew; a table capped by memory gets what these leave
    import torch
    from pysurf_b200.sphGpu import PairSums
    from pysurf_b200.state import ParticleState
    n = 1 << 21
    x = np.random.default_rng(1).uniform(size=(n, dim))
    state = ParticleState(x, np.zeros_like(x), np.zeros_like(x), np.full(n, RHO0), np.zeros(n), np.ones(n),
                          np.ones(n, dtype=bool))
    torch.zeros(1, device='cuda')
    s = PairSums(dim, 0.01, np.zeros(dim), np.ones(dim))
    s.setSweepOptions(False, 4)
    before = torch.cuda.mem_get_info()[0]
    s.push(state)
    assert before - torch.cuda.mem_get_info()[0] <= 623 * n


@pytest.mark.parametrize('dim', [2, 3])
def test_gradients_between_shifting_steps(dim):
    # the whole velocity gradients lie where the shifting's fields do: a call between two spans of shifting
    # steps, and shifts between two such calls, change neither's bits
    from pysurf_b200.state import ContainerBoundary, ParticleState
    x, v, rho, m, fluid, h = cloud(dim, 600, 51, ratio=2.0)
    g = np.zeros(dim)
    g[-1] = -9.81
    ends, gradients = [], []
    for asks in (False, True):
        s = pairSums(dim, h, True)
        s.setShifting(True, 0.1, 0.5 * h, C0, False)
        s.setPhysics(RHO0, C0, 0.1, 0.0, g, 0.0, 0.0)
        state = ParticleState(x.copy(), 0.01 * v, np.zeros_like(x), rho.copy(), np.zeros(len(x)), m, fluid)
        s.push(state)
        s.setBoundary(ContainerBoundary(np.zeros(dim), np.ones(dim), h), state)
        time, step, dt = s.advance(0.0, 0, math.inf, 3, h, 0.2, 1.0)
        if asks:
            gradients.append(s.velocityGradients(v, rho))
            s.shiftingDisplacement(rho, 1e-4, v)
            gradients.append(s.velocityGradients(v, rho))
        s.advance(time, step, math.inf, 6, h, 0.2, 1.0, 0, dt)
        ends.append(s.pullState())
    for name in ('positions', 'velocities', 'densities'):
        assert np.array_equal(ends[0][name], ends[1][name]), name
    assert np.abs(gradients[0]).max() > 0.0 and np.array_equal(*gradients)

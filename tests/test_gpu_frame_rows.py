"""The packed frame's two entries: rows are handed out only while they are the ones that were packed, and
they are the fluid's rows of the frame that holds every particle."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_pairs import C0, RHO0, cloud, pairSums

pytestmark = pytest.mark.gpu

INVALID, STATE = -1, -6


def pushed(dim, n=300):
    from pysurf_b200.state import ParticleState
    x, v, rho, m, fluid, h = cloud(dim, n, 9)
    s = pairSums(dim, h, True)
    state = ParticleState(x, v, np.zeros_like(x), rho, np.zeros(n), m, fluid)
    s.push(state)
    return s, state


def pack(s):
    count = C.c_int64(-1)
    assert s._lib.sph_fluid_frame(s._handle, C.byref(count)) == 0
    return count.value


def rows(s, count, dim):
    from pysurf_b200 import _lib
    positions, speeds = np.zeros((max(count, 1), dim), np.float32), np.zeros(max(count, 1), np.float32)
    status = s._lib.sph_fluid_frame_rows(s._handle, positions.ctypes.data_as(_lib._pf), speeds.ctypes.data_as(_lib._pf),
                                         count)
    return status, positions[:count], speeds[:count]


@pytest.mark.parametrize('dim', [2, 3])
def test_rows_are_refused_once_another_call_has_used_their_memory(dim):
    s, state = pushed(dim)
    fluid = int(state.isFluid.sum())
    assert rows(s, fluid, dim)[0] == STATE                  # nothing was packed
    g = np.zeros(dim)
    between = {'sum': lambda: s.shepardDensity(state.densities), 'pull': lambda: s.pullState(),
               'push': lambda: s.push(state), 'energy': lambda: s.fluidEnergy(),
               'list': lambda: s.neighborList(),
               'acceleration': lambda: s.pairAccelerations(state.velocities, state.densities, state.pressures, C0, 0.1,
                                                           0.5, g)}
    s.setPhysics(RHO0, C0, 0.1, 0.0, g, 0.0, 0.0)
    for name, call in between.items():
        assert pack(s) == fluid
        call()
        assert rows(s, fluid, dim)[0] == STATE, name
    assert pack(s) == fluid
    assert rows(s, fluid + 1, dim)[0] == INVALID and rows(s, -1, dim)[0] == INVALID
    for count in (fluid, fluid, 3, 0):                      # again, and the first few
        status, positions, speeds = rows(s, count, dim)
        assert status == 0
        assert np.array_equal(positions, state.positions[state.isFluid][:count].astype(np.float32))


@pytest.mark.parametrize('dim', [2, 3])
def test_packed_rows_are_the_whole_frames_fluid(dim):
    # sph_frame hands out every particle's row and its kind; a C program may use either
    from pysurf_b200 import _lib
    s, state = pushed(dim, 2100)
    n = state.nParticles
    positions, speeds, kind = np.empty((n, dim), np.float32), np.empty(n, np.float32), np.empty(n, np.uint8)
    assert s._lib.sph_frame(s._handle, positions.ctypes.data_as(_lib._pf), speeds.ctypes.data_as(_lib._pf),
                            kind.ctypes.data_as(_lib._pu8)) == 0
    assert np.array_equal(kind.astype(bool), state.isFluid)
    packedPositions, packedSpeeds = s.frame()
    assert np.array_equal(packedPositions, positions[kind == 1])
    assert np.array_equal(packedSpeeds, speeds[kind == 1])

"""The workloads whose speed is followed: spans of a run, as a user's program steps them.

A pass hands a particle state to the device, steps it and takes the result back: the next frame of
the run (the float32 positions and speeds that a run's frames hold) and every density.  Most passes
run the device loop (`PairSums.advance`, the time step taken on the device); one runs the loop that
a host solver drives (`residentRates`, the solver's own time step, `residentIntegrate`) from host
arrays.  The states are the repository's cases with the disorder of a running flow: the fluid's
lattice jittered, and a velocity noise on the wave.

`exact` is the same scheme in float64 in plain torch, over explicit pair lists.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pysurf_b200 import cases

JITTER = 0.08       # of the spacing: the disorder of a running flow
NOISE = 0.004       # of the sound speed / 10 (about the flow's own speed)


def listed() -> list:
    return [
        # a tank of a few hundred particles under the default scheme (cubic spline, XSPH, Shepard
        # filter): the tests' and tutorials' size, all launches and latency
        dict(name='sloshing-600', flow='sloshing', spacing=0.005, tilt=10.0, steps=31, loop='device', options=''),
        # the 5,000-particle dam break, driven step by step by a host solver from host arrays
        dict(name='dam-5k-host-loop', flow='dam', spacing=0.02, steps=12, loop='host', options=''),
        # a larger dam break on the device loop, cubic spline and renormalized diffusion
        dict(name='dam-31k-antuono', flow='dam', spacing=0.008, steps=16, loop='device', options='cubic,antuono'),
        # the small end of a beach sweep: about 8,000 particles
        dict(name='beach-16', flow='beach', ppd=16, height=0.45, slope=1 / 15, steps=24, loop='device', options=''),
        # an odd size in the middle of the sweep, with the turbulence closure
        dict(name='beach-37-closure', flow='beach', ppd=37, height=0.31, slope=1 / 23, steps=16, loop='device',
             options='closure'),
        # the 2D benchmark: 122,000 particles
        dict(name='beach-64', flow='beach', ppd=64, height=0.45, slope=1 / 15, steps=16, loop='device', options=''),
        # a beach well resolved for 2D, about 400,000 particles
        dict(name='beach-120', flow='beach', ppd=120, height=0.45, slope=1 / 15, steps=8, loop='device', options=''),
        # a small 3D run: the beach across a periodic axis
        dict(name='channel-8', flow='channel', ppd=8, width=1.75, height=0.6, slope=1 / 15, steps=5, loop='device',
             options=''),
        # the 3D ridge at sizes a server's requests have
        dict(name='ridge-10', flow='ridge', ppd=10, height=0.5, angle=25.0, steps=3, loop='device', options=''),
        # the 3D benchmark's two grid levels: the crest zone split into daughters of half the length
        dict(name='ridge-11-refined', flow='ridge', ppd=11, height=0.5, angle=25.0, steps=2, loop='device',
             options='refined'),
        # the largest: 4.4 million particles
        dict(name='ridge-20', flow='ridge', ppd=20, height=0.5, angle=25.0, steps=3, loop='device', options=''),
    ]


def _log(rng, low: float, high: float) -> float:
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng) -> dict:
    flow = rng.choice(['sloshing', 'dam', 'beach', 'beach', 'channel', 'ridge', 'ridge', 'refined'])
    if flow == 'sloshing':
        return dict(flow=flow, spacing=_log(rng, 0.0018, 0.006), tilt=rng.uniform(4.0, 14.0),
                    steps=rng.randint(16, 31), loop='device', options='')
    if flow == 'dam':
        return dict(flow=flow, spacing=_log(rng, 0.006, 0.03), steps=rng.randint(6, 20),
                    loop=rng.choice(['device', 'device', 'host']),
                    options=rng.choice(['', 'cubic', 'antuono', 'cubic,antuono']))
    if flow == 'beach':
        return dict(flow=flow, ppd=int(_log(rng, 14, 121)), height=rng.uniform(0.2, 0.6),
                    slope=1.0 / rng.uniform(8.0, 35.0), steps=rng.randint(4, 8), loop='device',
                    options=rng.choice(['', '', 'closure']))
    if flow == 'channel':
        return dict(flow=flow, ppd=rng.randint(6, 10), width=rng.uniform(2.2, 3.0), height=rng.uniform(0.3, 0.6),
                    slope=1.0 / rng.uniform(10.0, 20.0), steps=rng.randint(2, 5), loop='device', options='')
    refined = flow == 'refined'
    return dict(flow='ridge', ppd=int(_log(rng, 6, 10) if refined else _log(rng, 6, 19)),
                height=rng.uniform(0.35, 0.55), angle=rng.uniform(0.0, 40.0), steps=rng.randint(1, 3), loop='device',
                options='refined' if refined else '')


# -- inputs -- #

@functools.lru_cache(maxsize=4)
def _flow(key: tuple):
    """The repository's case of these sizes (its lattice, walls and scheme)."""
    spec = dict(key)
    flow, options = spec['flow'], spec['options'].split(',')
    if flow == 'sloshing':
        return cases.sloshingTank(tilt=spec['tilt'], spacing=spec['spacing'])
    if flow == 'dam':
        return cases.damBreak(spec['spacing'], kernelType='cubicSpline' if 'cubic' in options else 'wendlandC2',
                              diffusion='antuono' if 'antuono' in options else 'hydrostatic')
    if flow == 'beach':
        case = cases.solitaryBeach(spec['ppd'], height=spec['height'], slope=spec['slope'], length=40.0)
        case.turbulenceClosure = 'deltaLes' if 'closure' in options else 'none'
        return case
    if flow == 'channel':
        return cases.extrudedBeach(spec['ppd'], width=spec['width'], height=spec['height'], slope=spec['slope'])
    return cases.ridgeWave3D(spec['ppd'], height=spec['height'], angle=spec['angle'])


def _inputs(case: dict, seed: int):
    """The flow, and its state from the seed as float64 tensors on the GPU."""
    flow = _flow(tuple(sorted((k, v) for k, v in case.items() if k not in ('name', 'steps', 'loop'))))
    state, device = flow.state, torch.device('cuda', torch.cuda.current_device())
    fluid = torch.as_tensor(state.isFluid, device=device)
    to = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)
    positions, velocities = to(state.positions), to(state.velocities)
    generator = torch.Generator(device=device).manual_seed(int(seed))
    draw01 = lambda: torch.rand(positions.shape, generator=generator, device=device, dtype=torch.float64)
    positions += fluid[:, None] * (JITTER * flow.spacing) * (2.0 * draw01() - 1.0)
    velocities += fluid[:, None] * (NOISE * 0.1 * flow.soundSpeed) * (2.0 * draw01() - 1.0)
    return flow, dict(positions=positions.contiguous(), velocities=velocities.contiguous(),
                      densities=to(state.densities), masses=to(state.masses), isFluid=fluid.to(torch.uint8),
                      lengths=None)


def prepare(case: dict, seed: int) -> dict:
    """The solver's handle, set up for the flow, and the state to step; with 'refined' the crest zone
    is split first."""
    flow, state = _inputs(case, seed)
    sums = cases.pairSumsFor(flow, device=state['positions'].device.index)
    torch.cuda.synchronize()
    if 'refined' in case['options']:
        sums.pushDevice(**state)
        cases.refineCrestZone(sums, flow)
        n, kept = sums.count, state['positions']
        empty = lambda *shape, dtype=torch.float64: torch.empty(shape, dtype=dtype, device=kept.device)
        state = dict(positions=empty(n, 3), velocities=empty(n, 3), densities=empty(n), masses=empty(n),
                     isFluid=empty(n, dtype=torch.uint8), lengths=empty(n))
        sums.pullDevice(**state)
    host = None
    if case['loop'] == 'host':
        host = flow.state.copy()
        for name in ('positions', 'velocities', 'densities', 'masses'):
            setattr(host, name, state[name].cpu().numpy())
    sums.setBoundary(flow.boundary, flow.state)
    shortest = flow.smoothingLength if state['lengths'] is None else float(state['lengths'].min())
    densities = torch.empty_like(state['densities'])
    torch.cuda.synchronize()
    return dict(case=case, flow=flow, sums=sums, state=state, host=host, shortest=shortest, densities=densities)


def run(prepared: dict) -> dict:
    """One span: the state to the device, `steps` steps, the frame and the densities."""
    sums, flow, steps = prepared['sums'], prepared['flow'], prepared['case']['steps']
    shortest = prepared['shortest']
    if prepared['host'] is None:
        sums.pushDevice(**prepared['state'])
        time, _, _ = sums.advance(0.0, 0, math.inf, steps, shortest, flow.cflNumber, flow.maxTimeStep,
                                  flow.densityFilterInterval)
    else:
        sums.push(prepared['host'])
        time = 0.0
        for _ in range(steps):
            speed, acceleration = sums.residentRates(False)
            step = flow.cflNumber * shortest / (flow.soundSpeed + speed)
            if acceleration > 1e-12:
                step = min(step, flow.cflNumber * math.sqrt(shortest / acceleration))
            step = min(step, flow.maxTimeStep)
            sums.residentIntegrate(step)
            time += step
    positions, speeds = sums.frame()
    sums.pullDevice(densities=prepared['densities'])
    return dict(time=time, positions=positions, speeds=speeds, densities=prepared['densities'])


# -- work -- #

def work(case: dict) -> dict:
    """Per step and fluid particle: read x, v, rho, m and the kind, write x, v and rho (53 bytes in 2D,
    69 in 3D, the positions as an offset in a cell), and 150 flop a directed pair over the gradients,
    momentum and continuity sums."""
    flow = _flow(tuple(sorted((k, v) for k, v in case.items() if k not in ('name', 'steps', 'loop'))))
    dim, reach = flow.dimensions, 2.0 * flow.smoothingLength / flow.spacing
    fluid = flow.fluidCount
    if 'refined' in case['options']:
        # the share of the tank's water in the crest zone, each particle eight daughters
        x, depth = flow.state.positions[:fluid, 0], flow.info['depth']
        height = flow.info['H/d'] * depth
        crest = cases.solitaryWaveProfile(x, height, depth, flow.info['crestX']) > 0.3 * height
        fluid += 7 * int(np.count_nonzero(crest))
    pairs = (math.pi * reach ** 2 if dim == 2 else 4.0 / 3.0 * math.pi * reach ** 3) - 1.0
    return dict(bytes=float((53 if dim == 2 else 69) * fluid * case['steps']),
                flops=float(150.0 * pairs * fluid * case['steps']))


# -- the scheme in float64 -- #

def _pairLists(x, h, width: float, period: float, most: int = 20_000_000):
    """Every ordered pair closer than h_i + h_j, as chunks (i, j) with i ascending, from cells `width` wide."""
    n, dim = x.shape
    low = x.min(0).values
    cell = torch.floor((x - low) / width).long()
    count = cell.max(0).values + 1
    if period > 0.0:
        # the y axis in whole cells around the period
        count[1] = max(int(period / width), 1)
        cell[:, 1] = torch.remainder(torch.floor(x[:, 1] * (float(count[1]) / period)).long(), count[1])
    shape = [int(c) for c in count]
    number = lambda c: (c[2] * shape[1] + c[1]) * shape[0] + c[0] if dim == 3 else c[1] * shape[0] + c[0]
    key = number([cell[:, a] for a in range(dim)])
    order = torch.argsort(key)
    start = torch.searchsorted(key[order], torch.arange(math.prod(shape) + 1, device=x.device))
    runs = []
    # a period of fewer than three cells: every cell across it, each once
    across = range(shape[1]) if period > 0.0 and shape[1] < 3 else (-1, 0, 1)
    for dz in ((-1, 0, 1) if dim == 3 else (0,)):
        for dy in across:
            c = [cell[:, a] for a in range(dim)]
            inside = torch.ones(n, dtype=torch.bool, device=x.device)
            for axis, step in ((1, dy), (2, dz))[:dim - 1]:
                moved = c[axis] + step
                if axis == 1 and period > 0.0:
                    moved = torch.remainder(moved, shape[1])
                else:
                    inside &= (moved >= 0) & (moved < shape[axis])
                c[axis] = moved.clamp(0, shape[axis] - 1)
            first = number([(c[0] - 1).clamp(min=0)] + c[1:])
            last = number([(c[0] + 1).clamp(max=shape[0] - 1)] + c[1:])
            runs.append((start[first], torch.where(inside, start[last + 1] - start[first], 0)))
    begin, length = (torch.stack(v, 1) for v in zip(*runs))
    total = length.sum(1).cumsum(0)
    chunks, done = [], 0
    while done < n:
        before = int(total[done - 1]) if done else 0
        stop = max(int(torch.searchsorted(total, before + most, right=True)), done + 1)
        b, l = begin[done:stop].reshape(-1), length[done:stop].reshape(-1)
        owner = torch.repeat_interleave(l)
        place = torch.arange(len(owner), device=x.device) - (l.cumsum(0) - l)[owner]
        i, j = done + owner // begin.shape[1], order[b[owner] + place]
        d = _separation(x, i, j, period)
        near = ((d * d).sum(1) < (h[i] + h[j]) ** 2) & (i != j)
        chunks.append((i[near].int(), j[near].int()))
        done = stop
    return chunks


def _separation(x, i, j, period: float):
    d = x[i] - x[j]
    if period > 0.0:
        d[:, 1] -= period * torch.round(d[:, 1] / period)
    return d


class _Scheme:
    """The step in float64: every sum over the pair lists, every constant from the flow's case."""

    def __init__(self, flow, state):
        self.flow, self.dim = flow, flow.dimensions
        self.x, self.v = state['positions'].clone(), state['velocities'].clone()
        self.rho, self.m = state['densities'].clone(), state['masses']
        self.fluid = state['isFluid'].bool()
        n = len(self.rho)
        self.h = torch.full_like(self.rho, flow.smoothingLength) if state['lengths'] is None else state['lengths']
        self.g = torch.as_tensor(flow.gravity, dtype=torch.float64, device=self.x.device)
        self.stiffness = flow.referenceDensity * flow.soundSpeed ** 2 / 7.0
        self.time, self.step, self.n = 0.0, 0, n
        if flow.kernelType == 'wendlandC2':
            self.sigma = 7.0 / (4.0 * math.pi) if self.dim == 2 else 21.0 / (16.0 * math.pi)
        else:
            self.sigma = 10.0 / (7.0 * math.pi) if self.dim == 2 else 1.0 / math.pi

    # the kernel and (dW/dr) / r
    def kernel(self, r, h):
        q, s = r / h, self.sigma / h ** self.dim
        if self.flow.kernelType == 'wendlandC2':
            return s * (1.0 - 0.5 * q) ** 4 * (2.0 * q + 1.0)
        return s * torch.where(q < 1.0, 1.0 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2.0 - q) ** 3)

    def slope(self, r, h):
        q, s = r / h, self.sigma / h ** (self.dim + 2)
        if self.flow.kernelType == 'wendlandC2':
            return -5.0 * s * (1.0 - 0.5 * q) ** 3
        return s * torch.where(q < 1.0, 2.25 * q - 3.0, -0.75 * (2.0 - q) ** 2 / q)

    def tait(self, rho):
        p = self.stiffness * ((rho / self.flow.referenceDensity) ** 7 - 1.0)
        return p if self.flow.negativePressure else p.clamp(min=0.0)

    def gathered(self, terms, columns):
        """sum over each i's pairs of terms(i, j, d, r, h), (n, columns)."""
        out = torch.zeros(self.n, columns, dtype=torch.float64, device=self.x.device)
        for i, j in self.pairs:
            i, j = i.long(), j.long()
            d = _separation(self.x0, i, j, self.flow.period)
            r = d.norm(dim=1)
            out.index_add_(0, i, terms(i, j, d, r, 0.5 * (self.h[i] + self.h[j])))
        return out

    def rows(self, i):
        return self.fluid[i].double()[:, None]

    def wall(self):
        def terms(i, j, d, r, h):
            w = self.kernel(r, h) * (~self.fluid[i] & self.fluid[j])
            return torch.stack([w, w * (self.p[j] + self.rho[j] * (d @ self.g))], 1)
        weight, total = self.gathered(terms, 2).unbind(1)
        p = torch.where(weight > 0.0, total / weight.clamp(min=1e-300), 0.0).clamp(min=0.0)
        rho = self.flow.referenceDensity * (1.0 + p / self.stiffness) ** (1.0 / 7.0)
        self.p, self.rho = torch.where(self.fluid, self.p, p), torch.where(self.fluid, self.rho, rho)

    def gradients(self):
        D, volume, rho = self.dim, self.m / self.rho, self.rho
        def terms(i, j, d, r, h):
            w = (volume[j] * self.slope(r, h))[:, None]
            outer = -w * (d[:, :, None] * d[:, None, :]).reshape(-1, D * D)
            both = self.fluid[j].double()[:, None]
            jump = w * ((self.v[j] - self.v[i])[:, :, None] * d[:, None, :]).reshape(-1, D * D)
            return torch.cat([both * jump, both * outer, outer, w * (rho[j] - rho[i])[:, None] * d], 1) * self.rows(i)
        sums = self.gathered(terms, 3 * D * D + D)
        S, M, A = (sums[:, k * D * D:(k + 1) * D * D].reshape(-1, D, D) for k in range(3))
        eye, floor = torch.eye(D, dtype=torch.float64, device=self.x.device), 0.25 ** D
        def inverse(matrix, other):
            good = (torch.linalg.det(matrix) >= floor)[:, None, None]
            return torch.where(good, torch.linalg.inv(torch.where(good, matrix, eye)), other)
        self.G = S @ inverse(M, torch.zeros_like(eye))
        self.L = inverse(A, eye)
        self.gradRho = (self.L @ sums[:, 3 * D * D:, None])[:, :, 0]
        f = self.flow
        if f.turbulenceClosure == 'deltaLes':
            strain = 0.5 * (self.G + self.G.transpose(1, 2))
            scale = self.h * (2.0 * (strain ** 2).sum((1, 2))).sqrt() / f.soundSpeed * self.fluid
            self.eddyAlpha = (2.0 * (D + 2) * 0.24 ** 2 * scale).clamp(max=0.2)
            self.eddyDelta = (9.0 * scale).clamp(max=0.2)

    @staticmethod
    def product(matrix, d):
        return (matrix * d[:, None, :]).sum(2)

    @staticmethod
    def harmonic(a, b):
        return torch.where(a + b > 0.0, 2.0 * a * b / (a + b).clamp(min=1e-300), 0.0)

    def momentum(self):
        f, ratio, dim = self.flow, self.p / self.rho ** 2, self.dim
        def terms(i, j, d, r, h):
            approach = plain = ((self.v[i] - self.v[j]) * d).sum(1)
            if f.viscosityLimiter:
                si, sj = ((d * self.product(self.G[k], d)).sum(1) for k in (i, j))
                total = torch.where(si + sj != 0.0, si + sj, 1.0)
                phi = torch.where(si * sj > 0.0, (4.0 * si * sj / total ** 2).clamp(max=1.0), 0.0)
                q = r / h
                phi = torch.where(q < 0.3, phi * torch.exp(-((q - 0.3) / 0.2) ** 2), phi)
                approach = torch.where(self.fluid[j] & (plain < 0.0), plain - 0.5 * phi * (si + sj), plain)
            mu = h * approach / (r * r + 0.01 * h * h)
            wall = torch.where(self.fluid[j], 1.0, f.boundaryViscosityFactor)
            Pi = torch.where(approach < 0.0, -f.alpha * f.soundSpeed * mu / (0.5 * (self.rho[i] + self.rho[j])) * wall, 0.0)
            if f.turbulenceClosure == 'deltaLes':
                water = 2.0 * (dim + 2) * f.kinematicViscosity / (f.soundSpeed * h)
                eddy = water + self.harmonic(self.eddyAlpha[i], self.eddyAlpha[j])
                Pi = Pi - self.fluid[j] * eddy * f.soundSpeed * h * f.referenceDensity * plain / (
                    r * r * self.rho[i] * self.rho[j])
            return (-(ratio[i] + ratio[j] + Pi) * self.m[j] * self.slope(r, h))[:, None] * d * self.rows(i)
        return (self.gathered(terms, dim) + self.g) * self.rows(slice(None))

    def continuity(self):
        f, reference = self.flow, self.flow.referenceDensity
        g = abs(float(f.gravity[-1]))
        def terms(i, j, d, r, h):
            slope, both = self.slope(r, h), self.fluid[i] & self.fluid[j]
            lever = d
            if f.continuityCorrection:
                lever = torch.where(self.fluid[i][:, None], self.product(self.L[i], d), d)
            rate = self.m[j] * ((self.v[i] - self.v[j]) * lever).sum(1) * slope * (self.fluid[i] | self.fluid[j])
            if f.densityDiffusion != 'none':
                jump = self.rho[j] - self.rho[i]
                if f.densityDiffusion == 'hydrostatic':
                    mean = 0.5 * (self.rho[i] + self.rho[j]) / reference
                    jump = jump - reference * g / f.soundSpeed ** 2 * d[:, -1] / mean ** 5
                if f.densityDiffusion == 'antuono':
                    jump = jump + 0.5 * ((self.gradRho[i] + self.gradRho[j]) * d).sum(1)
                delta = f.diffusionDelta
                if f.turbulenceClosure == 'deltaLes':
                    delta = self.harmonic(self.eddyDelta[i], self.eddyDelta[j])
                rate = rate - both * 2.0 * delta * f.soundSpeed * h * self.m[j] / self.rho[j] * jump * slope * (
                    r * r / (r * r + 0.01 * h * h))
            return rate[:, None]
        return self.gathered(terms, 1)[:, 0]

    def transport(self):
        """XSPH: the velocity the fluid drifts with, from the advanced densities."""
        def terms(i, j, d, r, h):
            weight = self.m[j] * self.kernel(r, h) / (0.5 * (self.rho[i] + self.rho[j])) * (self.fluid[i] & self.fluid[j])
            return weight[:, None] * (self.v[j] - self.v[i])
        return self.v + self.flow.xsphEpsilon * self.gathered(terms, self.dim)

    def filter(self):
        """The Shepard density of the fluid, the particle itself included."""
        volume = self.m / self.rho
        def terms(i, j, d, r, h):
            w = self.kernel(r, h)
            return torch.stack([self.m[j] * w, volume[j] * w], 1)
        own = self.kernel(torch.zeros_like(self.h), self.h)
        sums = self.gathered(terms, 2) + torch.stack([self.m * own, volume * own], 1)
        self.rho = torch.where(self.fluid, sums[:, 0] / sums[:, 1], self.rho)

    def enforce(self):
        """The boundary's hold on the fluid: positions put back, the velocity into it taken off."""
        b, x, v, vert = self.flow.boundary, self.x, self.v, self.dim - 1
        def hold(axis, low, high):
            for beyond, edge, sign in ((x[:, axis] < low, low, 1.0), (x[:, axis] > high, high, -1.0)):
                beyond = beyond & self.fluid
                v[:, axis] = torch.where(beyond, sign * (sign * v[:, axis]).clamp(min=0.0), v[:, axis])
                x[:, axis] = torch.where(beyond, torch.full_like(x[:, axis], edge), x[:, axis])
        def rest(bed, normal):
            below = (x[:, vert] < bed + clearance) & self.fluid
            x[:, vert] = torch.where(below, bed + clearance, x[:, vert])
            inward = (v * normal).sum(1)
            v.copy_(torch.where((below & (inward < 0.0))[:, None], v - inward[:, None] * normal, v))
        if hasattr(b, 'containerMin'):
            for a in range(self.dim):
                hold(a, float(b.containerMin[a]), math.inf if b.openTop and a == vert else float(b.containerMax[a]))
            return
        clearance = 0.25 * b.spacing
        to = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=x.device)
        if hasattr(b, 'bathymetry'):
            bx, bz = to(b.bathymetry.x), to(b.bathymetry.z)
            k = (torch.searchsorted(bx, x[:, 0].contiguous(), right=True) - 1).clamp(0, len(bx) - 2)
            run, rise = bx[k + 1] - bx[k], bz[k + 1] - bz[k]
            bed = bz[k] + ((x[:, 0] - bx[k]) / run).clamp(0.0, 1.0) * rise
            normal = torch.zeros_like(x)
            normal[:, 0], normal[:, vert] = -rise / run, 1.0
            rest(bed, normal / normal.norm(dim=1, keepdim=True))
            end = b.bathymetry.endX - (clearance if b.endWallTop is not None else 0.0)
            hold(0, b.wallX + clearance if b.wallTop is not None else -math.inf, end)
            return
        field = b.field
        z = to(field.z)
        raw = [(x[:, a] - float(axis[0])) / float(axis[1] - axis[0]) for a, axis in enumerate((field.x, field.y))]
        f = [r.clamp(0.0, s - 1.0) for r, s in zip(raw, (z.shape[1], z.shape[0]))]
        base = [t.floor() for t in f]
        # cubic convolution, its weights and their slopes
        weights, slopes = [], []
        for t, c in zip(f, base):
            u = t - c
            weights.append([-0.5 * u ** 3 + u ** 2 - 0.5 * u, 1.5 * u ** 3 - 2.5 * u ** 2 + 1.0,
                            -1.5 * u ** 3 + 2.0 * u ** 2 + 0.5 * u, 0.5 * u ** 3 - 0.5 * u ** 2])
            slopes.append([-1.5 * u ** 2 + 2.0 * u - 0.5, 4.5 * u ** 2 - 5.0 * u, -4.5 * u ** 2 + 4.0 * u + 0.5,
                           1.5 * u ** 2 - u])
        bed = bedX = bedY = torch.zeros_like(f[0])
        for p in range(4):
            row = (base[1].long() - 1 + p).clamp(0, z.shape[0] - 1)
            for q in range(4):
                value = z[row, (base[0].long() - 1 + q).clamp(0, z.shape[1] - 1)]
                bed = bed + weights[1][p] * weights[0][q] * value
                bedX = bedX + weights[1][p] * slopes[0][q] * value / field.spacingX
                bedY = bedY + slopes[1][p] * weights[0][q] * value / field.spacingY
        outside = [(r < 0.0) | (r > s - 1.0) for r, s in zip(raw, (z.shape[1], z.shape[0]))]
        normal = torch.stack([torch.where(outside[0], 0.0, -bedX), torch.where(outside[1], 0.0, -bedY),
                              torch.ones_like(bed)], 1)
        rest(bed, normal / normal.norm(dim=1, keepdim=True))
        startX, endX, startY, endY = field.bounds
        hold(1, startY + clearance, endY - clearance)
        hold(0, startX + clearance if b.offshoreWall else -math.inf, endX - clearance if b.endWall else endX)

    def advance(self):
        f = self.flow
        self.x0 = self.x.clone()
        self.pairs = _pairLists(self.x, self.h, 2.0 * f.smoothingLength, f.period)
        if f.densityFilterInterval and self.step > 0 and self.step % f.densityFilterInterval == 0:
            self.filter()
        self.p = self.tait(self.rho)
        if f.wallExtrapolated:
            self.wall()
        self.gradients()
        a = self.momentum()
        shortest = float(self.h.min())
        dt = f.cflNumber * shortest / (f.soundSpeed + float(self.v[self.fluid].norm(dim=1).max()))
        fastest = float(a[self.fluid].norm(dim=1).max())
        if fastest > 1e-12:
            dt = min(dt, f.cflNumber * math.sqrt(shortest / fastest))
        dt = min(dt, f.maxTimeStep)
        self.v = self.v + a * dt
        rho = self.rho + self.continuity() * dt
        self.rho = torch.where(self.fluid, rho.clamp(min=f.densityFloor), rho) if f.densityFloor > 0.0 else rho
        drift = self.transport() if f.xsphEpsilon > 0.0 else self.v
        self.x = torch.where(self.fluid[:, None], self.x + drift * dt, self.x)
        if f.period > 0.0:
            y = self.x[:, 1]
            self.x[:, 1] = torch.where(self.fluid, y - f.period * torch.floor(y / f.period), y)
        self.enforce()
        self.time, self.step = self.time + dt, self.step + 1


def exact(case: dict, seed: int):
    if work(case)['flops'] > 3e11:
        return None     # minutes of float64 pair sums
    prepared = prepare(case, seed)
    scheme = _Scheme(prepared['flow'], prepared['state'])
    del prepared
    for _ in range(case['steps']):
        scheme.advance()
    fluid = scheme.fluid
    return dict(time=scheme.time, positions=scheme.x[fluid], speeds=scheme.v[fluid].norm(dim=1), densities=scheme.rho)

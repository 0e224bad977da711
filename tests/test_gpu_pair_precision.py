"""What a pair's arithmetic keeps: float64's digits where a sum is taken in float64, and every bit of a
float32 quotient whose terms are small."""
from decimal import Decimal, getcontext

import numpy as np
import pytest

from test_gpu_pairs import C0, RHO0, cloud, pairSums

pytestmark = pytest.mark.gpu

getcontext().prec = 60


def exactRoot(value):
    return Decimal(value).sqrt()


@pytest.mark.parametrize('threads', [1, 4])
@pytest.mark.parametrize('dim', [2, 3])
def test_a_wall_pairs_distance_has_float64s_digits(dim, threads):
    # A fluid particle between two boundary particles whose terms cancel to about 1e-12 of either: the rate
    # is what is left, so an error of a term's distance shows in it.  h and every coordinate are exact in
    # binary, the velocities in 40 bits, and the rest is worked out in 60 digits.  Each term's roundings:
    # 2 of the root, which (1 - q / 2)^3 magnifies by at most 4.5 at q <= 1.2, and 5 of the products, each
    # 1.1e-16; two terms, 3e-15 in all.
    rng = np.random.default_rng(dim)
    h = 2.0 ** -6
    places = np.stack(np.meshgrid(*[np.arange(24 if dim == 2 else 8)] * dim, indexing='ij'), -1).reshape(-1, dim)
    centres = (places + 1) * (8 * h)
    n = len(centres)

    def offsets():
        direction = rng.normal(size=(n, dim))
        direction[:, 0] = np.sign(direction[:, 0]) * (np.abs(direction[:, 0]) + 0.5)     # well along x
        direction /= np.linalg.norm(direction, axis=1)[:, None]
        return np.round(direction * (h * rng.uniform(0.3, 1.2, (n, 1))) * 2.0 ** 36) / 2.0 ** 36

    first, second = offsets(), offsets()
    speed, left, size = np.empty(n), np.empty(n), np.empty(n)
    for k in range(n):
        terms = []
        for d in (first[k], second[k]):
            r = exactRoot(sum(Decimal(float(a)) ** 2 for a in d))
            terms.append((1 - r / (2 * Decimal(h))) ** 3 * Decimal(float(d[0])))
        s = float(-terms[0] / terms[1])
        speed[k] = np.round(s * 2.0 ** (39 - np.floor(np.log2(abs(s))))) / 2.0 ** (39 - np.floor(np.log2(abs(s))))
        left[k] = float(terms[0] + Decimal(speed[k]) * terms[1])
        size[k] = abs(float(terms[0]))
    x = np.concatenate([centres, centres - first, centres - second])
    v = np.zeros_like(x)
    v[n:2 * n, 0] = -1.0            # v_i - v_j along x: 1 and `speed`
    v[2 * n:, 0] = -speed
    fluid = np.arange(len(x)) < n
    from pysurf_b200.sphGpu import PairSums
    sums = PairSums(dim, h, np.zeros(dim), x.max(axis=0) + 8 * h, kernelType='wendlandC2')
    sums.setSweepOptions(True, threads)
    sums.update(x, np.ones(len(x)), fluid)
    rate = sums.continuityRate(v)[:n]
    scale = -5.0 * sums.sigmaUnit / h ** dim / h ** 2       # (dW/dr) / r = scale (1 - q / 2)^3
    assert np.median(np.abs(left) / size) > 1e-13           # there is something left to be found
    assert np.max(np.abs(rate / scale - left) / size) < 4e-15


@pytest.mark.parametrize('kernel', ['wendlandC2', 'cubicSpline'])
@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('power', [40, 60, 70])
def test_the_limited_viscosity_scales_with_the_velocities(dim, power, kernel):
    # Without pressure and gravity the limited viscosity is of degree one in the velocities, so velocities
    # scaled by a power of two scale every acceleration by it, bit for bit, down to slopes of 1e-22 whose
    # squares have no float32: the tail of a wave is such a flow.
    x, v, rho, m, fluid, h = cloud(dim, 900, 31, ratio=2.0)
    rho = np.full(len(x), RHO0)
    s = pairSums(dim, h, True, kernel=kernel)
    s.update(x, m, fluid)
    zero = np.zeros(len(x))
    whole = s.pairAccelerations(v, rho, zero, C0, 0.05, 0.5, np.zeros(dim))
    small = s.pairAccelerations(v * 2.0 ** -power, rho, zero, C0, 0.05, 0.5, np.zeros(dim))
    assert np.abs(whole).max() > 0.0 and np.array_equal(small, whole * 2.0 ** -power)


@pytest.mark.parametrize('dim', [2, 3])
def test_the_smallest_viscosity_is_not_lost(dim):
    # The same without the limiter at 2^-118, where the viscosity's numerator, alpha c0 h (v_ij . r_ij), has
    # no normal float32.  A product v d is off by half the least float32, 2^-150, three of them against the
    # largest v_ij . r_ij, some 2^-121: 1e-8 of it, and the acceleration's sums keep 1e-6 of the largest.
    x, v, rho, m, fluid, h = cloud(dim, 900, 37, ratio=2.0)
    rho = np.full(len(x), RHO0)
    s = pairSums(dim, h, True, limited=False)
    s.update(x, m, fluid)
    zero = np.zeros(len(x))
    whole = s.pairAccelerations(v, rho, zero, C0, 0.05, 0.5, np.zeros(dim))
    small = s.pairAccelerations(v * 2.0 ** -118, rho, zero, C0, 0.05, 0.5, np.zeros(dim))
    assert np.abs(small * 2.0 ** 118 - whole).max() < 1e-6 * np.abs(whole).max()


@pytest.mark.parametrize('dim', [2, 3])
def test_a_wall_pair_far_from_the_origin(dim):
    # With separations from the float32 points alone, whose places at 2^18 are 2^-5 = h / 4 apart, a pair's
    # float32 distance can be less than half its own.  The wall's term takes its distance in float64 from
    # that one: it stays within its value at no distance, m (5 sigma / h^2) |(v_i - v_j) . (x_i - x_j)|.
    from pysurf_b200.sphGpu import PairSums
    rng = np.random.default_rng(70 + dim)
    h = 2.0 ** -3
    side = 64 if dim == 2 else 16
    places = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing='ij'), -1).reshape(-1, dim)
    n = len(places)
    centres = 2.0 ** 18 + (places + 1) * (8 * h) + rng.uniform(-0.5, 0.5, (n, dim)) * h
    x = np.concatenate([centres, centres + rng.uniform(-0.6, 0.6, (n, dim)) * h])
    v = rng.uniform(-1.0, 1.0, (2 * n, dim))
    sums = PairSums(dim, h, x.min(axis=0) - h, x.max(axis=0) + h, kernelType='wendlandC2',
                    separationPrecision='float32')
    sums.update(x, np.ones(2 * n), np.arange(2 * n) < n)
    rate = np.abs(sums.continuityRate(v)[:n])
    bound = 5.0 * sums.sigmaUnit / h ** dim / h ** 2 * np.abs(((v[:n] - v[n:]) * (x[:n] - x[n:])).sum(axis=1))
    assert rate.max() > 0.0 and np.all(rate <= bound * (1.0 + 1e-6))

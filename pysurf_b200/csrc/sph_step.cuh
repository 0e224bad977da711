// sph_step.cuh -- what a step does around its sums, shared by the sweeps: when the density filter is due,
// the fluid maxima and the time step, a slot's acceleration, density update and drift.
#pragma once

#include <math.h>

#include "sph_enforce.cuh"

namespace sph {

__device__ __forceinline__ bool filterDue(const Control *ctl)
{
    if (!ctl) return true;
    if (!ctl->active) return false;
    if (ctl->filterInterval > 0) return ctl->step > 0 && ctl->step % ctl->filterInterval == 0;
    return ctl->filterNow != 0;
}

__device__ __forceinline__ double cflTimeStep(double h, double c0, double vmax, double amax, double cfl, double maxdt)
{
    double dt = cfl * h / (c0 + vmax);
    if (amax > 1e-12) dt = fmin(dt, cfl * sqrt(h / amax));
    return fmin(dt, maxdt);
}

__device__ __forceinline__ double warpMax(double value)
{
    for (int offset = 16; offset > 0; offset >>= 1) value = fmax(value, __shfl_xor_sync(0xFFFFFFFFu, value, offset));
    return value;
}

// The step's fluid maxima without a block barrier: each warp folds its lanes' values and lane 0
// raises the running maxima (atomicMax on the bits of non-negative doubles, which is order-free);
// the last warp to finish takes the time step in float64 and clears the running values.
__device__ __forceinline__ void foldMaxima(Control *ctl, double speed, double accel, int warps)
{
    // non-negative, and a NaN counts as 0 as fmax would take it
    speed = warpMax(speed > 0.0 ? speed : 0.0);
    accel = warpMax(accel > 0.0 ? accel : 0.0);
    if ((threadIdx.x & 31) != 0) return;
    atomicMax(&ctl->vmaxBits, (unsigned long long)__double_as_longlong(speed));
    atomicMax(&ctl->amaxBits, (unsigned long long)__double_as_longlong(accel));
    __threadfence();
    if (atomicAdd(&ctl->ticket, 1u) != (unsigned)(warps - 1)) return;
    __threadfence();
    const double vmax = __longlong_as_double((long long)atomicMax(&ctl->vmaxBits, 0ull));
    const double amax = __longlong_as_double((long long)atomicMax(&ctl->amaxBits, 0ull));
    ctl->vmax = vmax;
    ctl->amax = amax;
    ctl->vmaxBits = 0;
    ctl->amaxBits = 0;
    ctl->ticket = 0;
    if (!ctl->hostDt) {
        const double dt = cflTimeStep(ctl->hMin, ctl->soundSpeed, vmax, amax, ctl->cfl, ctl->maxTimeStep);
        if (!(dt > 0.0) || !isfinite(dt)) ctl->error |= kErrTimeStep;
        ctl->dt = dt;
    }
}

// A fluid slot's acceleration from its pair sum and gravity, with its speed and the acceleration's size
// for the maxima.
template <int D>
__device__ __forceinline__ void takeAcceleration(const Params &P, const Frame &F, int i, const float total[3], double &speed,
                                                 double &accel)
{
    float a[3] = {total[0] + P.g[0], total[1] + P.g[1], D == 3 ? total[2] + P.g[2] : 0.0f};
    F.acc[i] = make_float4(a[0], a[1], a[2], 0.0f);
    double v2 = 0.0;
    for (int c = 0; c < D; ++c) v2 += F.v[c][i] * F.v[c][i];
    speed = sqrt(v2);
    accel = (double)sqrtf(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
}

// rho += rate dt, the fluid floored (src/pysurf/sphGpu.py:1111-1140); returns the density before the floor.
__device__ __forceinline__ double advanceDensity(const Params &P, const Frame &F, int i, float rate, double dt, bool fluid,
                                                 Control *ctl)
{
    double rho = F.rho[i] + (double)rate * dt;
    const double unfloored = rho;
    if (P.densityFloor > 0.0 && fluid) rho = fmax(rho, P.densityFloor);
    F.rho[i] = rho;
    if (!isfinite(rho)) atomicOr(&ctl->error, kErrNonFinite);
    return unfloored;
}

// Drift (src/pysurf/sphGpu.py:1142-1186), the periodic wrap and the enforcement of one fluid slot.
template <int D>
__device__ __forceinline__ void driftAndEnforce(const Params &P, const Frame &F, const Enforcement &E, int i, double dt,
                                                const double *transport, Control *ctl)
{
    double x[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0}, lift = 0.0;
    for (int a = 0; a < D; ++a) {
        v[a] = F.v[a][i];
        const double start = F.x[a][i];
        x[a] = start + (transport ? transport[a] : v[a]) * dt;
        lift += P.gravity64[a] * (x[a] - start);
    }
    // the drift's change of potential energy, from the displacement as stored (src/pysurf/sphGpu.py:1168-1170)
    if (P.budget) addEnergy(P, F, i, kDrift, -F.m[i] * lift);
    if (P.period > 0.0) x[1] = x[1] - P.period * floor(x[1] / P.period);
    enforceTracked(P, F, E, D, i, x, v);
    bool finite = true;
    for (int a = 0; a < D; ++a) {
        F.x[a][i] = x[a];
        F.v[a][i] = v[a];
        finite = finite && isfinite(x[a]) && isfinite(v[a]);
    }
    if (!finite) atomicOr(&ctl->error, kErrNonFinite);
}

}  // namespace sph

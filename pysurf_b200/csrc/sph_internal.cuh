// sph_internal.cuh -- shared types and device helpers of the B200 delta-SPH backend.
//
// Layout in HBM (all arrays in the current sort order, slot s = 0..n-1):
//   master float64 state, double-buffered so a re-sort is one gather:
//     x[a], v[a] (a < dim), rho            integrated in float64, as the reference integrates
//   per-particle constants carried through each re-sort:
//     m, h (float64), fluid (uint8), orig (int32: the caller's index of the slot)
//   the sweeps' float32 frame, rebuilt from the master each step:
//     pa   float4  2D (hx, hy, lx, ly)      3D (hx, hy, hz, hs)
//     pb   float4  2D (m, hs, P2, rho)      3D (lx, ly, lz, V)
//     kin  float4  2D (vx, vy, V, dev)      3D (vx, vy, vz, dev)
//     aux  float4  3D (P2, rho, m, -)
//     low  float4  (vlx, vly, 2D m, 3D vlz, devLo): the float32 remainders of the float64 velocity and
//                  deviation
//     pres float   the pressure p
//   The rows lie so that each sweep reads few: gradients pa, kin (3D pb too); momentum pa, pb, kin (3D aux
//   too); continuity pa, kin, low (3D pb and m alone).
//   hi + lo is each float64 coordinate split into a float32 point and its float32 remainder, so a
//   separation (hi_i - hi_j) + (lo_i - lo_j) keeps the float64 positions' digits without float64
//   arithmetic (src/pysurf/sphGpu.py:227-242 states the same split).  hs is +h for a fluid
//   particle and -h for a boundary particle; dev is rho - rho0 in float32, taken in float64
//   (src/pysurf/sphGpu.py:1031-1038), so neighbours' density differences keep their digits.
//   The continuity sweep takes velocity and deviation differences from the float32 values and their
//   remainders, (v_i - v_j) + (vl_i - vl_j), so they keep float64's digits: continuity sums terms
//   that cancel (the velocity's divergence next to a wall, the hydrostatic subtraction near rest),
//   where a float32 value's rounding would otherwise dominate the rate.
//   V = m / rho and P2 = p / rho^2 are each particle's own, taken once per step instead of once per
//   pair: the same float32 quotients the pair sums would take.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sph {

constexpr int kBlock = 128;                 // threads per sweep block
// Resident sweep blocks an SM, which caps a sweep's registers (momentum, XSPH and the shifting's fields).
// Momentum, ms: 3D 4 (17.1 on the 20-ppd ridge, 21.2 at 3, 20.1 at 5); 2D 5 (0.078 on the 64-ppd beach,
// 0.090 at 4).  At 6 in 2D, with continuity at 6 too, the beach's plain form takes 0.073 and its step 2% less,
// but the forms that carry more spill: the closure's, the compensated, the mixed lengths' and the cubic
// spline's steps and those of 10,000 particles take 3 to 14% more.
template <int D>
constexpr int sweepMinBlocks() { return D == 2 ? 5 : 4; }
constexpr float kViscositySoftening = 0.01f;   // mu_ij's r^2 + 0.01 h^2 (src/pysurf/sphSolver.py:213)
constexpr float kCloseDistance = 0.3f;      // limiter fade (src/pysurf/sphSolver.py:220-221)
constexpr float kFoldWidth = 0.2f;
constexpr float kCandidateMargin = 1.0001f; // on r^2, as the reference's coarse test (src/pysurf/sphGpu.py:99)

constexpr int kStageCount = 7;              // a step's stages: cells, filter, wall, gradients, momentum, kick, continuity

// Error flags the device raises; the host reads them after each call that syncs.
enum DeviceError : int {
    kErrNonFinite = 1,      // a position, velocity or density stopped being finite
    kErrTimeStep = 2,       // the step collapsed (dt not positive and finite)
};

// Everything a sweep needs besides the arrays; passed by value.
struct Params {
    int n;                  // particles
    int dim;
    int kind;               // 0 cubic spline, 1 Wendland C2
    int mixedH;             // particles carry different smoothing lengths
    float hMax;             // longest smoothing length, sizes the cells
    float sigmaUnit;        // kernel sigma at h = 1
    // grid: cell c = (cz * ny + cy) * nx + cx, x fastest; coordinates clamped onto the grid
    double origin[3];
    double cellWidth;
    double perCell, perFine;    // 1 / cellWidth and 1 / fineWidth, for what needs no cell's exact bound
    int nc[3];
    int ncs;                // cells per support: the stencil is +-ncs cells
    int precise;            // separations from point + remainder (1) or the float32 points alone (0)
    // the fine level, for mixed smoothing lengths: a particle whose h is below fineBelow is sorted
    // into a second grid of fineWidth-wide cells (ncs to the fine level's longest h, fineMax),
    // numbered from fineFirst after the coarse grid's; a particle searches each grid only as far as
    // that grid's particles reach.  levels is 1 when no particle is on the fine level.
    int levels;
    double fineOrigin[3];
    double fineWidth;
    int fineNc[3];
    int fineFirst;
    int cells;              // both grids' cells
    float fineMax;
    double fineBelow;
    double period;          // periodic y axis length, 0 for none
    float periodF;
    // physics
    float c0, alpha, boundaryFactor;
    float g[3];
    double rho0, stiffness, densityFloor;  // the equation of state's rho0 and B = rho0 c0^2 / 7
    double devReference;    // the diffusion's rho0: deviations are rho - devReference
    float halfInvRho0;      // 0.5 / devReference: a pair's mean deviation over rho0
    int tension;            // the fluid may carry negative pressure
    int diffusion;          // 0 none, 1 molteni, 2 hydrostatic, 3 antuono
    float diffusionFactor;  // 2 delta c0
    float hydrostaticSlope; // rho0 g / c0^2, rounded once from float64: the hydrostatic density's slope in z
    int corrected;          // continuity takes L_i grad W
    int limited;            // viscosity limiter
    int wallExtrapolated;
    float xsphEpsilon;
    double gravity64[3];
    // delta-LES-SPH closure (src/pysurf/sphSolver.py:1232-1326): the eddy coefficients from the
    // velocity gradients, a viscous term on every fluid pair, the pair's diffusion coefficient
    int closure;
    float waterTerm;        // 2 (dim + 2) nu / c0: the water's own viscosity as an alpha times h
    float closureRho0;
    float closureC0;        // the closure's sound speed: its coefficients and its diffusion's 2 c0
    // particle shifting (src/pysurf/sphSolver.py:824-1010): W(dx) for the anti-clumping weight, the
    // free surface's divergence and lopsidedness thresholds, the size CFL Ma (2h)^2 or 2 h |v| dt
    int shifting, shiftLocal;
    float spacingKernel, shiftThreshold, lopsidedness;
    double shiftScale;      // c0 Ma 4 h: the size CFL Ma (2h)^2 = shiftScale dt
    double shiftDt;         // the host-step call's dt (the device steps take ctl->dt)
    // neighbour table: up to listCap entries a particle (a multiple of 8), entry k of slot i at
    // 4 ((k / 4) listStride + i) + k % 4, fluid neighbours from the front (0, 1, ...) and boundary
    // neighbours from the back (listCap - 1, listCap - 2, ...); listCap 0: no table, the sweeps walk the cells
    int listCap;
    int listStride;
    int together;           // the classic scheme's rows: both kinds from the front, in the walk's order
    // energy budget (src/pysurf/sphEnergy.py): each particle's running total of each term, by caller
    // index, column t at t * energyStride; the momentum sweep's parts of a at q * energyStride + slot
    int budget;
    int energyStride;
    // the momentum and continuity sums compensated (never with the budget: its sweeps keep plain sums)
    int compensated;
    // the stages of a step that start with this launch, one bit each (Control::stamps); 0 outside a step
    int stages;
};

// A step's kernels are launched to follow one another closely (launchNext): each starts here, waits for the
// kernel before it to be complete, and lets the next be set up as soon as all its own blocks run.  It reads
// and writes nothing before the wait.  The wait comes first, so that one kernel at most waits on the chip
// beside the running one, whatever streams share it.
__device__ __forceinline__ void awaitPrevious()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

// A load of what an earlier kernel of the step wrote: a plain one, since that kernel may still run when
// this one's blocks are set up (awaitPrevious), which the read-only path does not allow for.
template <class T>
__device__ __forceinline__ T fetch(const T *at) { return *at; }

// The float32 frame and the float64 master state, current buffers.
struct Frame {
    float4 *pa, *pb, *kin, *aux;
    float4 *low;            // remainders: velocity (xyz) and deviation (w)
    float *pres;            // pressure
    int *cell;              // sorted cell index of each slot
    const int *cellStart;   // lower bound of each cell in the sorted order, numCells + 1 entries
    float4 *G0, *G1, *G2;   // velocity gradient rows (2D: G0 = (G00, G01, G10, G11))
    // the slopes' coefficients, r . G r = sum over a <= b of them times r_a r_b: G_aa, and G_ab + G_ba.
    // 2D: S0 = (G00, G01 + G10, G11, -); 3D: S0 = (00, 01 + 10, 02 + 20, 11), S1 = (12 + 21, 22);
    // each times kSlopeScale
    float4 *S0;
    float2 *S1;
    float4 *L0, *L1, *L2;   // correction matrix rows, same packing
    float4 *gradRho;        // renormalized density gradient
    float4 *acc;            // acceleration (w: unused)
    float *rate;            // d rho / dt
    float *scalar;          // scratch per particle (Shepard, wall pressure outputs)
    float4 *vec;            // scratch per particle (XSPH transport velocity)
    float2 *eddy;           // closure: each particle's (alpha_i, delta_i)
    // shifting: grad C (w unused), grad C0 (w: div r, -1 where the support is lopsided, 1e6 on the
    // boundary), grad rho; the shift (w: the density change) and the velocity change
    float4 *shiftGrad, *shiftPlain, *shiftRhoGrad, *shift, *shiftDv;
    double *energy;         // energy budget: kEnergyTerms columns, by caller index
    float4 *parts;          // energy budget: pressure and viscosity of a from fluid and from boundary neighbours
    unsigned *wallBits;     // one bit a slot, set where it is boundary, 32 slots a word
    int *nbr;               // neighbour table (chunks of four), top bit: a pair across the periodic seam
    int2 *ncount;           // each slot's fluid and boundary neighbours (together they may exceed the row)
    // master (current buffers)
    double *x[3], *v[3], *rho, *m, *h;
    uint8_t *fluid;
    int *orig;
};

// Step control on the device: the time step is taken from the step's own maxima on the device,
// so a run of steps needs no host round trip (src/pysurf/sphSolver.py:1410-1424, 1980-1989).
struct Control {
    double time, untilTime, dt;
    long long step, lastStep;
    double vmax, amax;          // this step's fluid maxima
    double hMin, cfl, maxTimeStep, soundSpeed;   // the CFL step's inputs, float64 as the host takes them
    int active;                 // this step runs
    int hostDt;                 // dt comes from the host (residentIntegrate), not the maxima
    int filterNow;              // host-driven steps: this step filters the density (Shepard)
    long long filterInterval;   // device loop: filter every this many steps, 0 for none
    unsigned int ticket;        // last-warp-done counter of the maxima reduction
    int error;                  // DeviceError flags
    // the maxima reduction's running values: the bits of non-negative doubles, which order as the
    // doubles do, so an integer atomicMax takes their maximum in any order; zero between steps
    unsigned long long vmaxBits, amaxBits;
    // when each stage of the step started, and the step's end, in nanoseconds of the device's timer
    unsigned long long stamps[kStageCount + 1];
};

// Notes the time as the start of the stages whose bits are set (a stage without a kernel starts with the
// next one's).
__device__ __forceinline__ void stampStages(Control *ctl, int stages)
{
    if (!stages || blockIdx.x != 0 || threadIdx.x != 0 || !ctl || !ctl->active) return;
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    for (int k = 0; k <= kStageCount; ++k)
        if (stages >> k & 1) ctl->stamps[k] = now;
}

// ------------------------------------------------------------------------------------------
// Kernels W and (dW/dr) / r: src/pysurf/sphKernels.py:108-648; src/pysurf/sphGpu.py:139-204.
// The pair sums only ever take dW/dr divided by r (grad W = (dW/dr) r_ij / r), which for the
// Wendland C2 is -5 sigma (1 - q/2)^3 / h^2 with no division by r, and for the cubic spline
// sigma (2.25 q - 3) / h^2 inside q < 1.  The constants depend on h alone, so with one smoothing
// length they are taken once per thread.
// ------------------------------------------------------------------------------------------

struct KernelAt {
    float invH;     // 1 / h
    float sigma;    // sigma at h
    float gradC;    // Wendland: -5 sigma / h^2; cubic: sigma / h^2
    float soft;     // the viscosity's and the diffusion's softening 0.01 h^2
};

template <int K, int D>
__device__ __forceinline__ KernelAt kernelAt(float unit, float h)
{
    KernelAt k;
    k.invH = 1.0f / h;
    float s = unit * k.invH * k.invH;
    if (D == 3) s *= k.invH;
    k.sigma = s;
    k.gradC = (K == 1 ? -5.0f : 1.0f) * s * k.invH * k.invH;
    k.soft = kViscositySoftening * h * h;
    return k;
}

// The constants of two neighbours' pairs, side by side.
struct KernelPair {
    float2 invH, sigma, gradC, soft;
    __device__ __forceinline__ KernelAt of(int q) const
    {
        return q ? KernelAt{invH.y, sigma.y, gradC.y, soft.y} : KernelAt{invH.x, sigma.x, gradC.x, soft.x};
    }
};
__device__ __forceinline__ KernelPair kernelPair(const KernelAt &a, const KernelAt &b)
{
    return KernelPair{make_float2(a.invH, b.invH), make_float2(a.sigma, b.sigma), make_float2(a.gradC, b.gradC),
                      make_float2(a.soft, b.soft)};
}

// A pair's kernel constants at h_ij: one set a thread when every particle has the same smoothing
// length (then h_ij = hMax), else the set is held at the particle's own length, which every pair with
// a neighbour of the same length has (0.5 (h + h) = h exactly), so those pairs, all but the few across
// a refinement zone's edge, take the held set and the rest take theirs per pair, with the same bits
// either way.
template <int K, int D, bool MIXED>
struct Smoothing {
    KernelAt fixed;
    float held;     // the length `fixed` is taken at
    float unit;
    // own: the particle's smoothing length
    __device__ __forceinline__ explicit Smoothing(const Params &P, float own)
        : fixed(kernelAt<K, D>(P.sigmaUnit, MIXED ? own : P.hMax)), held(own), unit(P.sigmaUnit) {}
    __device__ __forceinline__ KernelPair at(const float2 &h) const
    {
        if (!MIXED || (h.x == held && h.y == held)) return kernelPair(fixed, fixed);
        return kernelPair(kernelAt<K, D>(unit, h.x), kernelAt<K, D>(unit, h.y));
    }
};

// W(q h), q < 2.  Roundings are explicit, so every sweep that inlines these takes the same bits.
template <int K>
__device__ __forceinline__ float kernelValue(float q, const KernelAt &k)
{
    if (K == 1) {
        const float rest = __fmaf_rn(-0.5f, q, 1.0f), sq = __fmul_rn(rest, rest);
        return __fmul_rn(__fmul_rn(__fmul_rn(k.sigma, sq), sq), __fmaf_rn(2.0f, q, 1.0f));
    }
    if (q < 1.0f) {
        const float q2 = __fmul_rn(q, q);
        return __fmul_rn(k.sigma, __fmaf_rn(__fmul_rn(0.75f, q2), q, __fmaf_rn(-1.5f, q2, 1.0f)));
    }
    const float rest = __fsub_rn(2.0f, q);
    return __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(k.sigma, 0.25f), rest), rest), rest);
}

// (dW/dr) / r at r = q h, 0 < q < 2.
template <int K>
__device__ __forceinline__ float kernelGradient(float q, const KernelAt &k)
{
    if (K == 1) {
        const float rest = __fmaf_rn(-0.5f, q, 1.0f);
        return __fmul_rn(__fmul_rn(__fmul_rn(k.gradC, rest), rest), rest);
    }
    if (q < 1.0f) return __fmul_rn(k.gradC, __fmaf_rn(2.25f, q, -3.0f));
    const float rest = __fsub_rn(2.0f, q);
    return __fdividef(__fmul_rn(__fmul_rn(__fmul_rn(-0.75f, k.gradC), rest), rest), q);
}

// (dW/dr) / r of two neighbours, each rounded as the single form.
template <int K>
__device__ __forceinline__ float2 kernelGradient(const float2 &q, const KernelPair &k)
{
    if (K == 1) {
        const float2 rest = __ffma2_rn(make_float2(-0.5f, -0.5f), q, make_float2(1.0f, 1.0f));
        return __fmul2_rn(__fmul2_rn(__fmul2_rn(k.gradC, rest), rest), rest);
    }
    return make_float2(kernelGradient<K>(q.x, k.of(0)), kernelGradient<K>(q.y, k.of(1)));
}

// (dW/dr) / r in float64 at a pair's float64 distance r, with the pair's (float32) kernel constants:
// the continuity sweep's wall pairs, whose terms cancel across a particle's neighbours, so each
// term's own rounding must stay well below float32's.
template <int K>
__device__ __forceinline__ double kernelGradient64(double r, const KernelAt &k)
{
    const double q = r * (double)k.invH;
    if (K == 1) {
        const double rest = 1.0 - 0.5 * q;
        return (double)k.gradC * rest * rest * rest;
    }
    if (q < 1.0) return (double)k.gradC * (2.25 * q - 3.0);
    const double rest = 2.0 - q;
    return -0.75 * (double)k.gradC * rest * rest / q;
}

__device__ __forceinline__ float sigmaAt(float unit, float h, int dim)
{
    return dim == 2 ? unit / (h * h) : unit / (h * h * h);
}

__device__ __forceinline__ int clampi(int a, int lo, int hi) { return a < lo ? lo : (a > hi ? hi : a); }

// Tait pressure B ((rho / rho0)^7 - 1), the power as three multiplies, clamped at zero unless the
// fluid may carry tension (src/pysurf/sphGpu.py:1058-1070).
__device__ __forceinline__ double taitPressure(const Params &P, double rho, bool fluid)
{
    double ratio = rho / P.rho0, sq = ratio * ratio;
    double p = P.stiffness * (sq * sq * sq * ratio - 1.0);
    if (!P.tension || !fluid) p = p > 0.0 ? p : 0.0;
    return p;
}

// The energy budget's terms, the columns of F.energy (src/pysurf/sphEnergy.py:92-98, deviceTerms).
enum EnergyTerm {
    kPressureFluid, kViscosityFluid, kPressureWall, kViscosityWall, kGravityWork, kContinuityFluid,
    kContinuityWall, kCorrection, kDiffusion, kFloor, kDrift, kClamp, kShifting, kFilter, kEnergyTerms
};

// e(rho), the Tait equation of state's elastic energy per unit mass (src/pysurf/sphEnergy.py:100-139):
// (c0^2 / 7) x^2 (21 + 35 x + 35 x^2 + 21 x^3 + 7 x^4 + x^5) / (6 (1 + x)), x = rho / rho0 - 1, so no
// digits cancel near rho0; zero below rho0 unless the fluid carries tension.
__device__ __forceinline__ double elasticEnergy(const Params &P, double rho)
{
    const double x = rho / P.rho0 - 1.0;
    if (!P.tension && x < 0.0) return 0.0;
    const double poly = 21.0 + x * (35.0 + x * (35.0 + x * (21.0 + x * (7.0 + x))));
    return (P.stiffness / P.rho0) * x * x * poly / (6.0 * (1.0 + x));
}

// The secant slope (e(after) - e(before)) / (after - before), or p / rho^2 at the midpoint for a
// change under 1e-10 rho0, where the two energies would lose their digits (src/pysurf/sphEnergy.py:141-160).
__device__ __forceinline__ double elasticSlope(const Params &P, double before, double after)
{
    const double change = after - before;
    if (fabs(change) > 1e-10 * P.rho0) return (elasticEnergy(P, after) - elasticEnergy(P, before)) / change;
    const double middle = 0.5 * (before + after);
    return taitPressure(P, middle, true) / (middle * middle);
}

// Adds to a fluid slot's running total of one term of the budget.
__device__ __forceinline__ void addEnergy(const Params &P, const Frame &F, int i, int term, double value)
{
    F.energy[(size_t)term * P.energyStride + F.orig[i]] += value;
}

// Cell coordinate of a float64 coordinate along an axis, clamped onto the grid.  Clamping is
// monotone and never parts two cells further than they were, so the +-ncs stencil still finds
// every neighbour of a particle outside the grid; only its candidates grow.
__device__ __forceinline__ int cellCoordinate(double value, double origin, double width, int count)
{
    double f = floor((value - origin) / width);
    if (!(f >= 0.0)) return 0;      // below the grid, or not a number: never an index outside it
    if (f > (double)(count - 1)) return count - 1;
    return (int)f;
}

// A box of cells of one grid around a centre cell, clamped to the grid: rows (y, z) of the
// x range [x0, x1]; the grid's cells are numbered from `first`, x fastest.
struct CellBox {
    int first, nx, ny;
    int cx, cy, cz;
    int x0, x1, y0, y1, z0, z1;
};

// The half-width in cells of a particle's search of a level's grid: the coarse grid's ncs (its
// cells are 2 hMax / ncs wide, and no pair reaches past 2 hMax), the fine grid's as many cells as
// hI + fineMax, the farthest a fine neighbour can be, spans.
__device__ __forceinline__ int searchCells(const Params &P, int level, float hI)
{
    if (level == 0) return P.ncs;
    return (int)ceil(((double)hI + (double)P.fineMax) / P.fineWidth - 1e-9);
}

// The box of +-n cells of a level's grid (0 coarse, 1 fine) around the cell holding pos; in the
// particle's own grid the centre is its sorted cell ownCell (y taken from pos when `image`, the
// search of a periodic image).  single: there is one level, so the own grid is the searched one.
__device__ __forceinline__ CellBox cellBox(const Params &P, int level, int ownCell, const double pos[3], bool image,
                                           int dim, int n, bool single = false)
{
    CellBox B;
    const bool fine = level == 1;
    B.nx = fine ? P.fineNc[0] : P.nc[0];
    B.ny = fine ? P.fineNc[1] : P.nc[1];
    const int nz = fine ? P.fineNc[2] : P.nc[2];
    B.first = fine ? P.fineFirst : 0;
    const double width = fine ? P.fineWidth : P.cellWidth;
    const double *origin = fine ? P.fineOrigin : P.origin;
    if (single || (ownCell >= P.fineFirst) == fine) {
        const int local = ownCell - B.first, row = local / B.nx;
        B.cx = local - row * B.nx;
        B.cz = dim == 3 ? row / B.ny : 0;
        B.cy = row - B.cz * B.ny;
        if (image) B.cy = cellCoordinate(pos[1], origin[1], width, B.ny);
    } else {
        B.cx = cellCoordinate(pos[0], origin[0], width, B.nx);
        B.cy = cellCoordinate(pos[1], origin[1], width, B.ny);
        B.cz = dim == 3 ? cellCoordinate(pos[2], origin[2], width, nz) : 0;
    }
    B.x0 = max(B.cx - n, 0);
    B.x1 = min(B.cx + n, B.nx - 1);
    B.y0 = max(B.cy - n, 0);
    B.y1 = min(B.cy + n, B.ny - 1);
    B.z0 = dim == 3 ? max(B.cz - n, 0) : 0;
    B.z1 = dim == 3 ? min(B.cz + n, nz - 1) : 0;
    return B;
}

// ------------------------------------------------------------------------------------------
// Frame access per dimension.
// ------------------------------------------------------------------------------------------

// A particle's signed smoothing length (+h fluid, -h boundary).
template <int D> __device__ __forceinline__ float signedLength(const Frame &F, int j);
template <> __device__ __forceinline__ float signedLength<2>(const Frame &F, int j) { return fetch(&F.pb[j].y); }
template <> __device__ __forceinline__ float signedLength<3>(const Frame &F, int j) { return fetch(&F.pa[j].w); }

// A slot's own fields.
template <int D> __device__ __forceinline__ float massOf(const Frame &F, int j)
{ return D == 2 ? fetch(&F.pb[j].x) : fetch(&F.aux[j].z); }
template <int D> __device__ __forceinline__ float pressureOf(const Frame &F, int j) { return fetch(&F.pres[j]); }
// p / rho^2
template <int D> __device__ __forceinline__ float pressureRatioOf(const Frame &F, int j)
{ return D == 2 ? fetch(&F.pb[j].z) : fetch(&F.aux[j].x); }
template <int D> __device__ __forceinline__ float deviationOf(const Frame &F, int j) { return fetch(&F.kin[j].w); }
// m / rho
template <int D> __device__ __forceinline__ float volumeOf(const Frame &F, int j)
{ return D == 2 ? fetch(&F.kin[j].z) : fetch(&F.pb[j].w); }
template <int D> __device__ __forceinline__ float densityOf(const Frame &F, int j)
{ return D == 2 ? fetch(&F.pb[j].w) : fetch(&F.aux[j].y); }

// A neighbour's rows, and its fields from them: pa (A), pb (B), kin (K), aux (X, 3D), low (L), and its mass
// where a sweep reads it apart from them.
struct NeighbourRows {
    float4 A, B, K, X, L;
    float m;
};
template <int D> __device__ __forceinline__ float signedLengthIn(const float4 &A, const float4 &B)
{ return D == 2 ? B.y : A.w; }
template <int D> __device__ __forceinline__ float massIn(const NeighbourRows &R) { return D == 2 ? R.B.x : R.X.z; }
template <int D> __device__ __forceinline__ float volumeIn(const NeighbourRows &R) { return D == 2 ? R.K.z : R.B.w; }
template <int D> __device__ __forceinline__ float deviationIn(const NeighbourRows &R) { return R.K.w; }
template <int D> __device__ __forceinline__ float densityIn(const NeighbourRows &R) { return D == 2 ? R.B.w : R.X.y; }
template <int D> __device__ __forceinline__ float pressureRatioIn(const NeighbourRows &R)
{ return D == 2 ? R.B.z : R.X.x; }
template <int D> __device__ __forceinline__ void pointIn(const float4 &A, float p[3])
{
    p[0] = A.x; p[1] = A.y; p[2] = D == 3 ? A.z : 0.0f;
}
template <int D> __device__ __forceinline__ void remainderIn(const float4 &A, const float4 &B, float l[3])
{
    if (D == 2) { l[0] = A.z; l[1] = A.w; l[2] = 0.0f; }
    else { l[0] = B.x; l[1] = B.y; l[2] = B.z; }
}
template <int D> __device__ __forceinline__ void velocityIn(const float4 &K, float v[3])
{
    v[0] = K.x; v[1] = K.y; v[2] = D == 3 ? K.z : 0.0f;
}

// Write a slot's density-derived fields: rho, rho - rho0, V = m / rho, p, p / rho^2.
template <int D>
__device__ __forceinline__ void storeDensity(const Frame &F, int i, float m, double rho64, double devReference, float p)
{
    const double dev64 = rho64 - devReference;
    const float rho = (float)rho64, dev = (float)dev64;
    const float volume = m / rho, ratio = p / (rho * rho);
    F.pres[i] = p;
    F.low[i].w = (float)(dev64 - (double)dev);
    F.kin[i].w = dev;
    if (D == 2) {
        F.pb[i].z = ratio; F.pb[i].w = rho;
        F.kin[i].z = volume;
    } else {
        F.pb[i].w = volume;
        F.aux[i].x = ratio; F.aux[i].y = rho;
    }
}

// Velocity (float32) of slot j.
template <int D> __device__ __forceinline__ void velocityOf(const Frame &F, int j, float v[3])
{
    float4 k = fetch(&F.kin[j]);
    v[0] = k.x; v[1] = k.y; v[2] = D == 3 ? k.z : 0.0f;
}

// Candidate coordinates (the float32 points alone) and the remainders.
template <int D> __device__ __forceinline__ void pointOf(const Frame &F, int j, float p[3]);
template <> __device__ __forceinline__ void pointOf<2>(const Frame &F, int j, float p[3])
{
    float4 a = fetch(&F.pa[j]); p[0] = a.x; p[1] = a.y; p[2] = 0.0f;
}
template <> __device__ __forceinline__ void pointOf<3>(const Frame &F, int j, float p[3])
{
    float4 a = fetch(&F.pa[j]); p[0] = a.x; p[1] = a.y; p[2] = a.z;
}

template <int D> __device__ __forceinline__ void remainderOf(const Frame &F, int j, float l[3]);
template <> __device__ __forceinline__ void remainderOf<2>(const Frame &F, int j, float l[3])
{
    float4 a = fetch(&F.pa[j]); l[0] = a.z; l[1] = a.w; l[2] = 0.0f;
}
template <> __device__ __forceinline__ void remainderOf<3>(const Frame &F, int j, float l[3])
{
    float4 b = fetch(&F.pb[j]); l[0] = b.x; l[1] = b.y; l[2] = b.z;
}

// Matrix rows (dim x dim) packed in float4 rows.
template <int D> __device__ __forceinline__ void loadMatrix(const float4 *R0, const float4 *R1, const float4 *R2,
                                                            int j, float M[3][3]);
template <> __device__ __forceinline__ void loadMatrix<2>(const float4 *R0, const float4 *, const float4 *, int j,
                                                          float M[3][3])
{
    float4 a = fetch(&R0[j]);
    M[0][0] = a.x; M[0][1] = a.y; M[1][0] = a.z; M[1][1] = a.w;
}
template <> __device__ __forceinline__ void loadMatrix<3>(const float4 *R0, const float4 *R1, const float4 *R2, int j,
                                                          float M[3][3])
{
    float4 a = fetch(&R0[j]), b = fetch(&R1[j]), c = fetch(&R2[j]);
    M[0][0] = a.x; M[0][1] = a.y; M[0][2] = a.z;
    M[1][0] = b.x; M[1][1] = b.y; M[1][2] = b.z;
    M[2][0] = c.x; M[2][1] = c.y; M[2][2] = c.z;
}

template <int D> __device__ __forceinline__ void storeMatrix(float4 *R0, float4 *R1, float4 *R2, int j,
                                                             const float M[3][3]);
template <> __device__ __forceinline__ void storeMatrix<2>(float4 *R0, float4 *, float4 *, int j, const float M[3][3])
{
    R0[j] = make_float4(M[0][0], M[0][1], M[1][0], M[1][1]);
}
template <> __device__ __forceinline__ void storeMatrix<3>(float4 *R0, float4 *R1, float4 *R2, int j,
                                                           const float M[3][3])
{
    R0[j] = make_float4(M[0][0], M[0][1], M[0][2], 0.0f);
    R1[j] = make_float4(M[1][0], M[1][1], M[1][2], 0.0f);
    R2[j] = make_float4(M[2][0], M[2][1], M[2][2], 0.0f);
}

// The slopes' coefficients are kept times 2^24, so that the limiter's products of two slopes stay normal
// floats down to slopes of 1e-26 m^2 / s (the tail of a wave has some of 1e-19, whose plain product is
// subnormal or zero); they overflow past 5e11.  A power of two changes no other bit.
constexpr float kSlopeScale = 16777216.0f;

// The slopes' coefficients of slot j (Frame::S0, S1), in the order (0,0), (0,1), (0,2), (1,1), ...
template <int D> __device__ __forceinline__ void loadSlopes(const Frame &F, int j, float s[6])
{
    const float4 a = fetch(&F.S0[j]);
    s[0] = a.x; s[1] = a.y; s[2] = a.z;
    if (D == 3) {
        const float2 b = fetch(&F.S1[j]);
        s[3] = a.w; s[4] = b.x; s[5] = b.y;
    }
}
template <int D> __device__ __forceinline__ void storeSlopes(const Frame &F, int j, const float G[3][3])
{
    constexpr float s = kSlopeScale;
    if (D == 2) {
        F.S0[j] = make_float4(s * G[0][0], s * (G[0][1] + G[1][0]), s * G[1][1], 0.0f);
    } else {
        F.S0[j] = make_float4(s * G[0][0], s * (G[0][1] + G[1][0]), s * (G[0][2] + G[2][0]), s * G[1][1]);
        F.S1[j] = make_float2(s * (G[1][2] + G[2][1]), s * G[2][2]);
    }
}

template <int D, class R> __device__ __forceinline__ R determinant(const R M[3][3])
{
    if (D == 2) return M[0][0] * M[1][1] - M[0][1] * M[1][0];
    return M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) - M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0])
         + M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
}

template <int D, class R> __device__ __forceinline__ void inverse(const R M[3][3], R out[3][3])
{
    R det = determinant<D>(M);
    R s = R(1) / det;
    if (D == 2) {
        out[0][0] = M[1][1] * s; out[0][1] = -M[0][1] * s;
        out[1][0] = -M[1][0] * s; out[1][1] = M[0][0] * s;
        return;
    }
    out[0][0] = (M[1][1] * M[2][2] - M[1][2] * M[2][1]) * s;
    out[0][1] = (M[0][2] * M[2][1] - M[0][1] * M[2][2]) * s;
    out[0][2] = (M[0][1] * M[1][2] - M[0][2] * M[1][1]) * s;
    out[1][0] = (M[1][2] * M[2][0] - M[1][0] * M[2][2]) * s;
    out[1][1] = (M[0][0] * M[2][2] - M[0][2] * M[2][0]) * s;
    out[1][2] = (M[0][2] * M[1][0] - M[0][0] * M[1][2]) * s;
    out[2][0] = (M[1][0] * M[2][1] - M[1][1] * M[2][0]) * s;
    out[2][1] = (M[0][1] * M[2][0] - M[0][0] * M[2][1]) * s;
    out[2][2] = (M[0][0] * M[1][1] - M[0][1] * M[1][0]) * s;
}

}  // namespace sph

// sph_classic_sweeps.cu -- the sweeps of the classic scheme: XSPH with the plain artificial viscosity and
// the plain continuity sum at one smoothing length, as the reference's default options run it.
//
// These runs take one neighbour at a time, in the walk's order, in chunks of four to a lane, and not the
// pairs of neighbours of sph_sweep_kernels.cu.  Their Shepard filter rounds the fluid's densities to
// float32 every few steps, so a rounding of one sum, which elsewhere stays below 1e-9 of a density, shows
// as a step of 6e-8 in it: the order of the sums and their roundings are part of the scheme's results.
// The default scheme's supports are short (h = 1.3 dx: some 20 neighbours in 2D, five or so a lane).
//
//   M  momentum     src/pysurf/sphSolver.py:1122-1149, 1192-1230; src/pysurf/sphGpu.py:303-414
//   D  continuity   src/pysurf/sphSolver.py:623-654; src/pysurf/sphGpu.py:430-545, 1111-1140
//   X  XSPH         src/pysurf/sphSolver.py:1358-1377; src/pysurf/sphGpu.py:725-766
//   S  Shepard      src/pysurf/sphGpu.py:768-802
#include <math.h>

#include "sph_enforce.cuh"
#include "sph_kernels.h"
#include "sph_step.cuh"
#include "sph_sweeps.cuh"

namespace sph {
namespace classic {

// W(q h) and (dW/dr) / r, as sph_internal.cuh's, the compiler choosing where a product and a sum fuse.
template <int K>
__device__ __forceinline__ float value(float q, const KernelAt &k)
{
    if (K == 1) {
        float rest = 1.0f - 0.5f * q, sq = rest * rest;
        return k.sigma * sq * sq * (2.0f * q + 1.0f);
    }
    if (q < 1.0f) return k.sigma * (1.0f - 1.5f * q * q + 0.75f * q * q * q);
    float rest = 2.0f - q;
    return k.sigma * 0.25f * rest * rest * rest;
}

template <int K>
__device__ __forceinline__ float gradient(float q, const KernelAt &k)
{
    if (K == 1) {
        float rest = 1.0f - 0.5f * q;
        return k.gradC * rest * rest * rest;
    }
    if (q < 1.0f) return k.gradC * (2.25f * q - 3.0f);
    float rest = 2.0f - q;
    return __fdividef(-0.75f * k.gradC * rest * rest, q);
}

// A neighbour's rows as far as the visitor reads them: kKinetic, kAux (3D) and kLow the rows, kMass the mass
// alone (3D).  `early` keeps the loads where they stand.
template <int D, bool early, class Visitor>
__device__ __forceinline__ void loadRows(const Frame &F, int j, const float4 &A, NeighbourRows &R)
{
    auto row = [](const float4 *at) { return early ? loadEarly(at) : fetch(at); };
    R.A = A;
    R.B = row(&F.pb[j]);
    if (Visitor::kKinetic) R.K = row(&F.kin[j]);
    if (D == 3 && Visitor::kAux) R.X = row(&F.aux[j]);
    if (D == 3 && Visitor::kMass) R.X.z = fetch(&F.aux[j].z);
    if (Visitor::kLow) R.L = row(&F.low[j]);
}

// Visits slot i's neighbours in the walk's order: of those counted (a boundary row's are its fluid
// neighbours, unless `whole`), lane t of T takes those whose count k has k / 4 = t mod T, from the table's
// row (all of them from its front; P.together) when it holds them, else from the cells.  The visitor gets
// (j, d, r, whether j is fluid, whether the pair lies across the seam, j's rows) when accept(fluidJ).
//
// From the table, a lane's next neighbour's rows load while one is summed, and its next chunk of entries a
// chunk ahead; the visits keep their order, and so the bits.  The 12-ppd ridge's momentum takes 3.2 ms so and
// 4.2 without, its continuity and XSPH 7.9 and 9.2; the 64-ppd beach's 0.065 and 0.074, 0.123 and 0.143.
template <int D, int T, class Visitor>
__device__ __forceinline__ void forEachNeighbour(const Params &P, const Frame &F, int i, int t, bool whole, Visitor &visit)
{
    const bool boundaryRow = signedLength<D>(F, i) <= 0.0f, fluidOnly = boundaryRow && !whole;
    float pi[3], li[3];
    pointOf<D>(F, i, pi);
    remainderOf<D>(F, i, li);
    const float reach = 2.0f * P.hMax, limit = kCandidateMargin * reach * reach;
    Origin O{0, P.hMax, false, 0.0};
    if (D == 3 && P.period > 0.0 && (pi[1] < reach || pi[1] > P.periodF - reach)) {
        O.seam = true;
        O.shift64 = pi[1] < 0.5f * P.periodF ? P.period : -P.period;
    }
    // a neighbour within the support, its separation taken
    auto take = [&](int j, int image, const float d[3], float r2, const NeighbourRows &R) {
        const float r = r2 > 0.0f ? r2 * rsqrtf(r2) : 0.0f;
        if (Visitor::kSkipCoincident && r < 1.0e-12f) return;
        visit(j, d, r, signedLengthIn<D>(R.A, R.B) > 0.0f, image, R);
    };
    auto separation = [&](const NeighbourRows &R, int image, float d[3]) {
        float pj[3], lj[3];
        pointIn<D>(R.A, pj);
        remainderIn<D>(R.A, R.B, lj);
        return separation2<D>(P, pi, li, pj, lj, image ? (float)O.shift64 : 0.0f, image, O.shift64, d);
    };
    const int held = P.listCap > 0 && !(whole && boundaryRow) ? fetch(&F.ncount[i]).x : P.listCap + 1;
    if (P.listCap > 0 && held <= P.listCap) {
        const int4 *column = reinterpret_cast<const int4 *>(F.nbr) + i;
        int k = 4 * t;
        if (k >= held) return;
        int4 chunk = make_int4(0, 0, 0, 0), ahead = fetch(column + (size_t)t * P.listStride);
        auto next = [&](int &entry) {
            if (k >= held) return false;
            if ((k & 3) == 0) {
                chunk = ahead;
                const int after = (k >> 2) + T;
                if (4 * after < held) ahead = fetch(column + (size_t)after * P.listStride);
            }
            entry = chunk.x;
            chunk.x = chunk.y; chunk.y = chunk.z; chunk.z = chunk.w;
            k = (k & 3) == 3 ? k + 1 + 4 * (T - 1) : k + 1;
            return true;
        };
        int entry = 0;
        NeighbourRows R;
        bool more = next(entry);
        loadRows<D, true, Visitor>(F, entry & 0x7FFFFFFF, loadEarly(&F.pa[entry & 0x7FFFFFFF]), R);
        while (more) {
            int entryAfter = 0;
            NeighbourRows after;
            more = next(entryAfter);
            if (more) loadRows<D, true, Visitor>(F, entryAfter & 0x7FFFFFFF, loadEarly(&F.pa[entryAfter & 0x7FFFFFFF]), after);
            if (visit.accept(signedLengthIn<D>(R.A, R.B) > 0.0f)) {
                const int image = entry < 0 ? 1 : 0;
                float d[3];
                const float r2 = separation(R, image, d);
                take(entry & 0x7FFFFFFF, image, d, r2, R);
            }
            entry = entryAfter;
            R = after;
        }
        return;
    }
    O.cell = F.cell[i];
    Candidates<D, false> C;
    C.cellStart = F.cellStart;
    C.startSearch(P, O, pi, li, 0);
    int counted = 0, j = 0, image = 0, level = 0;
    while (C.next(P, O, pi, li, j, image, level)) {
        const float4 A = fetch(&F.pa[j]);
        float pj[3], d[3];
        pointIn<D>(A, pj);
        const float offset = image ? (float)O.shift64 : 0.0f;     // the search's origin: particle or image
        if (coarseDistance2<D>(pi, pj, offset) >= limit || j == i) continue;
        NeighbourRows R;
        loadRows<D, false, Visitor>(F, j, A, R);
        const bool fluidJ = signedLengthIn<D>(A, R.B) > 0.0f;
        if (fluidOnly && !fluidJ) continue;     // not in the row: not counted either
        if (T == 1 && !visit.accept(fluidJ)) continue;
        const float r2 = separation(R, image, d);
        if (r2 >= support2(P.hMax)) continue;
        if (T > 1) {
            if ((counted++ >> 2) % T != t) continue;
            if (!visit.accept(fluidJ)) continue;
        }
        take(j, image, d, r2, R);
    }
}

template <int D, int K>
struct ShepardVisit {
    static constexpr bool kSkipCoincident = false;
    static constexpr bool kKinetic = D == 2, kAux = false, kMass = true, kLow = false;
    const Frame &F;
    KernelAt k;
    float num, den;
    __device__ bool accept(bool) const { return true; }
    __device__ void operator()(int j, const float *, float r, bool, int, const NeighbourRows &R)
    {
        float w = value<K>(r * k.invH, k);
        num += massIn<D>(R) * w;
        den += volumeIn<D>(R) * w;
    }
};

template <int D, int K, int T>
__global__ void __launch_bounds__(kBlock, 6) shepardKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    stampStages(const_cast<Control *>(ctl), P.stages);
    if (!filterDue(ctl)) return;
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    const float hs = signedLength<D>(F, i);
    // a device step filters the fluid alone; the host-step call (no control block) returns every row
    if (ctl && hs <= 0.0f) return;
    float own = sigmaAt(P.sigmaUnit, fabsf(hs), D);
    float mi = massOf<D>(F, i);
    ShepardVisit<D, K> visit{F, kernelAt<K, D>(P.sigmaUnit, P.hMax), G.t == 0 ? mi * own : 0.0f,
                             G.t == 0 ? volumeOf<D>(F, i) * own : 0.0f};
    forEachNeighbour<D, T>(P, F, i, G.t, true, visit);
    float num = groupSum<T>(visit.num, G.mask), den = groupSum<T>(visit.den, G.mask);
    if (G.t != 0) return;
    F.scalar[i] = num / den;
}

// BUDGET: the sum split for the energy budget too, into the pressure and the viscosity of fluid and of
// boundary neighbours (src/pysurf/sphGpu.py:400-414); the sum's own roundings are explicit, so a tracked
// run is the plain run bit for bit.
template <int D, int K, bool BUDGET>
struct MomentumVisit {
    static constexpr bool kSkipCoincident = true;
    static constexpr bool kKinetic = true, kAux = true, kMass = false, kLow = false;
    const Params &P; const Frame &F;
    KernelAt k;
    float vi[3], rhoI, own, viscosityScale;   // viscosityScale: -alpha c0
    float total[3], parts[BUDGET ? 4 : 1][3];
    __device__ bool accept(bool) const { return true; }
    __device__ void operator()(int j, const float *d, float r, bool fluidJ, int, const NeighbourRows &R)
    {
        const float h = P.hMax, q = r * k.invH;
        float vj[3];
        velocityIn<D>(R.K, vj);
        float rel[3] = {vi[0] - vj[0], vi[1] - vj[1], vi[2] - vj[2]};
        float approach = rel[0] * d[0] + rel[1] * d[1] + (D == 3 ? rel[2] * d[2] : 0.0f);
        float viscosity = 0.0f;
        if (approach < 0.0f) {
            // -alpha c0 h (v_ij . r_ij) / ((r^2 + 0.01 h^2) (rho_i + rho_j) / 2); the denominator is
            // a positive normal float for any physical pair, which __fdividef takes to 2 ulp
            viscosity = __fdividef(viscosityScale * h * approach,
                                   (r * r + k.soft) * (0.5f * (rhoI + densityIn<D>(R))));
            if (!fluidJ) viscosity *= P.boundaryFactor;
        }
        const float ratioJ = pressureRatioIn<D>(R);
        const float pressureTerm = __fadd_rn(own, ratioJ);
        float coefficient = -__fadd_rn(pressureTerm, viscosity) * massIn<D>(R);
        float f = coefficient * gradient<K>(q, k);
        for (int a = 0; a < D; ++a) total[a] = __fmaf_rn(f, d[a], total[a]);
        if constexpr (BUDGET) {
            const float grad = massIn<D>(R) * gradient<K>(q, k);
            const float fp = -pressureTerm * grad, fv = -viscosity * grad;
            if (fluidJ) {
                for (int a = 0; a < D; ++a) { parts[0][a] += fp * d[a]; parts[1][a] += fv * d[a]; }
            } else {
                for (int a = 0; a < D; ++a) { parts[2][a] += fp * d[a]; parts[3][a] += fv * d[a]; }
            }
        }
    }
};

template <int D, int K, int T, bool BUDGET>
__global__ void __launch_bounds__(kBlock, BUDGET ? 4 : D == 2 ? 8 : 6) momentumKernel(Params P, Frame F, Control *ctl, int maxima)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(ctl, P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    double speed = 0.0, accel = 0.0;
    if (i < P.n) {
        if (signedLength<D>(F, i) <= 0.0f) {
            if (G.t == 0) F.acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            MomentumVisit<D, K, BUDGET> visit{P, F, kernelAt<K, D>(P.sigmaUnit, P.hMax)};
            velocityOf<D>(F, i, visit.vi);
            visit.rhoI = densityOf<D>(F, i);
            visit.own = pressureRatioOf<D>(F, i);
            visit.viscosityScale = -P.alpha * P.c0;
            visit.total[0] = visit.total[1] = visit.total[2] = 0.0f;
            if constexpr (BUDGET)
                for (int q = 0; q < 4; ++q) visit.parts[q][0] = visit.parts[q][1] = visit.parts[q][2] = 0.0f;
            forEachNeighbour<D, T>(P, F, i, G.t, false, visit);
            for (int a = 0; a < D; ++a) visit.total[a] = groupSum<T>(visit.total[a], G.mask);
            if constexpr (BUDGET) {
                for (int q = 0; q < 4; ++q) {
                    for (int a = 0; a < D; ++a) visit.parts[q][a] = groupSum<T>(visit.parts[q][a], G.mask);
                    if (G.t == 0)
                        F.parts[(size_t)q * P.energyStride + i] =
                            make_float4(visit.parts[q][0], visit.parts[q][1], D == 3 ? visit.parts[q][2] : 0.0f, 0.0f);
                }
            }
            if (G.t == 0) takeAcceleration<D>(P, F, i, visit.total, speed, accel);
        }
    }
    if (maxima) foldMaxima(ctl, speed, accel, (int)(gridDim.x * (blockDim.x >> 5)));
}

// Fluid pairs in float32 from the velocities and their remainders; a fluid-boundary pair in float64, as
// the paired sweep's.  BUDGET: the sum over fluid and over boundary neighbours apart.
template <int D, int K, bool BUDGET>
struct ContinuityVisit {
    static constexpr bool kSkipCoincident = true;
    static constexpr bool kKinetic = true, kAux = false, kMass = true, kLow = true;
    const Params &P; const Frame &F;
    KernelAt k;
    int self;               // this particle's slot
    bool boundaryI;
    float vi[3], vlI[3];
    float total;
    double cross;           // the fluid-boundary pairs' terms in float64
    float plainFluid, plainWall;    // BUDGET
    __device__ bool accept(bool fluidJ) const { return !(boundaryI && !fluidJ); }
    __device__ void operator()(int j, const float *d, float r, bool fluidJ, int image, const NeighbourRows &R)
    {
        float vj[3];
        velocityIn<D>(R.K, vj);
        const float vlJ[3] = {R.L.x, R.L.y, R.L.z};
        if (boundaryI == fluidJ) {
            float pi[3], li[3], pj[3], lj[3];
            pointOf<D>(F, self, pi);
            remainderOf<D>(F, self, li);
            pointIn<D>(R.A, pj);
            remainderIn<D>(R.A, R.B, lj);
            double dd[3] = {0.0, 0.0, 0.0}, r2 = 0.0;
            for (int a = 0; a < D; ++a) {
                dd[a] = ((double)pi[a] - (double)pj[a]) + ((double)li[a] - (double)lj[a]);
                if (a == 1 && image) dd[a] += pi[1] < 0.5f * P.periodF ? P.period : -P.period;
                r2 = fma(dd[a], dd[a], r2);
            }
            const double rf = (double)r, rr = fma(fma(-rf, rf, r2), 0.5 / rf, rf);
            const double grad = kernelGradient64<K>(rr, k);
            double dot = 0.0;
            for (int a = 0; a < D; ++a)
                dot = fma(((double)vi[a] + (double)vlI[a]) - ((double)vj[a] + (double)vlJ[a]), dd[a], dot);
            const double term = (double)massIn<D>(R) * dot * grad;
            cross += term;
            if constexpr (BUDGET) {
                if (fluidJ) plainFluid += (float)term;
                else plainWall += (float)term;
            }
            return;
        }
        const float grad = gradient<K>(r * k.invH, k);    // (dW/dr) / r
        float dv[3];
        for (int a = 0; a < D; ++a)
            dv[a] = __fadd_rn(__fsub_rn(vi[a], vj[a]), __fsub_rn(vlI[a], vlJ[a]));
        float dot = 0.0f;
        for (int a = 0; a < D; ++a) dot += dv[a] * d[a];
        const float massDot = massIn<D>(R) * dot;
        total = __fmaf_rn(massDot, grad, total);
        if constexpr (BUDGET) plainFluid = __fmaf_rn(massDot, grad, plainFluid);
    }
};

// mode 0: the rate only; 1: advance the density (XSPH drifts).
template <int D, int K, int T, bool BUDGET>
__global__ void __launch_bounds__(kBlock, BUDGET || D == 3 ? 4 : 5) continuityKernel(Params P, Frame F, Control *ctl, int mode)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(ctl, P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    const float hs = signedLength<D>(F, i);
    ContinuityVisit<D, K, BUDGET> visit{P, F, kernelAt<K, D>(P.sigmaUnit, P.hMax)};
    visit.boundaryI = hs <= 0.0f;
    velocityOf<D>(F, i, visit.vi);
    const float4 lowI = F.low[i];
    visit.vlI[0] = lowI.x; visit.vlI[1] = lowI.y; visit.vlI[2] = lowI.z;
    visit.self = i;
    visit.cross = 0.0;
    visit.total = visit.plainFluid = visit.plainWall = 0.0f;
    forEachNeighbour<D, T>(P, F, i, G.t, false, visit);
    float rate = groupSum<T>(visit.total, G.mask);
    // the fluid-boundary pairs' float64 sum joins before the one rounding to float32
    rate = (float)((double)rate + groupSum<T>(visit.cross, G.mask));
    float parts[2] = {0.0f, 0.0f};
    if constexpr (BUDGET) {
        parts[0] = groupSum<T>(visit.plainFluid, G.mask);
        parts[1] = groupSum<T>(visit.plainWall, G.mask);
    }
    if (G.t != 0) return;
    F.rate[i] = rate;
    if (mode == 0) return;
    const double dt = ctl->dt, start = F.rho[i], unfloored = advanceDensity(P, F, i, rate, dt, hs > 0.0f, ctl);
    if (BUDGET && hs > 0.0f) {
        const double m = F.m[i], slope = elasticSlope(P, start, unfloored);
        for (int q = 0; q < 2; ++q) addEnergy(P, F, i, kContinuityFluid + q, m * slope * (double)parts[q] * dt);
        addEnergy(P, F, i, kFloor, m * (elasticEnergy(P, F.rho[i]) - elasticEnergy(P, unfloored)));
    }
}

template <int D, int K>
struct XsphVisit {
    static constexpr bool kSkipCoincident = false;
    static constexpr bool kKinetic = true, kAux = true, kMass = false, kLow = false;
    const float *densities;
    KernelAt k;
    float vi[3], rhoI, corr[3];
    __device__ bool accept(bool fluidJ) const { return fluidJ; }
    __device__ void operator()(int j, const float *, float r, bool, int, const NeighbourRows &R)
    {
        float w = value<K>(r * k.invH, k);
        float rhoJ = densities ? densities[j] : densityIn<D>(R);
        float weight = massIn<D>(R) * w / (0.5f * (rhoI + rhoJ));
        float vj[3];
        velocityIn<D>(R.K, vj);
        for (int a = 0; a < D; ++a) corr[a] += weight * (vj[a] - vi[a]);
    }
};

template <int D, int K, int T>
__global__ void __launch_bounds__(kBlock, D == 2 ? 8 : 6)
xsphKernel(Params P, Frame F, Control *ctl, Enforcement E, const float *densities, int mode)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    float v[3];
    velocityOf<D>(F, i, v);
    if (signedLength<D>(F, i) <= 0.0f) {
        if (G.t == 0) F.vec[i] = make_float4(v[0], v[1], v[2], 0.0f);
        return;
    }
    XsphVisit<D, K> visit{densities, kernelAt<K, D>(P.sigmaUnit, P.hMax)};
    visit.vi[0] = v[0]; visit.vi[1] = v[1]; visit.vi[2] = v[2];
    visit.rhoI = densities ? densities[i] : densityOf<D>(F, i);
    visit.corr[0] = visit.corr[1] = visit.corr[2] = 0.0f;
    forEachNeighbour<D, T>(P, F, i, G.t, false, visit);
    for (int a = 0; a < D; ++a) visit.corr[a] = groupSum<T>(visit.corr[a], G.mask);
    if (G.t != 0) return;
    float t[3];
    for (int a = 0; a < 3; ++a) t[a] = v[a] + P.xsphEpsilon * visit.corr[a];
    F.vec[i] = make_float4(t[0], t[1], t[2], 0.0f);
    if (mode != 2) return;
    double transport[3] = {(double)t[0], (double)t[1], (double)t[2]};
    driftAndEnforce<D>(P, F, E, i, ctl->dt, transport, ctl);
}

template <int D, int K, int T>
static void launchT(const LaunchArgs &A, Stage stage)
{
    const int grid = (int)(((long long)A.P.n * T + kBlock - 1) / kBlock);
    cudaStream_t st = A.stream;
    switch (stage) {
    case Stage::ShepardSum: launchNext(shepardKernel<D, K, T>, grid, kBlock, st, A.P, A.F, A.ctl); break;
    case Stage::Momentum:
        if (A.P.budget && A.maxima) launchNext(momentumKernel<D, K, T, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxima);
        else launchNext(momentumKernel<D, K, T, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxima);
        break;
    case Stage::Continuity:
        // the budget's parts matter only where the step advances the density
        if (A.P.budget && A.flag != 0) launchNext(continuityKernel<D, K, T, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.flag);
        else launchNext(continuityKernel<D, K, T, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.flag);
        break;
    case Stage::Xsph: launchNext(xsphKernel<D, K, T>, grid, kBlock, st, A.P, A.F, A.ctl, A.E, A.densities, A.flag); break;
    default: break;
    }
}

template <int D, int K>
static void launchDK(const LaunchArgs &A, Stage stage)
{
    if (A.threads >= 8) return launchT<D, K, 8>(A, stage);
    if (A.threads == 4) return launchT<D, K, 4>(A, stage);
    if (A.threads == 2) return launchT<D, K, 2>(A, stage);
    return launchT<D, K, 1>(A, stage);
}

}  // namespace classic

void launchClassicStage(const LaunchArgs &A, Stage stage)
{
    if (A.P.n == 0) return;
    if (A.P.dim == 2) return A.P.kind == 0 ? classic::launchDK<2, 0>(A, stage) : classic::launchDK<2, 1>(A, stage);
    return A.P.kind == 0 ? classic::launchDK<3, 0>(A, stage) : classic::launchDK<3, 1>(A, stage);
}

}  // namespace sph

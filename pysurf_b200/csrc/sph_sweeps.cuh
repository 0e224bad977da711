// sph_sweeps.cuh -- the neighbour walk every sweep shares, and its neighbour table.
//
// A particle's neighbours lie in the cells within +-ncs of its own along each axis; cells are
// numbered x fastest, so each (y, z) row of the stencil is one contiguous run of the sorted
// order, [cellStart[first], cellStart[last + 1]).  Candidates are tested on their float32 points
// first (the reference's coarse test, src/pysurf/sphGpu.py:330-336), and only survivors take the
// precise separation (hi_i - hi_j) + (lo_i - lo_j).
//
// Each step the table kernel walks the cells once and records, per particle, the neighbours the
// walk accepts, in the walk's order, in a table of 16-byte chunks: entries 4c .. 4c + 3 of particle
// i form chunk c, stored at c * stride + i, so the chunks c of a warp's particles are contiguous.  A
// row holds the fluid neighbours from its front and the boundary neighbours from its back, so that a
// sweep sums each kind in a loop of its own, without a test of each neighbour's kind.
// The sweeps then read the table
// instead of walking the cells: no candidate that fails the distance test is visited again, so
// a warp's lanes stay busy.  A particle with more neighbours than its row holds walks the cells
// instead.  Table and walk hand the same pairs of neighbours to the same arithmetic, whose roundings
// are explicit on every path that differs, so a sweep gives the same bits either way.
//
// T threads serve one particle: lane t of the group takes the particle's neighbours of a kind
// k = t, t + T, t + 2T, ..., counted in the walk's order, so that the lanes read neighbouring slots' rows together
// (the order runs along the grid's rows, where slots follow one another), and the group sums its
// partial sums with a butterfly of shuffles, which gives every lane the same bits (each level adds two values whose
// order does not matter).  T = 1 is the plain one-thread-per-particle sweep.
//
// A periodic y axis (3D) is searched a second time from the particle's image across the seam
// when it lies within its reach of the seam (src/pysurf/sphGpu.py:206-225).  Each search tests
// its candidates against its own origin (the particle, or its image); a period longer than twice
// the reach (the solver requires twice the support, src/pysurf/sphSolver.py:1465-1467) keeps any
// neighbour from passing both tests.  Pairs across the seam take their separation in float64:
// their points are a period apart and their float32 difference would lose the digits the split
// keeps.  The table marks such pairs in the entry's top bit.
#pragma once

#include <type_traits>

#include "sph_internal.cuh"

namespace sph {

// The lanes of a group of T threads that serve one particle.
template <int T>
struct Group {
    int i;              // the particle (sorted slot)
    int t;              // this thread's lane in the group
    unsigned mask;      // the group's lanes in the warp
};

template <int T>
__device__ __forceinline__ Group<T> groupOf()
{
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    Group<T> G;
    G.i = (int)(g / T);
    G.t = (int)(g % T);
    const int lane = threadIdx.x & 31;
    G.mask = T >= 32 ? 0xFFFFFFFFu : (((1u << T) - 1u) << (lane & ~(T - 1)));
    return G;
}

// The group's sum, the same bits on every lane.
template <int T>
__device__ __forceinline__ float groupSum(float value, unsigned mask)
{
    for (int offset = T / 2; offset > 0; offset >>= 1) value += __shfl_xor_sync(mask, value, offset, T);
    return value;
}

template <int T>
__device__ __forceinline__ double groupSum(double value, unsigned mask)
{
    for (int offset = T / 2; offset > 0; offset >>= 1) value += __shfl_xor_sync(mask, value, offset, T);
    return value;
}

// Compensated accumulation (Ogita, Rump and Oishi, "Accurate sum and dot product", SIAM J. Sci.
// Comput. 26 (2005), Dot2): a running sum s with a running error c.  Each term a b enters as its
// rounded product p and the product's exact error fma(a, b, -p); Knuth's TwoSum gives the exact
// error of s + p.  Both errors gather in c, so s + c is the sum as if taken in twice the precision.
// Every rounding is an explicit intrinsic, so no contraction changes a bit.
__device__ __forceinline__ void twoSum(float a, float b, float &sum, float &error)
{
    sum = __fadd_rn(a, b);
    const float bv = __fsub_rn(sum, a);
    error = __fadd_rn(__fsub_rn(a, __fsub_rn(sum, bv)), __fsub_rn(b, bv));
}

__device__ __forceinline__ void addProduct(float a, float b, float &s, float &c)
{
    const float p = __fmul_rn(a, b);
    const float productError = __fmaf_rn(a, b, -p);
    float sum, sumError;
    twoSum(s, p, sum, sumError);
    s = sum;
    c = __fadd_rn(c, __fadd_rn(productError, sumError));
}

// The group's compensated sum, the same bits on every lane: TwoSum is exact whichever operand comes
// first, so each lane's pair of partner values combines to the same (s, c).
template <int T>
__device__ __forceinline__ float groupSumCompensated(float s, float c, unsigned mask)
{
    for (int offset = T / 2; offset > 0; offset >>= 1) {
        const float s2 = __shfl_xor_sync(mask, s, offset, T), c2 = __shfl_xor_sync(mask, c, offset, T);
        float sum, error;
        twoSum(s, s2, sum, error);
        s = sum;
        c = __fadd_rn(__fadd_rn(c, c2), error);
    }
    return __fadd_rn(s, c);
}

// The same from a lane's two running sums (its even and its odd neighbours').
template <int T>
__device__ __forceinline__ float groupSumCompensated(const float2 &s, const float2 &c, unsigned mask)
{
    float sum, error;
    twoSum(s.x, s.y, sum, error);
    return groupSumCompensated<T>(sum, __fadd_rn(__fadd_rn(c.x, c.y), error), mask);
}

// The coarse test's squared distance between float32 points, and a pair's separation and squared
// distance.  Each takes its roundings from explicit intrinsics, so that the table kernel and the
// walk, compiled apart, reach the same decision on a pair at the edge of the support.  The support
// test is r^2 < (2 h)^2, so a rejected candidate takes no square root; it parts from the
// reference's r < 2 h only where the two roundings straddle 2 h, where W and grad W vanish.
template <int D>
__device__ __forceinline__ float coarseDistance2(const float pi[3], const float pj[3])
{
    const float cx = __fsub_rn(pi[0], pj[0]), cy = __fsub_rn(pi[1], pj[1]);
    float r2 = __fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy));
    if (D == 3) {
        const float cz = __fsub_rn(pi[2], pj[2]);
        r2 = __fadd_rn(r2, __fmul_rn(cz, cz));
    }
    return r2;
}
// From pi moved by offset across the periodic seam.
template <int D>
__device__ __forceinline__ float coarseDistance2(const float pi[3], const float pj[3], float offset)
{
    const float at[3] = {pi[0], __fadd_rn(pi[1], offset), pi[2]};
    return coarseDistance2<D>(at, pj);
}

// d = x_i - x_j from the points and remainders (image: across the periodic seam, in float64); r^2.
// PRECISE 1 or 0 fixes the form at compile time, -1 takes it from P.precise.
template <int D, int PRECISE = -1>
__device__ __forceinline__ float separation2(const Params &P, const float pi[3], const float li[3], const float pj[3],
                                            const float lj[3], float offset, int image, double shift64, float d[3])
{
    if (PRECISE == 0 || (PRECISE < 0 && !P.precise)) {
        // separationPrecision 'float32': the points alone (src/pysurf/sphGpu.py:227-242)
        d[0] = __fsub_rn(pi[0], pj[0]);
        d[1] = __fsub_rn(__fadd_rn(pi[1], offset), pj[1]);
        d[2] = D == 3 ? __fsub_rn(pi[2], pj[2]) : 0.0f;
    } else if (!image) {
        for (int a = 0; a < D; ++a) d[a] = __fadd_rn(__fsub_rn(pi[a], pj[a]), __fsub_rn(li[a], lj[a]));
        if (D == 2) d[2] = 0.0f;
    } else {
        for (int a = 0; a < D; ++a)
            d[a] = (float)(((double)pi[a] + (double)li[a]) - ((double)pj[a] + (double)lj[a]));
        d[1] = (float)((((double)pi[1] + (double)li[1]) + shift64) - ((double)pj[1] + (double)lj[1]));
        if (D == 2) d[2] = 0.0f;
    }
    float r2 = __fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1]));
    if (D == 3) r2 = __fadd_rn(r2, __fmul_rn(d[2], d[2]));
    return r2;
}

// Two neighbours' values side by side: Blackwell's packed float32 instructions take both in one issue
// slot, each rounded as the single instruction rounds.
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(const float2 &a, const float2 &b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(const float2 &a, const float2 &b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(const float2 &a, const float2 &b, const float2 &c) { return __ffma2_rn(a, b, c); }

// A pair's distance from its squared distance: r^2 times the hardware reciprocal square root (about 2
// ulp), 0 for a coincident pair, and that reciprocal (finite always).  The support is decided on r^2,
// so r only enters the kernel's value and gradient, where its rounding is of the float32 terms' own
// size; continuity's and the correction matrix's float64 parts take preciseRoot() from it.  The .ftz form skips the subnormal scaling of rsqrtf; the floor keeps its argument
// normal, and a pair under it (r < 1e-15 m) is coincident to every kernel.
constexpr float kLeastDistance2 = 1.0e-30f;
__device__ __forceinline__ float inverseRoot(float r2)
{
    float inverse;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inverse) : "f"(fmaxf(r2, kLeastDistance2)));
    return inverse;
}

// A distance in float64 from its square, by way of y, the float32 reciprocal root of the square's float32
// value: with e = 1 - r2 y^2, about 5e-7, r = r2 y (1 - e)^(-1/2) = r2 y (1 + e / 2 + 3 e^2 / 8 + ...), and
// the next term, 5 e^3 / 16, lies below float64's rounding.  One Newton step scaled by y in float32 left up
// to 6e-14 and, for its conversions, took longer: the 64-ppd beach's gradients 0.0607 -> 0.0576 ms, the
// 10-ppd ridge's continuity 2.57 -> 2.52 (a division in place of y: 3.00).
//
// APART: y may be the root of another separation's square, the float32 points' alone, which far from the
// origin can be less than half of this one for a close pair: e goes no further than -2/3, where the series
// begins to rise again.  (A Newton step for those, behind a branch, took 25% off the 3D continuity's speed.)
template <bool APART = false>
__device__ __forceinline__ double preciseRoot(double r2, float inverse)
{
    const double y = (double)inverse, near = __dmul_rn(r2, y), rest = fma(-near, y, 1.0);
    const double e = APART && rest < -2.0 / 3.0 ? -2.0 / 3.0 : rest;
    return fma(__dmul_rn(near, e), fma(0.375, e, 0.5), near);
}

// a / b to 2 ulp for a normal b up to 2^126: __fdividef without its subnormal scaling.  A subnormal, taken or
// given, counts as zero, so it stands only where none can matter: the limiter's and the viscosity's quotients
// are of scaled values (kSlopeScale, kViscosityScale), and the diffusion's r^2 / (r^2 + 0.01 h^2) has r above
// 1e-12.  With __fdividef at these the ridges' steps take 0.5% longer.
__device__ __forceinline__ float quickDivide(float a, float b)
{
    float q;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(a), "f"(b));
    return q;
}

// (2 h)^2, the support test's bound.
__device__ __forceinline__ float support2(float h)
{
    const float w = __fmul_rn(2.0f, h);
    return __fmul_rn(w, w);
}

// A squared distance under which the coarse test's float32 points alone decide a pair at one
// smoothing length: a coarse r^2 below it leaves the precise r^2 (separation2, points plus
// remainders, not across the seam) below `support`.  The frame's remainders are the float32 rest
// of each float64 coordinate, |l| <= 2^-24 |x| (gatherKernel), so each axis of the separation
// moves by at most 6e-8 (|p_i| + |p_j|) over the points' difference, and a candidate under the
// bound has |p_j| <= |p_i| + 2h per axis; 1e-5 of 2h covers the roundings of both distances and of
// the bound itself (a few float32 roundings).  So a table built with it holds the same entries.
__device__ __forceinline__ float sureSupport2(float support, const float pi[3])
{
    const float s = sqrtf(support);
    const float spread = 6.0e-8f * (2.0f * (fabsf(pi[0]) + fabsf(pi[1]) + fabsf(pi[2])) + 3.0f * s) + 1.0e-37f;
    const float edge = fmaxf(s * (1.0f - 1.0e-5f) - spread, 0.0f);
    return edge * edge;
}

// The table kernels' bound for a particle of length hI at point pi: sureSupport2 of the support its
// coarse-grid candidates share.  One smoothing length: (2 h)^2.  Two grid levels: every particle on
// the coarse grid has h >= P.fineBelow, so its float32 length is at least P.hMax and each pair's
// support is at least that of (hI + P.hMax) / 2 (the roundings are monotone); the fine grid's
// candidates take the precise test.  Mixed lengths on one grid: none (0).
__device__ __forceinline__ float sureBound(const Params &P, float support, float hI, const float pi[3])
{
    if (P.mixedH) return P.levels > 1 ? sureSupport2(support2(0.5f * (hI + P.hMax)), pi) : 0.0f;
    return sureSupport2(support, pi);
}

// What a walk needs to set up each of a particle's searches: its sorted cell, point, remainder,
// length, and the periodic image's shift when it lies near the seam.
struct Origin {
    int cell;
    float hI;
    bool seam;
    double shift64;
};

// Whether a slot is fluid, and whether a run of slots holds any of a kind, from the slots' bits (32 a word,
// so a run of a stencil row is a few words).
__device__ __forceinline__ bool isFluid(const unsigned *wallBits, int j)
{
    return !(fetch(&wallBits[j >> 5]) >> (j & 31) & 1);
}
__device__ __forceinline__ bool runHas(const unsigned *wallBits, int first, int end, bool walls)
{
    const unsigned flip = walls ? 0u : 0xFFFFFFFFu;
    unsigned any = 0;
    for (int w = first >> 5; w <= (end - 1) >> 5; ++w) {
        unsigned bits = fetch(&wallBits[w]) ^ flip;
        if (w == first >> 5) bits &= 0xFFFFFFFFu << (first & 31);
        if (w == (end - 1) >> 5) bits &= 0xFFFFFFFFu >> (31 - ((end - 1) & 31));
        any |= bits;
    }
    return any != 0;
}

// The candidates of a walk over the cells of slot i's searches, one at a time.  Search s is of grid
// level s >> 1 (coarse, then fine when the particles carry two levels of smoothing length) from origin
// s & 1 (the particle, then its periodic image when it lies near the seam).
// FINE: the particles carry two levels of smoothing length (else only the coarse grid is searched).
template <int D, bool FINE>
struct Candidates {
    int search, first, nx, ny, x0, x1, y0, y1, z1, zz, yy, j, end;
    const int *cellStart;

    __device__ __forceinline__ void startRow()
    {
        const int row = first + (zz * ny + yy) * nx;
        j = fetch(&cellStart[row + x0]) - 1;
        end = fetch(&cellStart[row + x1 + 1]);
    }

    // Starts search s when it applies (its level is present, its image is wanted); false if not.
    __device__ __forceinline__ bool startSearch(const Params &P, const Origin &O, const float pi[3], const float li[3],
                                                int s)
    {
        const int level = FINE ? s >> 1 : 0, image = s & 1;
        if ((!FINE && s >= 2) || level >= P.levels || (image && !O.seam)) return false;
        const double pos[3] = {(double)pi[0] + (double)li[0],
                               (double)pi[1] + (double)li[1] + (image ? O.shift64 : 0.0),
                               D == 3 ? (double)pi[2] + (double)li[2] : 0.0};
        const CellBox B = cellBox(P, level, O.cell, pos, image != 0, D, searchCells(P, level, O.hI), !FINE);
        first = B.first;
        nx = B.nx;
        ny = B.ny;
        x0 = B.x0;
        x1 = B.x1;
        y0 = B.y0;
        y1 = B.y1;
        z1 = B.z1;
        zz = B.z0;
        yy = B.y0;
        search = s;
        startRow();
        return true;
    }

    // The next row's run, of slots j + 1 .. end - 1; false when there are none left.
    __device__ __forceinline__ bool nextRow(const Params &P, const Origin &O, const float pi[3], const float li[3])
    {
        if (yy < y1) {
            ++yy;
        } else if (zz < z1) {
            ++zz;
            yy = y0;
        } else {
            constexpr int searches = FINE ? 4 : 2;
            int s = search + 1;
            while (s < searches && !startSearch(P, O, pi, li, s)) ++s;
            return s < searches;
        }
        startRow();
        return true;
    }

    // The next candidate into (jOut, imageOut, levelOut); false when there are none left.
    __device__ __forceinline__ bool next(const Params &P, const Origin &O, const float pi[3], const float li[3],
                                         int &jOut, int &imageOut, int &levelOut)
    {
        while (++j >= end)
            if (!nextRow(P, O, pi, li)) return false;
        jOut = j;
        imageOut = search & 1;
        levelOut = FINE ? search >> 1 : 0;
        return true;
    }
};

// The pairs a sweep sums: of a fluid neighbour, of a boundary neighbour, or (continuity) of a fluid and
// a boundary particle, whichever way round.
enum PairKind { kFluidPair, kWallPair, kCrossPair };

// Whether a visitor takes two neighbours at a time (kPaired).
template <class V, class = void>
struct Paired {
    static constexpr bool value = false;
};
template <class V>
struct Paired<V, std::void_t<decltype(V::kPaired)>> {
    static constexpr bool value = V::kPaired;
};

// Whether a visitor's pipeline copies the rows and its walk is each lane's own (kAlone; sumPairs() says when).
template <class V, class = void>
struct Alone {
    static constexpr bool value = false;
};
template <class V>
struct Alone<V, std::void_t<decltype(V::kAlone)>> {
    static constexpr bool value = V::kAlone;
};

// A row's load, which stays where it is written: the compiler would otherwise move it down to its first
// use, and the software pipeline of sumPairs() with it.
__device__ __forceinline__ float4 loadEarly(const float4 *at)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
    return v;
}

// A neighbour's rows, as far as the visitor reads them: kBody the 2D body row (pb; 3D always, for the
// remainders), kKinetic, kAux (3D) and kLow the others, kMass the mass apart from its row.  FINE reads the
// length, in the 2D body row.
template <int D, bool FINE, class Visitor>
__device__ __forceinline__ void loadRows(const Frame &F, int j, NeighbourRows &R)
{
    R.A = loadEarly(&F.pa[j]);
    if constexpr (D == 3 || FINE || Visitor::kBody) R.B = loadEarly(&F.pb[j]);
    if constexpr (Visitor::kKinetic) R.K = loadEarly(&F.kin[j]);
    if constexpr (D == 3 && Visitor::kAux) R.X = loadEarly(&F.aux[j]);
    if constexpr (Visitor::kLow) R.L = loadEarly(&F.low[j]);
    if constexpr (Visitor::kMass && D == 2) R.m = R.L.z;
    if constexpr (Visitor::kMass && D == 3)
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(R.m) : "l"(&F.aux[j].z));
}

// Two neighbours of a particle as a paired visitor gets them: their slots, whether each counts and lies
// across the seam; d = x_i - x_j, h_ij, and, for finish(), r and 1 / r and the kernel's constants at h_ij.
struct Neighbours {
    int j[2];
    bool live[2];
    int image[2];
    float2 d[3], h, r, inverse;
    KernelPair k;
};

// A particle's row as its sweep opens it: its slot, this lane, its length, point and remainder, the
// periodic image's shift when it lies near the seam, its fluid and boundary neighbours in the table,
// and whether the table lists them (else the sweep walks the cells).  A boundary particle's row holds
// its fluid neighbours only: every sweep over boundary rows takes fluid neighbours alone, except the
// Shepard sum, which walks a boundary row's cells for all of them (whole).
struct Row {
    int i, t;
    float hI, pi[3], li[3], reach;
    double shift64;
    bool seam, listed;
    int2 count;
};

// FINE: the smoothing lengths differ; else every length is P.hMax.
template <int D, bool FINE>
__device__ __forceinline__ Row openRow(const Params &P, const Frame &F, int i, int t, float hI, bool whole = false)
{
    Row O;
    O.i = i;
    O.t = t;
    O.hI = hI;
    pointOf<D>(F, i, O.pi);
    remainderOf<D>(F, i, O.li);
    O.reach = FINE ? hI + P.hMax : 2.0f * P.hMax;
    O.seam = false;
    O.shift64 = 0.0;
    if (D == 3 && P.period > 0.0 && (O.pi[1] < O.reach || O.pi[1] > P.periodF - O.reach)) {
        O.seam = true;
        O.shift64 = O.pi[1] < 0.5f * P.periodF ? P.period : -P.period;
    }
    O.count = P.listCap > 0 && !whole ? fetch(&F.ncount[i]) : make_int2(0, 0);
    O.listed = P.listCap > 0 && !whole && O.count.x + O.count.y <= P.listCap;
    return O;
}

// Two neighbours' pairs go in two parts, so that the rows of the next two can load in between, into the
// registers these two's rows leave: takeBoth() reads all it needs from the rows, finishBoth() sums.
// A visitor with kPaired has a take<KIND>(N, R0, R1) that returns what its finish<KIND>(N, taken) adds,
// the two neighbours together in packed float32; any other is called with each that counts in turn, from
// its rows.
// entry0, entry1: table entries (the slot, the top bit a pair across the seam); second: whether there is
// an entry1 (else it repeats entry0, and does not count).  A neighbour at r < 1e-12 does not count where
// Visitor::kSkipCoincident.
struct BothRows {
    NeighbourRows R0, R1;
};
template <int D, int PRECISE, bool FINE, PairKind KIND, class Visitor>
__device__ __forceinline__ auto takeBoth(const Params &P, const Row &O, int entry0, int entry1, bool second,
                                         const NeighbourRows &R0, const NeighbourRows &R1, Visitor &visit,
                                         Neighbours &N)
{
    const int entries[2] = {entry0, entry1};
    float d[2][3], r2[2], h[2];
    for (int q = 0; q < 2; ++q) {
        const NeighbourRows &R = q ? R1 : R0;
        N.j[q] = entries[q] & 0x7FFFFFFF;
        N.image[q] = D == 3 && entries[q] < 0 ? 1 : 0;
        float pj[3], lj[3];
        pointIn<D>(R.A, pj);
        remainderIn<D>(R.A, R.B, lj);
        r2[q] = separation2<D, PRECISE>(P, O.pi, O.li, pj, lj, N.image[q] ? (float)O.shift64 : 0.0f, N.image[q],
                                        O.shift64, d[q]);
        h[q] = FINE ? 0.5f * (O.hI + fabsf(signedLengthIn<D>(R.A, R.B))) : P.hMax;
        N.live[q] = (q == 0 || second) && (!Visitor::kSkipCoincident || r2[q] >= 1.0e-24f);
    }
    for (int a = 0; a < 3; ++a) N.d[a] = make_float2(d[0][a], d[1][a]);
    N.r = make_float2(r2[0], r2[1]);        // r^2 until finishBoth()
    N.h = make_float2(h[0], h[1]);
    if constexpr (Paired<Visitor>::value) return visit.template take<KIND>(N, R0, R1);
    else return BothRows{R0, R1};
}

// What takeBoth() returns for a visitor.
template <int D, bool FINE, PairKind KIND, class Visitor>
using Taken = decltype(takeBoth<D, 1, FINE, KIND>(std::declval<const Params &>(), std::declval<const Row &>(), 0, 0, true,
                                                  std::declval<const NeighbourRows &>(),
                                                  std::declval<const NeighbourRows &>(), std::declval<Visitor &>(),
                                                  std::declval<Neighbours &>()));

template <PairKind KIND, class Visitor, class TakenValues>
__device__ __forceinline__ void finishBoth(Neighbours &N, const TakenValues &taken, Visitor &visit)
{
    N.inverse = make_float2(inverseRoot(N.r.x), inverseRoot(N.r.y));
    N.r = mul2(N.r, N.inverse);
    N.k = visit.S.at(N.h);
    if constexpr (Paired<Visitor>::value) {
        visit.template finish<KIND>(N, taken);
    } else {
        const float d0[3] = {N.d[0].x, N.d[1].x, N.d[2].x}, d1[3] = {N.d[0].y, N.d[1].y, N.d[2].y};
        if (N.live[0]) visit(N.j[0], d0, N.r.x, N.h.x, N.k.of(0), taken.R0);
        if (N.live[1]) visit(N.j[1], d1, N.r.y, N.h.y, N.k.of(1), taken.R1);
    }
}

template <int D, int PRECISE, bool FINE, PairKind KIND, class Visitor>
__device__ __forceinline__ void visitBoth(const Params &P, const Row &O, int entry0, int entry1, bool second,
                                          const NeighbourRows &R0, const NeighbourRows &R1, Visitor &visit)
{
    Neighbours N;
    const auto taken = takeBoth<D, PRECISE, FINE, KIND>(P, O, entry0, entry1, second, R0, R1, visit, N);
    finishBoth<KIND>(N, taken, visit);
}

// Visit the neighbours of one kind (fluid or boundary) of an open row, as pairs of KIND.  Every such
// neighbour j != i with r^2 < (2 h_ij)^2 (the table's criterion) is counted in the walk's order; lane t
// of T takes those whose count k has k = t mod T, two at a time.
template <int D, int T, bool FINE, PairKind KIND, class Visitor>
__device__ __forceinline__ void sumPairs(const Params &P, const Frame &F, const Row &O, bool fluid, Visitor &visit)
{
    if (O.listed) {
        // the lane's entries: k = t, t + T, ... from the row's front, or from its back
        const int count = fluid ? O.count.x : O.count.y;
        const int *column = F.nbr + 4 * (size_t)O.i;
        const long long stride = 4ll * P.listStride;
        auto place = [&](int k) {
            const int e = fluid ? k : P.listCap - 1 - k;
            return column + (e >> 2) * stride + (e & 3);
        };
        auto entry = [&](const int *at) {
            int value;
            asm volatile("ld.global.L1::no_allocate.b32 %0, [%1];" : "=r"(value) : "l"(at));
            return value;
        };
        int left = count > O.t ? (count - O.t - 1) / T + 1 : 0;
        if (P.precise) {
            // A software pipeline over the lane's entries: the next two neighbours' rows load while two
            // are summed, and the entries after them.  The T lanes of a particle read T neighbouring
            // entries, and the particles of a warp lie side by side in each chunk, so a warp's load of
            // one entry a lane is whole 128-byte lines; each line is read once, so it is kept out of L1,
            // which the neighbours' rows need.  The first entries load without waiting for the count:
            // whatever lies past it is not read as one.
            int ring[4];
            for (int q = 0; q < 4; ++q) ring[q] = O.t + q * T < P.listCap ? entry(place(O.t + q * T)) : 0;
            if (left == 0) return;
            // a chunk holds four entries, so with four lanes or more every entry a lane takes is the
            // same distance on
            const long long step = (fluid ? T : -T) * (stride / 4);
            const int *ahead = place(min(O.t + 4 * T, P.listCap - 1));
            int k = O.t;
            NeighbourRows R0, R1;
            if (left < 2) ring[1] = ring[0];
            loadRows<D, FINE, Visitor>(F, ring[0] & 0x7FFFFFFF, R0);
            loadRows<D, FINE, Visitor>(F, ring[1] & 0x7FFFFFFF, R1);
            while (true) {
                const int j0 = ring[0], j1 = ring[1];
                Neighbours N;
                // the rows' values that the sums need come first, or (kAlone) copies of the rows, so that the
                // next rows load into the same registers meanwhile
                BothRows C;
                Taken<D, FINE, KIND, Visitor> taken;
                if constexpr (Alone<Visitor>::value) C = BothRows{R0, R1};
                else taken = takeBoth<D, 1, FINE, KIND>(P, O, j0, j1, left > 1, R0, R1, visit, N);
                ring[0] = ring[2];
                ring[1] = left == 3 ? ring[2] : ring[3];
                // the entries first: issued after the rows, they were 8% slower to arrive (2D continuity)
                int e2 = 0, e3 = 0;
                if (left > 4) e2 = entry(T >= 4 ? ahead : place(k + 4 * T));
                if (left > 5) e3 = entry(T >= 4 ? ahead + step : place(k + 5 * T));
                if (left > 2) {
                    loadRows<D, FINE, Visitor>(F, ring[0] & 0x7FFFFFFF, R0);
                    loadRows<D, FINE, Visitor>(F, ring[1] & 0x7FFFFFFF, R1);
                }
                if (left > 4) ring[2] = e2;
                if (left > 5) ring[3] = e3;
                if constexpr (Alone<Visitor>::value)
                    taken = takeBoth<D, 1, FINE, KIND>(P, O, j0, j1, left > 1, C.R0, C.R1, visit, N);
                finishBoth<KIND>(N, taken, visit);
                if (left <= 2) break;
                left -= 2;
                if (T >= 4) ahead += 2 * step;
                else k += 2 * T;
            }
            return;
        }
        // separations from the float32 points alone
        for (int k = O.t; left > 0; left -= 2, k += 2 * T) {
            const int j0 = entry(place(k)), j1 = left > 1 ? entry(place(k + T)) : j0;
            NeighbourRows R0, R1;
            loadRows<D, FINE, Visitor>(F, j0 & 0x7FFFFFFF, R0);
            loadRows<D, FINE, Visitor>(F, j1 & 0x7FFFFFFF, R1);
            visitBoth<D, 0, FINE, KIND>(P, O, j0, j1, left > 1, R0, R1, visit);
        }
        return;
    }

    // The walk: the group's lanes test T candidates of a row's run at a time, and a ballot hands the
    // accepted ones to the lanes whose turn it is.  A row's run of one kind alone, as most are, is passed
    // over for the other.  Without a table the 64-ppd beach steps in 1.13 ms so (2.28 with every lane
    // testing all candidates of both kinds), the 8-ppd ridge in 27.0 (51.3).
    //
    // kAlone keeps that form, which has no ballot, for a sweep whose rows nearly all come from the table:
    // beside a walk with ballots the 3D gradients take 2.00 ms on the 10-ppd ridge (2.57 with copied rows),
    // beside this one 1.82.
    constexpr bool kAlone = Alone<Visitor>::value;
    constexpr int W = kAlone ? 1 : T;       // candidates a round
    const float limit = kCandidateMargin * O.reach * O.reach;
    // the coarse test's bound for fine candidates: no fine neighbour lies past hI + fineMax
    const float fineReach = O.hI + P.fineMax;
    const float fineLimit = kCandidateMargin * fineReach * fineReach;
    const Origin origin{F.cell[O.i], O.hI, O.seam, O.shift64};
    const int lane = (threadIdx.x & 31) & ~(W - 1);     // the group's first lane
    const unsigned group = W >= 32 ? 0xFFFFFFFFu : ((1u << W) - 1u) << lane;
    Candidates<D, FINE> C;
    C.cellStart = F.cellStart;
    C.startSearch(P, origin, O.pi, O.li, 0);
    int base = C.end, counted = 0, held = 0;
    bool holds = false, ended = false, asks = false, first = true;
    while (true) {
        while (base >= C.end && !ended) {
            if (!first) ended = !C.nextRow(P, origin, O.pi, O.li);
            first = false;
            base = C.j + 1;
            if (ended || base >= C.end) continue;
            asks = runHas(F.wallBits, base, C.end, fluid);      // the other kind
            if (asks && !runHas(F.wallBits, base, C.end, !fluid)) base = C.end;
        }
        int entry = held;
        if (!ended) {
            const int image = C.search & 1, level = FINE ? C.search >> 1 : 0, j = base + O.t % W;
            const float offset = image ? (float)O.shift64 : 0.0f;   // the search's origin: particle or image
            bool accepted = false;
            if (j < C.end && j != O.i && !(asks && isFluid(F.wallBits, j) != fluid)) {
                const float4 A = fetch(&F.pa[j]);
                float pj[3], lj[3], d[3];
                pointIn<D>(A, pj);
                if (coarseDistance2<D>(O.pi, pj, offset) < (FINE && level ? fineLimit : limit)) {
                    const float4 B = D == 3 || FINE ? fetch(&F.pb[j]) : A;
                    remainderIn<D>(A, B, lj);
                    const float r2 = separation2<D>(P, O.pi, O.li, pj, lj, offset, image, O.shift64, d);
                    accepted = r2 < support2(FINE ? 0.5f * (O.hI + fabsf(signedLengthIn<D>(A, B))) : P.hMax);
                }
            }
            int mine = j;
            if constexpr (kAlone) {
                accepted = accepted && (T == 1 || counted++ % T == O.t);
            } else if constexpr (T > 1) {
                // the accepted candidate whose count is this lane's turn, if there is one among these
                unsigned bits = (__ballot_sync(group, accepted) & group) >> lane;
                const int turn = (O.t - counted) & (T - 1);
                counted += __popc(bits);
                for (int q = 0; q < turn; ++q) bits &= bits - 1u;
                accepted = bits != 0;
                mine = base + __ffs(bits) - 1;
            }
            base += W;
            if (!accepted) continue;
            entry = image ? (mine | (int)0x80000000) : mine;
            if (!holds) {
                held = entry;
                holds = true;
                continue;
            }
        } else if (!holds) {
            return;
        }
        NeighbourRows R0, R1;
        loadRows<D, FINE, Visitor>(F, held & 0x7FFFFFFF, R0);
        loadRows<D, FINE, Visitor>(F, entry & 0x7FFFFFFF, R1);
        visitBoth<D, -1, FINE, KIND>(P, O, held, entry, !ended, R0, R1, visit);
        if (ended) return;
        holds = false;
    }
}

}  // namespace sph

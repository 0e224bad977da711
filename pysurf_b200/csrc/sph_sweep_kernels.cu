// sph_sweep_kernels.cu -- the neighbour sweeps of the delta-SPH step.
//
//   list  the step's neighbour table, from one walk over the cells
//   S     Shepard filter (src/pysurf/sphGpu.py:768-802, 1040-1056)
//   A     wall pressure: boundary rows over fluid neighbours (src/pysurf/sphSolver.py:1045-1106;
//         src/pysurf/sphGpu.py:804-854)
//   B     gradients: fluid rows, velocity gradient G (src/pysurf/sphSolver.py:1151-1190), correction L
//         (656-689) and renormalized density gradient (691-716), from one pass over the neighbours
//   C     momentum: fluid rows (src/pysurf/sphSolver.py:1122-1149, 1192-1230, 1328-1356;
//         src/pysurf/sphGpu.py:303-414), with the fluid maxima (1072-1082) and the time step
//         (src/pysurf/sphSolver.py:1410-1424) in the epilogue
//   D     continuity (src/pysurf/sphSolver.py:623-654, 718-822; src/pysurf/sphGpu.py:430-545), with
//         the density update (1111-1140), and, when XSPH is off, the drift and the enforcement
//   X     XSPH (src/pysurf/sphSolver.py:1358-1377; src/pysurf/sphGpu.py:725-766), then drift and
//         enforcement
//
// Each sweep is templated on the dimension D, the kernel K (0 cubic spline, 1 Wendland C2) and
// the threads per particle T.  Sums are float32 in a fixed order, no atomics on them.
#include <cfloat>
#include <climits>
#include <math.h>

#include "sph_enforce.cuh"
#include "sph_kernels.h"
#include "sph_step.cuh"
#include "sph_sweeps.cuh"

namespace sph {

// Resident blocks of 128 threads an SM each sweep is built for, which caps its registers (sweepMinBlocks()
// for the others).  A sweep holds two neighbours' rows, and the next two's in flight, so it wants 90 to 160
// registers.  ms on the 64-ppd beach (2D) and the 20-ppd ridge (3D):
// the energy budget's sweeps, which carry more sums: 4 (3D momentum and continuity on the 8-ppd ridge 1.03 and
// 1.37 ms against 1.25 and 1.61 at 3)
template <int D>
constexpr int budgetMinBlocks() { return 4; }
// continuity: 5 in 2D (0.058, 0.066 at 4; sweepMinBlocks() says why not 6), 4 in 3D (18.3, 22.3 at 3, 30.3 at
// 5)
template <int D>
constexpr int preciseMinBlocks() { return D == 2 ? 5 : 4; }
// gradients: 5 in 2D (0.056, 0.062 at 6), 3 in 3D (15.1, 24.2 at 4)
template <int D>
constexpr int gradientMinBlocks() { return D == 2 ? 5 : 3; }

// the filter and the wall pressure, of few sums: 7 in 2D, 6 in 3D (0.25 ms for the wall pressure on the 10-ppd
// ridge against 0.28 at 5)
template <int D>
constexpr int lightMinBlocks() { return D == 2 ? 7 : 6; }

// ------------------------------------------------------------------------------------------
// The neighbour table
// ------------------------------------------------------------------------------------------

#ifndef SPH_LIST_TRIM
#define SPH_LIST_TRIM 1
#endif

// Each slot's neighbours in the walk's order (sumPairs', with its tests), from a group of
// L lanes: lane t tests candidates t, t + L, ... of each run of the stencil, and the group's ballot
// places the accepted ones in order.  The count is the whole count even when the row is full (the
// sweeps then walk the cells for that slot).  maxCount: the largest count, when given.
//
// A stencil row is trimmed to the cells within the search's reach of the particle, taken in cell
// units from the particle's place in its cell (a particle outside the grid, whose cell is clamped,
// searches its whole stencil).  The reach carries slack over the coarse test's bound, so every
// candidate the coarse test passes stays: the accepted neighbours and their order are those of the
// whole stencil.  PRECISE: separations from point and remainder; MIXED: smoothing lengths differ.
//
// Bound by the instructions it issues (74-79% of the issue slots): eight lanes repeat a slot's set-up for its
// about 150 candidates, so that has no division (the cell's place by one integer quotient, the reach by the
// grid's reciprocal width), and 2D has no search of an image.  Sort and table on the 114,000-particle beach
// 0.114 -> 0.107 ms; 0.106 at 11 blocks an SM (40 registers, no spill) in place of 10.
template <int D, int L, bool PRECISE, bool MIXED>
__global__ void __launch_bounds__(kBlock, D == 2 && !MIXED ? 11 : 1) listKernel(Params P, Frame F, const Control *ctl, int *maxCount)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    const Group<L> G = groupOf<L>();
    const int i = G.i;
    if (i >= P.n) return;           // a group's lanes share i, so groups leave whole
    const int t = G.t;
    const int shift = (threadIdx.x & 31) & ~(L - 1);
    const unsigned lower = G.mask & ((1u << (threadIdx.x & 31)) - 1u);
    const float4 Ai = fetch(&F.pa[i]), Bi = fetch(&F.pb[i]);
    const float hI = fabsf(signedLengthIn<D>(Ai, Bi));
    // a boundary row holds its fluid neighbours only (Row says why)
    const bool fluidOnly = signedLengthIn<D>(Ai, Bi) <= 0.0f;
    float pi[3], li[3];
    pointIn<D>(Ai, pi);
    remainderIn<D>(Ai, Bi, li);
    const float reach = MIXED ? hI + P.hMax : 2.0f * P.hMax;
    const float limit = kCandidateMargin * reach * reach;
    const float support = MIXED ? 0.0f : support2(P.hMax);
    const float sure = PRECISE ? sureBound(P, support, hI, pi) : 0.0f;
    double shift64 = 0.0;
    bool seam = false;
    if (D == 3 && P.period > 0.0 && (pi[1] < reach || pi[1] > P.periodF - reach)) {
        seam = true;
        shift64 = pi[1] < 0.5f * P.periodF ? P.period : -P.period;
    }
    const int ownCell = F.cell[i];
    const float fineReach = hI + P.fineMax, fineLimit = kCandidateMargin * fineReach * fineReach;
    int *column = F.nbr + 4 * (size_t)i;
    int count = 0, wallCount = 0;
    // search s: grid level s >> 1 (coarse, fine), origin s & 1 (the particle, its periodic image)
    for (int search = 0; search < (MIXED ? 4 : 2); search += D == 2 ? 2 : 1) {
        const int level = MIXED ? search >> 1 : 0, image = D == 3 ? search & 1 : 0;
        if (level >= P.levels || (image && !seam)) continue;
        const double pos[3] = {(double)pi[0] + (double)li[0], (double)pi[1] + (double)li[1] + (image ? shift64 : 0.0),
                               D == 3 ? (double)pi[2] + (double)li[2] : 0.0};
        const CellBox box = cellBox(P, level, ownCell, pos, image != 0, D, searchCells(P, level, hI), !MIXED);
        const float searchLimit = level ? fineLimit : limit;
        const double perWidth = level ? P.perFine : P.perCell;
        const double *origin = level ? P.fineOrigin : P.origin;
        // the particle's place in the centre cell, in cell widths, and the reach in cell widths with slack
        const float fx = (float)(((double)pi[0] - origin[0]) * perWidth - box.cx);
        const float fz = D == 3 ? (float)(((double)pi[2] - origin[2]) * perWidth - box.cz) : 0.5f;
        const float R = (1.001f * sqrtf(searchLimit) + 5.0e-7f * (fabsf(pi[0]) + fabsf(pi[1]) + fabsf(pi[2]))) *
                            (float)perWidth + 1.0e-3f;
        const float offset = image ? (float)shift64 : 0.0f;
        const float at[3] = {pi[0], image ? __fadd_rn(pi[1], offset) : pi[1], pi[2]};     // the search's origin
        const float fy = (float)(((double)pi[1] + (image ? shift64 : 0.0) - origin[1]) * perWidth - box.cy);
        const bool trim = SPH_LIST_TRIM && fx >= 0.0f && fx < 1.0f && fy >= 0.0f && fy < 1.0f && fz >= 0.0f &&
                          fz < 1.0f;
        // one run of candidates, L at a time; WALLED: it holds boundary slots
        auto takeRun = [&](auto walled, int first, int end) {
            constexpr bool WALLED = decltype(walled)::value;
            for (int base = first; base < end; base += L) {
                const int j = base + t;
                bool accepted = false, fluidJ = true;
                if (j < end && j != i) {
                    const float4 A = fetch(&F.pa[j]);
                    float pj[3];
                    pointIn<D>(A, pj);
                    if (WALLED) fluidJ = isFluid(F.wallBits, j);
                    const float coarse = !WALLED || fluidJ || !fluidOnly ? coarseDistance2<D>(at, pj) : searchLimit;
                    if (PRECISE && !image && level == 0 && coarse < sure) {
                        accepted = true;
                    } else if (coarse < searchLimit) {
                        const float4 B = (D == 3 && PRECISE) || MIXED ? fetch(&F.pb[j]) : A;
                        float r2 = coarse;      // the float32 points' separation is the coarse one
                        if (PRECISE) {
                            float lj[3], d[3];
                            remainderIn<D>(A, B, lj);
                            r2 = separation2<D, 1>(P, pi, li, pj, lj, offset, image, shift64, d);
                        }
                        const float bound = MIXED ? support2(0.5f * (hI + fabsf(signedLengthIn<D>(A, B)))) : support;
                        accepted = r2 < bound;
                    }
                }
                const bool front = !WALLED || fluidJ || P.together;
                const unsigned bits = __ballot_sync(G.mask, accepted) & G.mask;
                const unsigned walls = WALLED ? __ballot_sync(G.mask, accepted && !front) & G.mask : 0u;
                if (accepted) {
                    const int k = front ? count + __popc(bits & ~walls & lower) : wallCount + __popc(walls & lower);
                    if (k < P.listCap) {
                        const int e = front ? k : P.listCap - 1 - k;
                        column[((size_t)(e >> 2) * P.listStride) * 4 + (e & 3)] = image ? (j | (int)0x80000000) : j;
                    }
                }
                count += __popc(bits & ~walls);
                if (WALLED) wallCount += __popc(walls);
            }
        };
        // lane t takes the run of every L-th stencil row, trimmed; the group then walks the rows in order
        const int across = box.y1 - box.y0 + 1, rows = D == 3 ? across * (box.z1 - box.z0 + 1) : across;
        for (int block = 0; block < rows; block += L) {
            int runFirst = 0, runEnd = 0;
            bool runWalls = false;
            if (block + t < rows) {
                const int zz = D == 3 ? box.z0 + (block + t) / across : 0;
                const int yy = box.y0 + (D == 3 ? (block + t) % across : block + t);
                int xa = box.x0, xb = box.x1;
                bool empty = false;
                if (trim) {
                    const int oz = zz - box.cz, oy = yy - box.cy;
                    const float dz = oz > 0 ? (float)oz - fz : (oz < 0 ? fz - (float)(oz + 1) : 0.0f);
                    const float dy = oy > 0 ? (float)oy - fy : (oy < 0 ? fy - (float)(oy + 1) : 0.0f);
                    const float rem = R * R - dy * dy - dz * dz;
                    empty = rem < 0.0f;
                    const float ext = sqrtf(fmaxf(rem, 0.0f));
                    xa = max(box.x0, box.cx + (int)floorf(fx - ext));
                    xb = min(box.x1, box.cx + (int)floorf(fx + ext));
                }
                if (!empty) {
                    const int row = box.first + (zz * box.ny + yy) * box.nx;
                    runFirst = fetch(&F.cellStart[row + xa]);
                    runEnd = fetch(&F.cellStart[row + xb + 1]);
                    runWalls = runHas(F.wallBits, runFirst, runEnd, true);
                }
            }
            const unsigned walledRows = __ballot_sync(G.mask, runWalls) >> shift;
            const int last = min(L, rows - block);
            for (int q = 0; q < last; ++q) {
                const int first = __shfl_sync(G.mask, runFirst, q, L), end = __shfl_sync(G.mask, runEnd, q, L);
                // most runs hold no boundary slot: their candidates' kinds are not read
                if (walledRows >> q & 1) takeRun(std::true_type{}, first, end);
                else takeRun(std::false_type{}, first, end);
            }
        }
    }
    if (t != 0) return;
    F.ncount[i] = make_int2(count, wallCount);
    if (maxCount) atomicMax(maxCount, count + wallCount);
}

// The same table from a warp that takes a batch of up to kBatch particles of one cell together
// (the 3D table; launchList says why):
// every particle of a cell has the same stencil, so each candidate is loaded once and tested against
// the whole batch, one ballot a particle placing the accepted ones in that particle's order.  Each
// particle accepts only the candidates of its own trimmed run of each row, exactly as listKernel
// (and the sweeps' walk) would offer them, so its row holds the same entries in the same order;
// the union of the batch's runs only decides which candidates the warp loads.
//
// A warp owns the batches that start in its kBatch slots: a batch starts at a cell's first slot and
// every kBatch slots after it, so each slot belongs to one batch.

// A batch member as the warp's lanes read it, in 16-byte rows so that each read is one shared load:
// the run and flags decide whether the member takes a chunk at all, the point its coarse test, the
// remainder only the few candidates near the edge of its support.  The set-up lane writes the
// search's bounds into point.w and rest.w as each search starts.
struct alignas(16) BatchMember {
    float4 point;       // the float32 point; w: this search's sure bound (0 where none applies)
    float4 rest;        // the remainder; w: this search's coarse limit
    float4 bounds;      // the limit on the coarse grid, on the fine grid, the sure bound, hI
    double shift64;     // the periodic image's shift (0 when it is not searched)
    float y;            // point.y before the image's shift, which it takes with one length
    int walls;          // its boundary neighbours so far
};

// Bound by the instructions it issues, most of them a member's test of a candidate.  So a member's point is
// kept as the search sees it (moved across the seam already), and a candidate surely inside or outside the
// support leaves the test without a load of the member's other rows: the 760,000-particle ridge's sort and
// table 3.15 -> 2.86 ms, the refined 11-ppd ridge's 8.55 -> 8.20, the 27,000-particle channel's 0.278 ->
// 0.263.  Two members' distances at a time in packed float32 took 96 registers and 3.7 ms.
// No blocks-a-multiprocessor bound: the compiler's own choice, 64 registers with a few spills at one
// smoothing length, against 3.28 ms at 8 blocks and 4.57 at 1 (118 registers, no spill).
template <int D, int kBatch, bool PRECISE, bool MIXED>
__global__ void __launch_bounds__(kBlock) cellListKernel(Params P, Frame F, const Control *ctl, int *maxCount)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    __shared__ BatchMember members[kBlock / 32][kBatch];
    const int lane = threadIdx.x & 31;
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    BatchMember *mine = members[threadIdx.x >> 5];
    const int first = warp * kBatch;
    if (first >= P.n) return;               // whole warps leave together
    const int last = min(first + kBatch, P.n);
    const float oneReach = 2.0f * P.hMax, oneLimit = kCandidateMargin * oneReach * oneReach;
    const unsigned lower = (1u << lane) - 1u;
    const float support = MIXED ? 0.0f : support2(P.hMax);
    // the batches that start in this warp's slots
    bool starts = false;
    if (lane < kBatch && first + lane < last) {
        const int s = first + lane;
        starts = (s - fetch(&F.cellStart[F.cell[s]])) % kBatch == 0;
    }
    unsigned pending = __ballot_sync(0xFFFFFFFFu, starts);
    while (pending) {
        const int b0 = first + __ffs(pending) - 1;
        pending &= pending - 1;
        const int ownCell = F.cell[b0];
        const int count = min(kBatch, fetch(&F.cellStart[ownCell + 1]) - b0);
        // lane p < count sets up member p
        float hIp = 0.0f, pip[3] = {0, 0, 0}, lip[3] = {0, 0, 0};
        double shiftp = 0.0;
        bool seamp = false, wholeRow = false;
        if (lane < count) {
            const int i = b0 + lane;
            const float4 Ai = fetch(&F.pa[i]), Bi = fetch(&F.pb[i]);
            hIp = fabsf(signedLengthIn<D>(Ai, Bi));
            pointIn<D>(Ai, pip);
            remainderIn<D>(Ai, Bi, lip);
            const float reach = MIXED ? hIp + P.hMax : 2.0f * P.hMax;
            if (D == 3 && P.period > 0.0 && (pip[1] < reach || pip[1] > P.periodF - reach)) {
                seamp = true;
                shiftp = pip[1] < 0.5f * P.periodF ? P.period : -P.period;
            }
            const float fineReach = hIp + P.fineMax;
            BatchMember &m = mine[lane];
            m.point = make_float4(pip[0], pip[1], pip[2], 0.0f);
            m.rest = make_float4(lip[0], lip[1], lip[2], 0.0f);
            m.walls = 0;
            wholeRow = signedLengthIn<D>(Ai, Bi) > 0.0f;
            m.bounds = make_float4(kCandidateMargin * reach * reach, kCandidateMargin * fineReach * fineReach,
                                   PRECISE ? sureBound(P, support, hIp, pip) : 0.0f, hIp);
            m.shift64 = shiftp;
            m.y = pip[1];
        }
        const bool anySeam = __any_sync(0xFFFFFFFFu, seamp);
        // the members that take boundary neighbours: a boundary member's row holds fluid neighbours only
        const unsigned wholeRows = __ballot_sync(0xFFFFFFFFu, wholeRow);
        int counted[kBatch];    // each member's fluid neighbours so far
#pragma unroll
        for (int p = 0; p < kBatch; ++p) counted[p] = 0;
        // search s: grid level s >> 1 (coarse, fine), origin s & 1 (the particle, its periodic image)
        for (int search = 0; search < (MIXED ? 4 : 2); ++search) {
            const int level = MIXED ? search >> 1 : 0, image = search & 1;
            if (level >= P.levels || (image && !anySeam)) continue;
            // lane p: this search's bounds for the others, its own box, its place in the centre cell,
            // and its reach in cell widths
            const bool takes = lane < count && (!image || seamp);
            CellBox box{};
            float fx = 0.0f, fy = 0.0f, fz = 0.0f, R = 0.0f;
            bool trim = false;
            if (lane < count) {
                const float4 bounds = mine[lane].bounds;
                const float lim = level ? bounds.y : bounds.x;
                mine[lane].point.w = PRECISE && !image && level == 0 ? bounds.z : 0.0f;
                mine[lane].rest.w = lim;
                if (!MIXED && image) mine[lane].point.y = __fadd_rn(pip[1], (float)shiftp);
                if (takes) {
                    const double pos[3] = {(double)pip[0] + (double)lip[0],
                                           (double)pip[1] + (double)lip[1] + (image ? shiftp : 0.0),
                                           D == 3 ? (double)pip[2] + (double)lip[2] : 0.0};
                    box = cellBox(P, level, ownCell, pos, image != 0, D, searchCells(P, level, hIp), !MIXED);
                    const double width = level ? P.fineWidth : P.cellWidth, perWidth = level ? P.perFine : P.perCell;
                    const double *origin = level ? P.fineOrigin : P.origin;
                    // A place in a cell, by the reciprocal where lengths differ (the refined 11-ppd ridge's
                    // table 9.34 -> 8.55 ms).  With one length the compiler fits the division's form in 64
                    // registers and the reciprocal's in 72 (the 10-ppd ridge's table 3.15 ms against 3.31).
                    auto placed = [&](double x, int cell) {
                        return MIXED ? (float)(x * perWidth - cell) : (float)(x / width) - (float)cell;
                    };
                    fx = placed((double)pip[0] - origin[0], box.cx);
                    fz = D == 3 ? placed((double)pip[2] - origin[2], box.cz) : 0.5f;
                    fy = placed((double)pip[1] + (image ? shiftp : 0.0) - origin[1], box.cy);
                    R = (1.001f * sqrtf(lim) + 5.0e-7f * (fabsf(pip[0]) + fabsf(pip[1]) + fabsf(pip[2]))) *
                            (MIXED ? (float)perWidth : (float)(1.0 / width)) + 1.0e-3f;
                    trim = SPH_LIST_TRIM && fx >= 0.0f && fx < 1.0f && fy >= 0.0f && fy < 1.0f && fz >= 0.0f &&
                           fz < 1.0f;
                }
            }
            // the grid's shape (the same for every member) and the union of the members' rows
            const int gridFirst = level ? P.fineFirst : 0;
            const int nx = level ? P.fineNc[0] : P.nc[0], ny = level ? P.fineNc[1] : P.nc[1];
            const int zLo = __reduce_min_sync(0xFFFFFFFFu, takes ? box.z0 : INT_MAX);
            const int zHi = __reduce_max_sync(0xFFFFFFFFu, takes ? box.z1 : INT_MIN);
            const int yLo = __reduce_min_sync(0xFFFFFFFFu, takes ? box.y0 : INT_MAX);
            const int yHi = __reduce_max_sync(0xFFFFFFFFu, takes ? box.y1 : INT_MIN);
            __syncwarp();
            for (int zz = zLo; zz <= zHi; ++zz) {
                for (int yy = yLo; yy <= yHi; ++yy) {
                    const int row = gridFirst + (zz * ny + yy) * nx;
                    // lane p: its run of this row, trimmed to its reach
                    int a = 0, b = 0;
                    if (takes && zz >= box.z0 && zz <= box.z1 && yy >= box.y0 && yy <= box.y1) {
                        int xa = box.x0, xb = box.x1;
                        bool empty = false;
                        if (trim) {
                            const int oz = zz - box.cz, oy = yy - box.cy;
                            const float dz = oz > 0 ? (float)oz - fz : (oz < 0 ? fz - (float)(oz + 1) : 0.0f);
                            const float dy = oy > 0 ? (float)oy - fy : (oy < 0 ? fy - (float)(oy + 1) : 0.0f);
                            const float rem = R * R - dy * dy - dz * dz;
                            if (rem < 0.0f) {
                                empty = true;
                            } else {
                                const float ext = sqrtf(rem);
                                xa = max(box.x0, box.cx + (int)floorf(fx - ext));
                                xb = min(box.x1, box.cx + (int)floorf(fx + ext));
                            }
                        }
                        if (!empty) {
                            a = fetch(&F.cellStart[row + xa]);
                            b = fetch(&F.cellStart[row + xb + 1]);
                        }
                    }
                    const int uA = __reduce_min_sync(0xFFFFFFFFu, a < b ? a : INT_MAX);
                    const int uB = __reduce_max_sync(0xFFFFFFFFu, a < b ? b : INT_MIN);
                    for (int base = uA; base < uB; base += 32) {
                        // the members whose own run meets this chunk; a candidate of another member's run
                        // lies past this one's reach, and its distance turns it away
                        const unsigned takers = __ballot_sync(0xFFFFFFFFu, a < b && a < base + 32 && b > base);
                        const int j = base + lane;
                        float4 A = make_float4(0, 0, 0, 0), B = A;
                        float pj[3] = {0, 0, 0}, lj[3] = {0, 0, 0}, hJ = 0.0f;
                        bool fluidJ = true;
                        unsigned offered = 0;       // the members this candidate is offered to
                        if (j < uB) {
                            A = fetch(&F.pa[j]);
                            pointIn<D>(A, pj);
                            // the remainders with the point, although a candidate under `sure` needs
                            // none: loading them only for the precise test slowed the 3D table by 11%
                            if ((D == 3 && PRECISE) || MIXED) B = fetch(&F.pb[j]);
                            if (PRECISE) remainderIn<D>(A, D == 3 ? B : A, lj);
                            if (MIXED) hJ = fabsf(signedLengthIn<D>(A, B));
                            fluidJ = D == 3 ? A.w > 0.0f : fetch(&F.fluid[j]) != 0;
                            offered = fluidJ ? 0xFFFFFFFFu : wholeRows;
                            if (j >= b0 && j < b0 + kBatch) offered &= ~(1u << (j - b0));      // not to itself
                        }
                        const bool front = fluidJ || P.together;
                        const unsigned fronts = __ballot_sync(0xFFFFFFFFu, front);
                        const int entry = image ? (j | (int)0x80000000) : j;
#pragma unroll
                        for (int p = 0; p < kBatch; ++p) {
                            if (!(takers >> p & 1)) continue;       // the whole warp
                            const float4 point = mine[p].point;
                            const float mp[3] = {point.x, point.y, point.z};
                            const float coarse = MIXED ? coarseDistance2<D>(mp, pj, image ? (float)mine[p].shift64 : 0.0f)
                                                       : coarseDistance2<D>(mp, pj);
                            const bool offer = offered >> p & 1;
                            bool accepted = PRECISE && offer && coarse < point.w;
                            // With one length the search's limit is every member's, so that the whole warp
                            // passes over this but for a candidate near the edge of the support.
                            if (offer && !accepted && (MIXED || coarse < oneLimit)) {
                                const float4 rest = mine[p].rest;
                                if (!MIXED || coarse < rest.w) {
                                    float r2 = coarse;
                                    if (PRECISE) {
                                        const float own[3] = {point.x, !MIXED && image ? mine[p].y : point.y, point.z};
                                        const float ml[3] = {rest.x, rest.y, rest.z};
                                        float d[3];
                                        r2 = separation2<D, 1>(P, own, ml, pj, lj, 0.0f, image,
                                                               image ? mine[p].shift64 : 0.0, d);
                                    }
                                    const float bound = MIXED ? support2(0.5f * (mine[p].bounds.w + hJ)) : support;
                                    accepted = r2 < bound;
                                }
                            }
                            const unsigned bits = __ballot_sync(0xFFFFFFFFu, accepted);
                            const unsigned got = bits & fronts, walls = bits & ~fronts;
                            int *column = F.nbr + 4 * (size_t)(b0 + p);
                            if (accepted && front) {
                                const int k = counted[p] + __popc(got & lower);
                                if (k < P.listCap) column[((size_t)(k >> 2) * P.listStride) * 4 + (k & 3)] = entry;
                            }
                            counted[p] += __popc(got);
                            if (walls) {        // the whole warp
                                const int before = mine[p].walls;
                                if (accepted && !front) {
                                    const int w = before + __popc(walls & lower), e = P.listCap - 1 - w;
                                    if (w < P.listCap) column[((size_t)(e >> 2) * P.listStride) * 4 + (e & 3)] = entry;
                                }
                                __syncwarp();
                                if (lane == 0) mine[p].walls = before + __popc(walls);
                                __syncwarp();
                            }
                        }
                    }
                }
            }
            __syncwarp();
        }
        int2 own = make_int2(0, 0);
#pragma unroll
        for (int p = 0; p < kBatch; ++p)
            if (lane == p) own = make_int2(counted[p], mine[p].walls);
        if (lane < count) {
            F.ncount[b0 + lane] = own;
            if (maxCount) atomicMax(maxCount, own.x + own.y);
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------
// Sweep S: the Shepard filter
// ------------------------------------------------------------------------------------------

template <int D, int K, bool FINE>
struct ShepardVisit {
    static constexpr bool kBody = true, kKinetic = D == 2, kAux = true, kLow = false, kMass = false;
    static constexpr bool kSkipCoincident = false;
    Smoothing<K, D, FINE> S;
    float num, den;
    __device__ void operator()(int, const float *, float r, float, const KernelAt &k, const NeighbourRows &R)
    {
        const float w = kernelValue<K>(__fmul_rn(r, k.invH), k);
        num = __fmaf_rn(massIn<D>(R), w, num);
        den = __fmaf_rn(volumeIn<D>(R), w, den);
    }
};

template <int D, int K, int T, bool FINE>
__global__ void __launch_bounds__(kBlock, lightMinBlocks<D>()) shepardKernel(Params P, Frame F, const Control *ctl)
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
    float hI = fabsf(hs);
    // the particle itself first, as the reference's sums start (src/pysurf/sphGpu.py:781-783)
    float own = sigmaAt(P.sigmaUnit, hI, D);
    float mi = massOf<D>(F, i);
    ShepardVisit<D, K, FINE> visit{Smoothing<K, D, FINE>(P, hI), G.t == 0 ? mi * own : 0.0f,
                             G.t == 0 ? volumeOf<D>(F, i) * own : 0.0f};
    // the host-step call returns boundary rows too, over all their neighbours, which the table does not hold
    const Row row = openRow<D, FINE>(P, F, i, G.t, hI, hs <= 0.0f);
    sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, visit);
    sumPairs<D, T, FINE, kWallPair>(P, F, row, false, visit);
    float num = groupSum<T>(visit.num, G.mask), den = groupSum<T>(visit.den, G.mask);
    if (G.t != 0) return;
    F.scalar[i] = num / den;
}

// The fluid takes its filtered density (float64 from the float32 filter, as the reference
// stores it), its deviation and its pressure; the boundary keeps its own.
template <int D>
__global__ void applyShepardKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    if (!filterDue(ctl)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n || !F.fluid[i]) return;
    float filtered = F.scalar[i];
    double rho = (double)filtered;
    // the filter's change of elastic energy (src/pysurf/sphGpu.py:1043-1056)
    if (P.budget) addEnergy(P, F, i, kFilter, F.m[i] * (elasticEnergy(P, rho) - elasticEnergy(P, F.rho[i])));
    F.rho[i] = rho;
    storeDensity<D>(F, i, massOf<D>(F, i), rho, P.devReference, (float)taitPressure(P, rho, true));
}

// ------------------------------------------------------------------------------------------
// Sweep A: extrapolated wall pressure
// ------------------------------------------------------------------------------------------

template <int D, int K, bool FINE>
struct WallVisit {
    static constexpr bool kBody = true, kKinetic = false, kAux = true, kLow = false, kMass = false;
    static constexpr bool kSkipCoincident = false;
    const Params &P; const Frame &F;
    Smoothing<K, D, FINE> S;
    float weight, total;
    __device__ void operator()(int j, const float *d, float r, float, const KernelAt &k, const NeighbourRows &R)
    {
        const float w = kernelValue<K>(__fmul_rn(r, k.invH), k);
        float gd = __fmaf_rn(P.g[1], d[1], __fmul_rn(P.g[0], d[0]));
        if (D == 3) gd = __fmaf_rn(P.g[2], d[2], gd);
        weight = __fadd_rn(weight, w);
        total = __fmaf_rn(w, __fmaf_rn(densityIn<D>(R), gd, pressureOf<D>(F, j)), total);
    }
};

// Boundary rows only write their own entries and only fluid entries are read, so the frame is
// updated in place.  writeDensity: the master float64 density takes Tait^-1(p_w) too.
template <int D, int K, int T, bool FINE>
__global__ void __launch_bounds__(kBlock, lightMinBlocks<D>())
wallPressureKernel(Params P, Frame F, const Control *ctl, int writeDensity)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(const_cast<Control *>(ctl), P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    float hs = signedLength<D>(F, i);
    if (hs > 0.0f) return;
    WallVisit<D, K, FINE> visit{P, F, Smoothing<K, D, FINE>(P, -hs), 0.0f, 0.0f};
    sumPairs<D, T, FINE, kCrossPair>(P, F, openRow<D, FINE>(P, F, i, G.t, -hs), true, visit);
    float weight = groupSum<T>(visit.weight, G.mask), total = groupSum<T>(visit.total, G.mask);
    if (G.t != 0) return;
    float p = 0.0f;
    if (weight > 0.0f) p = fmaxf(total / weight, 0.0f);
    F.scalar[i] = p;
    if (writeDensity) {
        double rho = P.rho0 * pow(1.0 + (double)p / P.stiffness, 1.0 / 7.0);
        storeDensity<D>(F, i, massOf<D>(F, i), rho, P.devReference, p);
        F.rho[i] = rho;
        return;
    }
    // the density stays; the pressure and p / rho^2 take p_w
    const float rho = densityOf<D>(F, i), ratio = p / (rho * rho);
    F.pres[i] = p;
    if (D == 2) F.pb[i].z = ratio;
    else F.aux[i].x = ratio;
}

// ------------------------------------------------------------------------------------------
// Sweep B: G, L and grad rho from one pass
// ------------------------------------------------------------------------------------------

// M (for L) is summed in float64 from float64 kernel gradients: L multiplies continuity's cancelling
// terms (a wall's velocity jump), where an L off by float32's summation error would move the rate by
// more than 1e-5 of its largest value against the float64 sums.  Its upper triangle, packed.
template <int D>
__device__ __forceinline__ constexpr int packed(int a, int b) { return a * D - a * (a - 1) / 2 + (b - a); }

template <int D, int K, bool FINE, bool RHO, bool TABLED>
struct GradientVisit {
    static constexpr bool kAlone = TABLED;
    static constexpr bool kBody = false, kKinetic = true, kAux = false, kLow = false, kMass = false;
    static constexpr bool kPaired = true;
    static constexpr bool kSkipCoincident = true;
    Smoothing<K, D, FINE> S;
    bool wantG, wantL;
    float vi[3], devI;
    // each lane's sums over its even and its odd neighbours: V (v_j - v_i) grad W, and M over the fluid
    // (its upper triangle, packed)
    float2 jump[D][D], Mf[D * (D + 1) / 2], gsum[RHO ? D : 1];   // gsum: RHO, the density gradient's sum
    double M[D * (D + 1) / 2];
    struct Taken {
        float volume[2];
        float2 rel[D], difference;      // v_j - v_i, the deviations' difference
    };
    template <PairKind KIND>
    __device__ __forceinline__ Taken take(const Neighbours &, const NeighbourRows &R0, const NeighbourRows &R1) const
    {
        Taken t;
        t.volume[0] = volumeIn<D>(R0);
        t.volume[1] = volumeIn<D>(R1);
        float vj0[3], vj1[3];
        velocityIn<D>(R0.K, vj0);
        velocityIn<D>(R1.K, vj1);
        if (KIND == kFluidPair)
            for (int a = 0; a < D; ++a) t.rel[a] = make_float2(__fsub_rn(vj0[a], vi[a]), __fsub_rn(vj1[a], vi[a]));
        t.difference = make_float2(__fsub_rn(deviationIn<D>(R0), devI), __fsub_rn(deviationIn<D>(R1), devI));
        return t;
    }
    template <PairKind KIND>
    __device__ __forceinline__ void finish(const Neighbours &N, const Taken &taken)
    {
        const float *volume = taken.volume;
        if (wantL) {
            for (int q = 0; q < 2; ++q) {
                if (!N.live[q]) continue;
                double dd[3], r2 = 0.0;
                for (int a = 0; a < D; ++a) {
                    dd[a] = (double)(q ? N.d[a].y : N.d[a].x);
                    r2 = fma(dd[a], dd[a], r2);
                }
                const double rr = preciseRoot(r2, q ? N.inverse.y : N.inverse.x);
                const double w64 = (double)volume[q] * kernelGradient64<K>(rr, N.k.of(q));
                for (int a = 0; a < D; ++a) {
                    const double wa = -w64 * dd[a];
                    for (int b = a; b < D; ++b) M[packed<D>(a, b)] = fma(wa, dd[b], M[packed<D>(a, b)]);
                }
            }
        }
        const float2 grad = kernelGradient<K>(mul2(N.r, N.k.invH), N.k);
        const float2 w = make_float2(N.live[0] ? __fmul_rn(volume[0], grad.x) : 0.0f,
                                     N.live[1] ? __fmul_rn(volume[1], grad.y) : 0.0f);
        if (KIND == kFluidPair && wantG) {
            for (int a = 0; a < D; ++a) {
                const float2 wv = mul2(w, taken.rel[a]);
                for (int b = 0; b < D; ++b) jump[a][b] = fma2(wv, N.d[b], jump[a][b]);
                const float2 wa = mul2(w, N.d[a]);     // minus M's weight; the sign comes off at the end
                for (int b = a; b < D; ++b) Mf[packed<D>(a, b)] = fma2(wa, N.d[b], Mf[packed<D>(a, b)]);
            }
        }
        if (RHO) {
            const float2 t = mul2(w, taken.difference);
            for (int a = 0; a < D; ++a) gsum[RHO ? a : 0] = fma2(t, N.d[a], gsum[RHO ? a : 0]);
        }
    }
};

// A lane's two halves and then the group's sum.
template <int T>
__device__ __forceinline__ float groupSum(const float2 &value, unsigned mask)
{
    return groupSum<T>(__fadd_rn(value.x, value.y), mask);
}

// TABLED: few rows walk (LaunchArgs::tabled), in 3D with one smoothing length; sumPairs() says why.
template <int D, int K, int T, bool FINE, bool RHO, bool TABLED>
__global__ void __launch_bounds__(kBlock, gradientMinBlocks<D>())
gradientKernel(Params P, Frame F, const Control *ctl, int wantG, int wantL, float floorDet)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(const_cast<Control *>(ctl), P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    float hs = signedLength<D>(F, i);
    if (hs <= 0.0f) {
        if (G.t != 0) return;
        float zero[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        float ident[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
        if (wantG == kWholeGradients) storeMatrix<D>(F.G0, F.G1, F.G2, i, zero);
        if (wantL) storeMatrix<D>(F.L0, F.L1, F.L2, i, ident);
        if (RHO) F.gradRho[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    GradientVisit<D, K, FINE, RHO, TABLED> visit{Smoothing<K, D, FINE>(P, hs), wantG != 0, wantL != 0 || RHO};
    velocityOf<D>(F, i, visit.vi);
    visit.devI = deviationOf<D>(F, i);
    for (int a = 0; a < D; ++a) {
        visit.gsum[RHO ? a : 0] = both(0.0f);
        for (int b = 0; b < D; ++b) visit.jump[a][b] = both(0.0f);
    }
    for (int q = 0; q < D * (D + 1) / 2; ++q) { visit.M[q] = 0.0; visit.Mf[q] = both(0.0f); }
    const Row row = openRow<D, FINE>(P, F, i, G.t, hs);
    sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, visit);
    if (visit.wantL) sumPairs<D, T, FINE, kWallPair>(P, F, row, false, visit);
    float Mf[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, jump[3][3] = {}, gsum[3] = {};
    if (wantG) {
        for (int a = 0; a < D; ++a) {
            for (int b = 0; b < D; ++b) jump[a][b] = groupSum<T>(visit.jump[a][b], G.mask);
            for (int b = a; b < D; ++b) Mf[a][b] = Mf[b][a] = -groupSum<T>(visit.Mf[packed<D>(a, b)], G.mask);
        }
    }
    double M[3][3] = {{1.0, 0.0, 0.0}, {0.0, 1.0, 0.0}, {0.0, 0.0, 1.0}};
    if (wantL || RHO)
        for (int a = 0; a < D; ++a)
            for (int b = a; b < D; ++b) M[a][b] = M[b][a] = groupSum<T>(visit.M[packed<D>(a, b)], G.mask);
    if (RHO)
        for (int a = 0; a < D; ++a) gsum[a] = groupSum<T>(visit.gsum[RHO ? a : 0], G.mask);
    if (G.t != 0) return;
    if (wantG) {
        float Gm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        if (determinant<D>(Mf) >= floorDet) {
            float inv[3][3];
            inverse<D>(Mf, inv);
            for (int a = 0; a < D; ++a)
                for (int b = 0; b < D; ++b) {
                    float t = 0.0f;
                    for (int c = 0; c < D; ++c) t += jump[a][c] * inv[c][b];
                    Gm[a][b] = t;
                }
        }
        // the steps read the symmetric part alone; the whole matrix goes to the caller who asks for it
        if (wantG == kWholeGradients) storeMatrix<D>(F.G0, F.G1, F.G2, i, Gm);
        else storeSlopes<D>(F, i, Gm);
    }
    if (wantL || RHO) {
        // L = M^-1 in float64, rounded once
        float L[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
        if (determinant<D>(M) >= (double)floorDet) {
            double inv[3][3];
            inverse<D>(M, inv);
            for (int a = 0; a < D; ++a)
                for (int b = 0; b < D; ++b) L[a][b] = (float)inv[a][b];
        }
        if (wantL) storeMatrix<D>(F.L0, F.L1, F.L2, i, L);
        if (RHO) {
            float g[3] = {0.0f, 0.0f, 0.0f};
            for (int a = 0; a < D; ++a)
                for (int b = 0; b < D; ++b) g[a] += L[a][b] * gsum[b];
            F.gradRho[i] = make_float4(g[0], g[1], g[2], 0.0f);
        }
    }
}

// ------------------------------------------------------------------------------------------
// Sweep C: accelerations, fluid maxima, time step
// ------------------------------------------------------------------------------------------

// What the viscosity is multiplied by until it joins the pressure, so that quickDivide, which takes and
// leaves no subnormal, loses none.
constexpr float kViscosityScale = 4294967296.0f;

// BUDGET: the sum split for the energy budget too, into the pressure and the viscosity of fluid
// and of boundary neighbours (src/pysurf/sphGpu.py:400-414).  COMP: the sum compensated (Dot2),
// its running error in comp.
template <int D, int K, bool BUDGET, bool FINE, bool COMP, bool CLOSURE>
struct MomentumVisit {
    static constexpr bool kBody = true, kKinetic = true, kAux = true, kLow = false, kMass = false;
    static constexpr bool kPaired = true;
    static constexpr bool kSkipCoincident = true;
    const Params &P; const Frame &F;
    Smoothing<K, D, FINE> S;
    float vi[3], rhoI, own, viscosityScale;   // viscosityScale: -alpha c0 kViscosityScale
    float alphaI;                               // closure: this particle's eddy alpha
    float slopeI[6];                            // r . G_i r's coefficients (Frame::S0, S1)
    float2 total[D];                            // minus the sum, over the lane's even and odd neighbours
    float2 comp[COMP ? D : 1];
    float parts[BUDGET ? 4 : 1][3];
    struct Taken {
        float2 plain;               // (v_i - v_j) . r
        float2 density, pressure;   // rho_i + rho_j, p_i / rho_i^2 + p_j / rho_j^2
        float mass[2], rho[2];
        float s0[6], s1[6];         // the approaching neighbours' slopes' coefficients
    };
    template <PairKind KIND>
    __device__ __forceinline__ Taken take(const Neighbours &N, const NeighbourRows &R0, const NeighbourRows &R1) const
    {
        Taken t;
        float vj0[3], vj1[3];
        velocityIn<D>(R0.K, vj0);
        velocityIn<D>(R1.K, vj1);
        for (int a = 0; a < D; ++a) {
            const float2 rel = make_float2(__fsub_rn(vi[a], vj0[a]), __fsub_rn(vi[a], vj1[a]));
            t.plain = a == 0 ? mul2(rel, N.d[0]) : fma2(rel, N.d[a], t.plain);
        }
        for (int c = 0; c < 6; ++c) t.s0[c] = t.s1[c] = 0.0f;
        if (KIND == kFluidPair && P.limited) {
            if (t.plain.x < 0.0f) loadSlopes<D>(F, N.j[0], t.s0);
            if (t.plain.y < 0.0f) loadSlopes<D>(F, N.j[1], t.s1);
        }
        t.rho[0] = densityIn<D>(R0);
        t.rho[1] = densityIn<D>(R1);
        t.density = make_float2(__fadd_rn(rhoI, t.rho[0]), __fadd_rn(rhoI, t.rho[1]));
        t.pressure = make_float2(__fadd_rn(own, pressureRatioIn<D>(R0)),
                                 __fadd_rn(own, pressureRatioIn<D>(R1)));
        t.mass[0] = massIn<D>(R0);
        t.mass[1] = massIn<D>(R1);
        return t;
    }
    template <PairKind KIND>
    __device__ __forceinline__ void finish(const Neighbours &N, const Taken &taken)
    {
        const float2 q = mul2(N.r, N.k.invH), grad = kernelGradient<K>(q, N.k);
        const float2 plain = taken.plain;
        const float *s0 = taken.s0, *s1 = taken.s1;
        float2 approach = plain;
        if (KIND == kFluidPair && P.limited) {
            const bool limit0 = plain.x < 0.0f, limit1 = plain.y < 0.0f;
            if (limit0 || limit1) {
                // the slopes r . G r along the pair, each a quadratic form in r: only G's symmetric part
                // enters, so r's products d_a d_b (a <= b) serve both particles
                float2 slopeI2 = both(0.0f), slopeJ = both(0.0f);
                for (int a = 0; a < D; ++a)
                    for (int b = a; b < D; ++b) {
                        const int c = packed<D>(a, b);
                        const float2 dd = mul2(N.d[a], N.d[b]);
                        slopeI2 = fma2(both(slopeI[c]), dd, slopeI2);
                        slopeJ = make_float2(__fmaf_rn(s0[c], dd.x, slopeJ.x), __fmaf_rn(s1[c], dd.y, slopeJ.y));
                    }
                // 4 R / (1 + R)^2 at R = slopeI / slopeJ, as 4 slopeI slopeJ / (slopeI + slopeJ)^2, which is
                // never less than what stands above it; 0 where that has no normal float
                const float2 sum = add2(slopeI2, slopeJ), product = mul2(slopeI2, slopeJ);
                const float2 four = mul2(both(4.0f), product), square = mul2(sum, sum);
                // the fast division takes 8% off the momentum sweep; its range limit (a denominator
                // past 2^126) lies far beyond any pair's slopes, and the scale keeps both sides normal
                float2 limiter = make_float2(four.x >= FLT_MIN ? fminf(1.0f, quickDivide(four.x, square.x)) : 0.0f,
                                             four.y >= FLT_MIN ? fminf(1.0f, quickDivide(four.y, square.y)) : 0.0f);
                if (q.x < kCloseDistance || q.y < kCloseDistance) {
                    const float fade0 = (q.x - kCloseDistance) * (1.0f / kFoldWidth);
                    const float fade1 = (q.y - kCloseDistance) * (1.0f / kFoldWidth);
                    if (q.x < kCloseDistance) limiter.x = __fmul_rn(limiter.x, expf(-__fmul_rn(fade0, fade0)));
                    if (q.y < kCloseDistance) limiter.y = __fmul_rn(limiter.y, expf(-__fmul_rn(fade1, fade1)));
                }
                // (v_ij - (phi / 2) (G_i + G_j) r) . r = v_ij . r - (phi / 2) (r . G_i r + r . G_j r)
                const float2 limited = fma2(mul2(both(-0.5f / kSlopeScale), limiter), sum, plain);
                if (limit0) approach.x = limited.x;
                if (limit1) approach.y = limited.y;
            }
        }
        // -alpha c0 h (v_ij . r_ij) / ((r^2 + 0.01 h^2) (rho_i + rho_j) / 2) where the pair approaches, times
        // kViscosityScale; the denominator is a positive normal float for any physical pair
        const float2 closing = make_float2(fminf(approach.x, 0.0f), fminf(approach.y, 0.0f));
        const float2 above = mul2(mul2(both(viscosityScale), N.h), closing);
        const float2 mean = mul2(both(0.5f), taken.density);
        const float2 below = mul2(fma2(N.r, N.r, N.k.soft), mean);
        float2 viscosity = make_float2(quickDivide(above.x, below.x), quickDivide(above.y, below.y));
        if (KIND == kWallPair) viscosity = mul2(viscosity, both(P.boundaryFactor));
        const float2 pressure = taken.pressure;
        float2 stress;
        if (KIND == kFluidPair && CLOSURE && P.closure) {
            viscosity = mul2(viscosity, both(1.0f / kViscosityScale));
            if (N.live[0])
                viscosity.x = __fadd_rn(viscosity.x, closureTerm(N.j[0], N.h.x, N.r.x, plain.x, taken.rho[0]));
            if (N.live[1])
                viscosity.y = __fadd_rn(viscosity.y, closureTerm(N.j[1], N.h.y, N.r.y, plain.y, taken.rho[1]));
            stress = add2(pressure, viscosity);
        } else {
            stress = fma2(viscosity, both(1.0f / kViscosityScale), pressure);
            if (BUDGET) viscosity = mul2(viscosity, both(1.0f / kViscosityScale));
        }
        const float m0 = taken.mass[0], m1 = taken.mass[1];
        const float2 f = mul2(make_float2(N.live[0] ? __fmul_rn(stress.x, m0) : 0.0f,
                                          N.live[1] ? __fmul_rn(stress.y, m1) : 0.0f), grad);
        if constexpr (COMP) {
            for (int a = 0; a < D; ++a) {
                addProduct(f.x, N.d[a].x, total[a].x, comp[a].x);
                addProduct(f.y, N.d[a].y, total[a].y, comp[a].y);
            }
        } else {
            for (int a = 0; a < D; ++a) total[a] = fma2(f, N.d[a], total[a]);
        }
        if constexpr (BUDGET) {
            for (int s = 0; s < 2; ++s) {
                if (!N.live[s]) continue;
                const float weight = __fmul_rn(s ? m1 : m0, s ? grad.y : grad.x);
                const float fp = -__fmul_rn(s ? pressure.y : pressure.x, weight);
                const float fv = -__fmul_rn(s ? viscosity.y : viscosity.x, weight);
                constexpr int side = KIND == kFluidPair ? 0 : 2;
                for (int a = 0; a < D; ++a) {
                    const float d = s ? N.d[a].y : N.d[a].x;
                    parts[BUDGET ? side : 0][a] = __fmaf_rn(fp, d, parts[BUDGET ? side : 0][a]);
                    parts[BUDGET ? side + 1 : 0][a] = __fmaf_rn(fv, d, parts[BUDGET ? side + 1 : 0][a]);
                }
            }
        }
    }
    // delta-LES-SPH: -(K nu / (c0 h) + harmonic mean of the alphas) c0 h rho0 (v_ij . r_ij) /
    // (r^2 rho_i rho_j) on every fluid pair, approaching or not (src/pysurf/sphGpu.py:388-396)
    __device__ __forceinline__ float closureTerm(int j, float h, float r, float plain, float rhoJ) const
    {
        const float alphaJ = fetch(&F.eddy[j].x), sum = __fadd_rn(alphaI, alphaJ);
        const float mean = sum > 0.0f ? __fdiv_rn(__fmul_rn(__fmul_rn(2.0f, alphaI), alphaJ), sum) : 0.0f;
        const float scale = __fmul_rn(__fmul_rn(__fmul_rn(__fadd_rn(__fdiv_rn(P.waterTerm, h), mean), P.c0), h), P.closureRho0);
        return __fdiv_rn(-__fmul_rn(scale, plain), __fmul_rn(__fmul_rn(__fmul_rn(r, r), rhoI), rhoJ));
    }
};

// maxima: fold the fluid maxima into ctl and take the time step (the device steps); 0 for the
// host-step sums.
template <int D, int K, int T, bool BUDGET, bool FINE, bool COMP, bool CLOSURE>
__global__ void __launch_bounds__(kBlock, BUDGET ? budgetMinBlocks<D>() : sweepMinBlocks<D>())
momentumKernel(Params P, Frame F, Control *ctl, int maxima)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(ctl, P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    double speed = 0.0, accel = 0.0;
    if (i < P.n) {
        float hs = signedLength<D>(F, i);
        if (hs <= 0.0f) {
            if (G.t == 0) F.acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            MomentumVisit<D, K, BUDGET, FINE, COMP, CLOSURE> visit{P, F, Smoothing<K, D, FINE>(P, hs)};
            velocityOf<D>(F, i, visit.vi);
            visit.rhoI = densityOf<D>(F, i);
            visit.own = pressureRatioOf<D>(F, i);
            visit.viscosityScale = -P.alpha * P.c0 * kViscosityScale;
            visit.alphaI = CLOSURE && P.closure ? F.eddy[i].x : 0.0f;
            if (P.limited) loadSlopes<D>(F, i, visit.slopeI);
            for (int a = 0; a < D; ++a) visit.total[a] = both(0.0f);
            if constexpr (COMP) for (int a = 0; a < D; ++a) visit.comp[a] = both(0.0f);
            if constexpr (BUDGET)
                for (int q = 0; q < 4; ++q) visit.parts[q][0] = visit.parts[q][1] = visit.parts[q][2] = 0.0f;
            const Row row = openRow<D, FINE>(P, F, i, G.t, hs);
            sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, visit);
            sumPairs<D, T, FINE, kWallPair>(P, F, row, false, visit);
            float total[3] = {0.0f, 0.0f, 0.0f};
            for (int a = 0; a < D; ++a) {
                if constexpr (COMP) total[a] = -groupSumCompensated<T>(visit.total[a], visit.comp[a], G.mask);
                else total[a] = -groupSum<T>(visit.total[a], G.mask);
            }
            if constexpr (BUDGET) {
                for (int q = 0; q < 4; ++q) {
                    for (int a = 0; a < D; ++a) visit.parts[q][a] = groupSum<T>(visit.parts[q][a], G.mask);
                    if (G.t == 0)
                        F.parts[(size_t)q * P.energyStride + i] =
                            make_float4(visit.parts[q][0], visit.parts[q][1], D == 3 ? visit.parts[q][2] : 0.0f, 0.0f);
                }
            }
            if (G.t == 0) {
                takeAcceleration<D>(P, F, i, total, speed, accel);
            }
        }
    }
    if (maxima) foldMaxima(ctl, speed, accel, (int)(gridDim.x * (blockDim.x >> 5)));
}

// The delta-LES-SPH closure's coefficients (src/pysurf/sphGpu.py:699-723): ||D|| = sqrt(2 D:D) of the
// strain D = (G + G^T) / 2, alpha_i = 2 (dim + 2) (C_S l / h)^2 h ||D|| / c0 and
// delta_i = (C_delta l / h)^2 h ||D|| / c0, l = 2 h, C_S 0.12, C_delta 1.5, each at most 0.2;
// zero on the boundary.  G is the gradients sweep's, from this step's starting velocities.
template <int D>
__global__ void closureKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const float hs = signedLength<D>(F, i);
    if (hs <= 0.0f) {
        F.eddy[i] = make_float2(0.0f, 0.0f);
        return;
    }
    float slopes[6];
    loadSlopes<D>(F, i, slopes);
    float sum = 0.0f;
    for (int a = 0; a < D; ++a)
        for (int b = 0; b < D; ++b) {
            const float scaled = a == b ? slopes[packed<D>(a, a)] : 0.5f * slopes[packed<D>(min(a, b), max(a, b))];
            const float e = scaled * (1.0f / kSlopeScale);
            sum += e * e;
        }
    const float scale = hs * sqrtf(2.0f * sum) / P.closureC0;
    constexpr float smagorinsky = (0.12f * 2.0f) * (0.12f * 2.0f), diffusion = (1.5f * 2.0f) * (1.5f * 2.0f);
    F.eddy[i] = make_float2(fminf(2.0f * (D + 2) * smagorinsky * scale, 0.2f), fminf(diffusion * scale, 0.2f));
}

// v += a dt on the fluid (src/pysurf/sphGpu.py:1084-1109); the frame takes the kicked velocity.
template <int D>
__global__ void kickKernel(Params P, Frame F, Control *ctl)
{
    awaitPrevious();
    if (!ctl->active) return;
    stampStages(ctl, P.stages);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n || !F.fluid[i]) return;
    double dt = ctl->dt;
    float4 a = F.acc[i];
    double v[3] = {0.0, 0.0, 0.0}, mean[3] = {0.0, 0.0, 0.0};
    float av[3] = {a.x, a.y, a.z};
    for (int c = 0; c < D; ++c) {
        const double start = F.v[c][i];
        v[c] = start + (double)av[c] * dt;
        F.v[c][i] = v[c];
        mean[c] = 0.5 * (start + v[c]);
    }
    if (P.budget) {
        // each part of a, and gravity, does the work m a . (v + v') / 2 dt (src/pysurf/sphGpu.py:1084-1109)
        const double m = F.m[i];
        for (int q = 0; q < 4; ++q) {
            const float4 part = F.parts[(size_t)q * P.energyStride + i];
            const float pv[3] = {part.x, part.y, part.z};
            double work = 0.0;
            for (int c = 0; c < D; ++c) work += (double)pv[c] * mean[c];
            addEnergy(P, F, i, kPressureFluid + q, m * work * dt);
        }
        double work = 0.0;
        for (int c = 0; c < D; ++c) work += (double)P.g[c] * mean[c];
        addEnergy(P, F, i, kGravityWork, m * work * dt);
    }
    float4 k = F.kin[i], low = F.low[i];
    k.x = (float)v[0]; k.y = (float)v[1];
    low.x = (float)(v[0] - (double)k.x); low.y = (float)(v[1] - (double)k.y);
    if (D == 3) { k.z = (float)v[2]; low.z = (float)(v[2] - (double)k.z); }
    F.kin[i] = k;
    F.low[i] = low;
}

// ------------------------------------------------------------------------------------------
// Sweep D: continuity with the density update, drift and enforcement
// ------------------------------------------------------------------------------------------

// BUDGET: the rate split for the energy budget too: the plain sum over fluid and over boundary
// neighbours, the corrected sum (the correction's part is its difference) and the diffusion
// (src/pysurf/sphGpu.py:476-545).  COMP: the float32 sum compensated (Dot2), its running error in comp.
//
// The rate's terms cancel: next to a wall a particle's velocity jumps to the boundary's zero, and
// sum_j m_j (v_i - v_j) . grad W_ij over a near-symmetric support is a small remainder of large
// terms.  So each term keeps float64's digits where that matters: velocity and deviation differences
// come from the float32 values and their remainders (the frame's low row), and the pairs of a fluid
// and a boundary particle -- every pair of a boundary row, the wall's pairs of a fluid row -- take
// their separation, distance, kernel gradient and term in float64, summed apart in float64 (cross).
// Fluid pairs, whose velocity differences are small, keep float32 arithmetic.
template <int D, int K, bool BUDGET, bool FINE, bool COMP, bool CLOSURE>
struct ContinuityVisit {
    static constexpr bool kBody = false, kKinetic = true, kAux = false, kLow = true, kMass = true;
    static constexpr bool kPaired = true;
    static constexpr bool kSkipCoincident = true;
    const Params &P; const Frame &F;
    Smoothing<K, D, FINE> S;
    bool diffuses, corrected;
    float vi[3], vlI[3], devI, devLoI, Li[3][3], gi[3];
    float deltaI;           // closure: this particle's eddy delta
    float2 total, comp;     // over the lane's even and odd neighbours
    double x[D], v[D];      // the particle's position and velocity in float64
    // the fluid-boundary pairs' sums in float64: m (dW/dr) / r (v_i - v_j)_a (x_i - x_j)_b where L enters
    // (cross[a D + b]), else its trace alone (cross[0])
    double cross[D * D];
    float plainFluid, continuity, diffusive;    // BUDGET: the fluid pairs' parts
    struct Taken {
        float2 dv[D];                       // v_i - v_j
        float mass[2];
        float2 volume, devJ, leading, remainder;    // V_j; rho_j - rho_i from the deviations and their remainders
    };
    // the fluid-boundary pairs': x_i - x_j and v_i - v_j in float64
    struct CrossTaken {
        double dd[2][D], dv[2][D];
        float mass[2];
    };
    template <PairKind KIND>
    __device__ __forceinline__ auto take(const Neighbours &N, const NeighbourRows &R0, const NeighbourRows &R1) const
    {
        float vj0[3], vj1[3];
        velocityIn<D>(R0.K, vj0);
        velocityIn<D>(R1.K, vj1);
        const float vl0[3] = {R0.L.x, R0.L.y, R0.L.z}, vl1[3] = {R1.L.x, R1.L.y, R1.L.z};
        if constexpr (KIND == kCrossPair) {
            CrossTaken t;
            for (int q = 0; q < 2; ++q) {
                const NeighbourRows &R = q ? R1 : R0;
                float pj[3], lj[3];
                pointIn<D>(R.A, pj);
                remainderIn<D>(R.A, R.B, lj);
                for (int a = 0; a < D; ++a) {
                    t.dd[q][a] = x[a] - ((double)pj[a] + (double)lj[a]);
                    if (a == 1 && N.image[q]) t.dd[q][a] += x[1] < 0.5 * P.period ? P.period : -P.period;
                    t.dv[q][a] = v[a] - ((double)(q ? vj1[a] : vj0[a]) + (double)(q ? vl1[a] : vl0[a]));
                }
                t.mass[q] = R.m;
            }
            return t;
        } else {
            Taken t;
            for (int a = 0; a < D; ++a)
                t.dv[a] = add2(make_float2(__fsub_rn(vi[a], vj0[a]), __fsub_rn(vi[a], vj1[a])),
                               make_float2(__fsub_rn(vlI[a], vl0[a]), __fsub_rn(vlI[a], vl1[a])));
            t.mass[0] = R0.m;
            t.mass[1] = R1.m;
            t.volume = make_float2(N.live[0] ? volumeIn<D>(R0) : 0.0f, N.live[1] ? volumeIn<D>(R1) : 0.0f);
            t.devJ = make_float2(deviationIn<D>(R0), deviationIn<D>(R1));
            // rho_j - rho_i from the float32 deviations and their remainders, so it keeps float64's
            // digits (the leading difference is exact for neighbours' nearly equal deviations)
            t.leading = make_float2(__fsub_rn(t.devJ.x, devI), __fsub_rn(t.devJ.y, devI));
            t.remainder = make_float2(__fsub_rn(R0.L.w, devLoI), __fsub_rn(R1.L.w, devLoI));
            return t;
        }
    }
    __device__ __forceinline__ void finishCross(const Neighbours &N, const CrossTaken &taken)
    {
        if (N.live[0]) wallPair<0>(N, taken);
        if (N.live[1]) wallPair<1>(N, taken);
    }
    template <PairKind KIND, class T>
    __device__ __forceinline__ void finish(const Neighbours &N, const T &taken)
    {
        if constexpr (KIND == kCrossPair) finishCross(N, taken);
        else finishFluid(N, taken);
    }
    __device__ __forceinline__ void finishFluid(const Neighbours &N, const Taken &taken)
    {
        const float2 grad = kernelGradient<K>(mul2(N.r, N.k.invH), N.k);    // (dW/dr) / r
        const float2 *dv = taken.dv;
        float2 dot = both(0.0f);
        if (corrected) {
            for (int a = 0; a < D; ++a) {
                float2 ld = mul2(both(Li[a][0]), N.d[0]);
                for (int b = 1; b < D; ++b) ld = fma2(both(Li[a][b]), N.d[b], ld);
                dot = a == 0 ? mul2(dv[a], ld) : fma2(dv[a], ld, dot);
            }
        } else {
            for (int a = 0; a < D; ++a) dot = a == 0 ? mul2(dv[a], N.d[a]) : fma2(dv[a], N.d[a], dot);
        }
        const bool live0 = N.live[0], live1 = N.live[1];
        const float m0 = taken.mass[0], m1 = taken.mass[1];
        const float2 massDot = make_float2(live0 ? __fmul_rn(m0, dot.x) : 0.0f, live1 ? __fmul_rn(m1, dot.y) : 0.0f);
        add(massDot, grad);
        if constexpr (BUDGET) {
            float2 plainDot = dot;
            if (corrected)
                for (int a = 0; a < D; ++a) plainDot = a == 0 ? mul2(dv[a], N.d[a]) : fma2(dv[a], N.d[a], plainDot);
            const float2 plain = mul2(plainDot, grad);
            if (live0) plainFluid = __fmaf_rn(m0, plain.x, plainFluid);
            if (live1) plainFluid = __fmaf_rn(m1, plain.y, plainFluid);
            if (live0) continuity = __fmaf_rn(massDot.x, grad.x, continuity);
            if (live1) continuity = __fmaf_rn(massDot.y, grad.y, continuity);
        }
        if (diffuses) {
            const float2 devJ = taken.devJ, leading = taken.leading, remainder = taken.remainder;
            float2 difference;
            if (P.diffusion == 2) {
                // less the hydrostatic difference k dz (1 + e)^-5 (src/pysurf/sphSolver.py:718-735), with
                // k = rho0 g / c0^2 and e the pair's mean deviation over rho0.  Near rest it cancels most
                // of rho_j - rho_i, so it is taken in two parts: k dz off the leading difference in one
                // fused rounding, then the small k dz e S / (1 + e)^5 back on, where
                // S = 1 + (1 + e) + ... + (1 + e)^4 makes (1 + e)^5 - 1 = e S without cancelling.
                const float2 e = mul2(make_float2(__fadd_rn(devI, devJ.x), __fadd_rn(devI, devJ.y)), both(P.halfInvRho0));
                const float2 one = both(1.0f), ratio = add2(one, e), sq = mul2(ratio, ratio), fourth = mul2(sq, sq);
                const float2 fifth = mul2(fourth, ratio);
                const float2 sum = add2(add2(add2(one, ratio), fma2(sq, ratio, sq)), fourth);
                const float2 slope = mul2(both(P.hydrostaticSlope), N.d[D - 1]);
                const float2 back = mul2(mul2(slope, e), sum);
                difference = add2(add2(fma2(both(-P.hydrostaticSlope), N.d[D - 1], leading), remainder),
                                  make_float2(__fdividef(back.x, fifth.x), __fdividef(back.y, fifth.y)));
            } else {
                difference = add2(leading, remainder);
            }
            if (P.diffusion == 3) {
                const float4 g0 = fetch(&F.gradRho[N.j[0]]), g1 = fetch(&F.gradRho[N.j[1]]);
                const float gj0[3] = {g0.x, g0.y, g0.z}, gj1[3] = {g1.x, g1.y, g1.z};
                float2 t = both(0.0f);
                for (int a = 0; a < D; ++a)
                    t = fma2(make_float2(__fadd_rn(gi[a], gj0[a]), __fadd_rn(gi[a], gj1[a])), N.d[a], t);
                difference = fma2(both(0.5f), t, difference);
            }
            // 2 delta c0 h V_j (difference) (-(dW/dr) r) / (r^2 + 0.01 h^2), with (dW/dr) r = grad r^2;
            // with the closure, 2 delta c0 is 2 c0 times the harmonic mean of the two deltas
            float2 factor = both(P.diffusionFactor);
            if (CLOSURE && P.closure) factor = make_float2(pairFactor(N.j[0]), pairFactor(N.j[1]));
            const float2 volume = taken.volume;
            const float2 r2 = mul2(N.r, N.r), below = add2(r2, N.k.soft);
            const float2 head = mul2(mul2(mul2(mul2(factor, N.h), volume), difference), mul2(both(-1.0f), grad));
            const float2 ratio = make_float2(quickDivide(r2.x, below.x), quickDivide(r2.y, below.y));
            add(head, ratio);
            if constexpr (BUDGET) diffusive = __fmaf_rn(head.y, ratio.y, __fmaf_rn(head.x, ratio.x, diffusive));
        }
    }
    __device__ __forceinline__ void add(const float2 &a, const float2 &b)
    {
        if constexpr (COMP) {
            addProduct(a.x, b.x, total.x, comp.x);
            addProduct(a.y, b.y, total.y, comp.y);
        } else {
            total = fma2(a, b, total);
        }
    }
    __device__ __forceinline__ float pairFactor(int j) const
    {
        const float deltaJ = fetch(&F.eddy[j].y), sum = __fadd_rn(deltaI, deltaJ);
        if (!(sum > 0.0f)) return 0.0f;
        return __fmul_rn(__fmul_rn(2.0f, P.closureC0), __fdiv_rn(__fmul_rn(__fmul_rn(2.0f, deltaI), deltaJ), sum));
    }
    // A fluid-boundary pair, in float64.
    template <int Q>
    __device__ __forceinline__ void wallPair(const Neighbours &N, const CrossTaken &taken)
    {
        const double *dd = taken.dd[Q], *dv = taken.dv[Q];
        double r2 = 0.0;
        for (int a = 0; a < D; ++a) r2 = fma(dd[a], dd[a], r2);
        const double rr = preciseRoot<true>(r2, Q ? N.inverse.y : N.inverse.x);
        const double weight = __dmul_rn((double)taken.mass[Q], kernelGradient64<K>(rr, N.k.of(Q)));
        if (corrected) {
            for (int a = 0; a < D; ++a) {
                const double wv = __dmul_rn(weight, dv[a]);
                for (int b = 0; b < D; ++b) cross[a * D + b] = fma(wv, dd[b], cross[a * D + b]);
            }
        } else {
            double dot = __dmul_rn(dv[0], dd[0]);
            for (int a = 1; a < D; ++a) dot = fma(dv[a], dd[a], dot);
            cross[0] = fma(weight, dot, cross[0]);
        }
    }
};

// mode 0: the rate only; 1: advance the density; 2: advance, drift and enforce.
template <int D, int K, int T, bool BUDGET, bool FINE, bool COMP, bool CLOSURE>
__global__ void __launch_bounds__(kBlock, BUDGET ? budgetMinBlocks<D>() : preciseMinBlocks<D>())
continuityKernel(Params P, Frame F, Control *ctl, Enforcement E, int mode)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    stampStages(ctl, P.stages);
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    float hs = signedLength<D>(F, i);
    ContinuityVisit<D, K, BUDGET, FINE, COMP, CLOSURE> visit{P, F, Smoothing<K, D, FINE>(P, fabsf(hs))};
    const bool boundary = hs <= 0.0f;
    visit.diffuses = P.diffusion != 0 && !boundary;
    visit.corrected = P.corrected && !boundary;
    velocityOf<D>(F, i, visit.vi);
    const float4 lowI = F.low[i];
    visit.vlI[0] = lowI.x; visit.vlI[1] = lowI.y; visit.vlI[2] = lowI.z;
    visit.devLoI = lowI.w;
    visit.devI = deviationOf<D>(F, i);
    visit.deltaI = CLOSURE && P.closure && visit.diffuses ? F.eddy[i].y : 0.0f;
    if (visit.corrected) loadMatrix<D>(F.L0, F.L1, F.L2, i, visit.Li);
    visit.gi[0] = visit.gi[1] = visit.gi[2] = 0.0f;
    if (visit.diffuses && P.diffusion == 3) {
        float4 g = F.gradRho[i];
        visit.gi[0] = g.x; visit.gi[1] = g.y; visit.gi[2] = g.z;
    }
    visit.total = visit.comp = both(0.0f);
    visit.plainFluid = visit.continuity = visit.diffusive = 0.0f;
    for (int q = 0; q < D * D; ++q) visit.cross[q] = 0.0;
    const Row row = openRow<D, FINE>(P, F, i, G.t, fabsf(hs));
    for (int a = 0; a < D; ++a) {
        visit.x[a] = (double)row.pi[a] + (double)row.li[a];
        visit.v[a] = (double)visit.vi[a] + (double)visit.vlI[a];
    }
    // the fluid pairs of a fluid row, then the fluid-boundary pairs of either
    if (!boundary) sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, visit);
    sumPairs<D, T, FINE, kCrossPair>(P, F, row, boundary, visit);
    float rate;
    if constexpr (COMP) rate = groupSumCompensated<T>(visit.total, visit.comp, G.mask);
    else rate = groupSum<T>(visit.total, G.mask);
    double cross = visit.cross[0], plainCross = visit.cross[0];
    if (visit.corrected) {
        cross = plainCross = 0.0;
        for (int a = 0; a < D; ++a) {
            for (int b = 0; b < D; ++b) cross = fma((double)visit.Li[a][b], visit.cross[a * D + b], cross);
            plainCross += visit.cross[a * D + a];
        }
    }
    // the fluid-boundary pairs' float64 sum joins before the one rounding to float32
    cross = groupSum<T>(cross, G.mask);
    rate = (float)((double)rate + cross);
    float parts[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if constexpr (BUDGET) {
        // a fluid row's parts (a boundary row keeps none)
        const float continuity = groupSum<T>(visit.continuity, G.mask) + (float)cross;
        parts[0] = groupSum<T>(visit.plainFluid, G.mask);
        parts[1] = (float)groupSum<T>(plainCross, G.mask);
        parts[2] = visit.corrected ? continuity - parts[0] - parts[1] : 0.0f;
        parts[3] = groupSum<T>(visit.diffusive, G.mask);
    }
    if (G.t != 0) return;
    F.rate[i] = rate;
    if (mode == 0) return;
    double dt = ctl->dt;
    const double start = F.rho[i];
    const bool fluid = hs > 0.0f;
    const double unfloored = advanceDensity(P, F, i, rate, dt, fluid, ctl);
    if (BUDGET && fluid) {
        // each part of the rate over the secant slope of e, and the floor's change (src/pysurf/sphGpu.py:1111-1140)
        const double m = F.m[i], slope = elasticSlope(P, start, unfloored);
        for (int q = 0; q < 4; ++q) addEnergy(P, F, i, kContinuityFluid + q, m * slope * (double)parts[q] * dt);
        addEnergy(P, F, i, kFloor, m * (elasticEnergy(P, F.rho[i]) - elasticEnergy(P, unfloored)));
    }
    if (mode == 2 && fluid) driftAndEnforce<D>(P, F, E, i, dt, nullptr, ctl);
}

// ------------------------------------------------------------------------------------------
// Sweep X: XSPH over fluid pairs, with the densities the step has just advanced
// ------------------------------------------------------------------------------------------

template <int D, int K, bool FINE>
struct XsphVisit {
    static constexpr bool kBody = true, kKinetic = true, kAux = true, kLow = false, kMass = false;
    static constexpr bool kSkipCoincident = false;
    const float *densities;
    Smoothing<K, D, FINE> S;
    float vi[3], rhoI, corr[3];
    __device__ void operator()(int j, const float *, float r, float, const KernelAt &k, const NeighbourRows &R)
    {
        const float w = kernelValue<K>(__fmul_rn(r, k.invH), k);
        const float rhoJ = densities ? densities[j] : densityIn<D>(R);
        const float weight = __fdiv_rn(__fmul_rn(massIn<D>(R), w), __fmul_rn(0.5f, __fadd_rn(rhoI, rhoJ)));
        float vj[3];
        velocityIn<D>(R.K, vj);
        for (int a = 0; a < D; ++a) corr[a] = __fmaf_rn(weight, __fsub_rn(vj[a], vi[a]), corr[a]);
    }
};

// densities: the float32 densities the sum divides by (null: the frame's).  mode 0: the transport
// velocity into F.vec only; 2: drift with it and enforce.
template <int D, int K, int T, bool FINE>
__global__ void __launch_bounds__(kBlock, sweepMinBlocks<D>())
xsphKernel(Params P, Frame F, Control *ctl, Enforcement E, const float *densities, int mode)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    float hs = signedLength<D>(F, i);
    float v[3];
    velocityOf<D>(F, i, v);
    if (hs <= 0.0f) {
        if (G.t == 0) F.vec[i] = make_float4(v[0], v[1], v[2], 0.0f);
        return;
    }
    XsphVisit<D, K, FINE> visit{densities, Smoothing<K, D, FINE>(P, hs)};
    visit.vi[0] = v[0]; visit.vi[1] = v[1]; visit.vi[2] = v[2];
    visit.rhoI = densities ? densities[i] : densityOf<D>(F, i);
    visit.corr[0] = visit.corr[1] = visit.corr[2] = 0.0f;
    sumPairs<D, T, FINE, kFluidPair>(P, F, openRow<D, FINE>(P, F, i, G.t, hs), true, visit);
    for (int a = 0; a < D; ++a) visit.corr[a] = groupSum<T>(visit.corr[a], G.mask);
    if (G.t != 0) return;
    float t[3];
    for (int a = 0; a < 3; ++a) t[a] = v[a] + P.xsphEpsilon * visit.corr[a];
    F.vec[i] = make_float4(t[0], t[1], t[2], 0.0f);
    if (mode != 2) return;
    double transport[3] = {(double)t[0], (double)t[1], (double)t[2]};
    driftAndEnforce<D>(P, F, E, i, ctl->dt, transport, ctl);
}

// ------------------------------------------------------------------------------------------
// Particle shifting (src/pysurf/sphGpu.py:856-1008; src/pysurf/sphSolver.py:824-1010), after the
// density update, from the step's starting geometry (the frame's points), the updated densities and
// the kicked velocities
// ------------------------------------------------------------------------------------------

// The frame takes the updated float64 densities: rho, rho - rho0, V = m / rho (p and p / rho^2
// are not read again this step).
template <int D>
__global__ void frameDensityKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    storeDensity<D>(F, i, massOf<D>(F, i), F.rho[i], P.devReference, F.pres[i]);
}

// Over every neighbour of a fluid slot: grad C with the anti-clumping weight 1 + 0.2 (W / W(dx))^4,
// grad C0, div r = -sum V_j r_ij . grad W_ij, grad rho from the deviations.
template <int D, int K>
struct ShiftFieldsVisit {
    static constexpr bool kBody = false, kKinetic = true, kAux = false, kLow = false, kMass = false;
    static constexpr bool kPaired = true;
    static constexpr bool kSkipCoincident = true;
    const Params &P;
    Smoothing<K, D, false> S;
    float devI;
    float2 gradient[D], plain[D], densityGradient[D], total;    // over the lane's even and odd neighbours
    struct Taken {
        float volume[2];
        float2 difference;
    };
    template <PairKind KIND>
    __device__ __forceinline__ Taken take(const Neighbours &, const NeighbourRows &R0, const NeighbourRows &R1) const
    {
        return Taken{{volumeIn<D>(R0), volumeIn<D>(R1)},
                     make_float2(__fsub_rn(deviationIn<D>(R0), devI), __fsub_rn(deviationIn<D>(R1), devI))};
    }
    template <PairKind KIND>
    __device__ __forceinline__ void finish(const Neighbours &N, const Taken &taken)
    {
        const float2 q = mul2(N.r, N.k.invH), grad = kernelGradient<K>(q, N.k);     // (dW/dr) / r
        const float2 ratio = make_float2(__fdiv_rn(kernelValue<K>(q.x, N.k.of(0)), P.spacingKernel),
                                         __fdiv_rn(kernelValue<K>(q.y, N.k.of(1)), P.spacingKernel));
        const float2 square = mul2(ratio, ratio), weight = fma2(mul2(both(0.2f), square), square, both(1.0f));
        const float2 scale = make_float2(N.live[0] ? __fmul_rn(taken.volume[0], grad.x) : 0.0f,
                                         N.live[1] ? __fmul_rn(taken.volume[1], grad.y) : 0.0f);
        for (int a = 0; a < D; ++a) {
            const float2 weighted = mul2(scale, N.d[a]);
            plain[a] = add2(plain[a], weighted);
            gradient[a] = fma2(weight, weighted, gradient[a]);
            densityGradient[a] = fma2(taken.difference, weighted, densityGradient[a]);
        }
        total = fma2(mul2(both(-1.0f), mul2(scale, N.r)), N.r, total);
    }
};

template <int D, int K, int T, bool FINE>
__global__ void __launch_bounds__(kBlock, sweepMinBlocks<D>()) shiftFieldsKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    const float hs = signedLength<D>(F, i);
    if (hs <= 0.0f) {
        if (G.t != 0) return;
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        F.shiftGrad[i] = zero;
        F.shiftPlain[i] = make_float4(0.0f, 0.0f, 0.0f, 1.0e6f);
        F.shiftRhoGrad[i] = zero;
        return;
    }
    ShiftFieldsVisit<D, K> visit{P, Smoothing<K, D, false>(P, hs)};
    visit.devI = deviationOf<D>(F, i);
    for (int a = 0; a < D; ++a) visit.gradient[a] = visit.plain[a] = visit.densityGradient[a] = both(0.0f);
    visit.total = both(0.0f);
    const Row row = openRow<D, FINE>(P, F, i, G.t, hs);
    sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, visit);
    sumPairs<D, T, FINE, kWallPair>(P, F, row, false, visit);
    float c[3] = {0.0f, 0.0f, 0.0f}, g[3] = {0.0f, 0.0f, 0.0f}, rg[3] = {0.0f, 0.0f, 0.0f};
    for (int a = 0; a < D; ++a) {
        c[a] = groupSum<T>(visit.plain[a], G.mask);
        g[a] = groupSum<T>(visit.gradient[a], G.mask);
        rg[a] = groupSum<T>(visit.densityGradient[a], G.mask);
    }
    float total = groupSum<T>(visit.total, G.mask);
    if (G.t != 0) return;
    // a lopsided support marks the free surface (src/pysurf/sphSolver.py:889-902)
    if (hs * sqrtf(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]) > P.lopsidedness) total = -1.0f;
    F.shiftGrad[i] = make_float4(g[0], g[1], g[2], 0.0f);
    F.shiftPlain[i] = make_float4(c[0], c[1], c[2], total);
    F.shiftRhoGrad[i] = make_float4(rg[0], rg[1], rg[2], 0.0f);
}

// The surface neighbours of a slot: whether there is one within the support, and the
// kernel-weighted sum of their outward normals -grad C0 / |grad C0|.
template <int D, int K>
struct SurfaceVisit {
    static constexpr bool kBody = false, kKinetic = false, kAux = false, kLow = false, kMass = false;
    static constexpr bool kSkipCoincident = false;
    const Params &P; const Frame &F;
    Smoothing<K, D, false> S;
    float normal[3];
    int vicinity;
    __device__ void operator()(int j, const float *, float r, float, const KernelAt &k, const NeighbourRows &)
    {
        const float4 plainJ = fetch(&F.shiftPlain[j]);
        if (!(plainJ.w < P.shiftThreshold)) return;
        vicinity = 1;
        const float length = sqrtf(__fmaf_rn(plainJ.z, plainJ.z, __fmaf_rn(plainJ.y, plainJ.y, __fmul_rn(plainJ.x, plainJ.x))));
        if (length > 0.0f) {
            const float w = __fdiv_rn(kernelValue<K>(__fmul_rn(r, k.invH), k), length);
            normal[0] = __fmaf_rn(-w, plainJ.x, normal[0]);
            normal[1] = __fmaf_rn(-w, plainJ.y, normal[1]);
            normal[2] = __fmaf_rn(-w, plainJ.z, normal[2]);
        }
    }
};

// The velocity at the shifted position: sum_j V_j (v_j - v_i) (grad W_ij . shift) over fluid pairs.
template <int D, int K>
struct ShiftedVelocityVisit {
    static constexpr bool kBody = false, kKinetic = true, kAux = false, kLow = false, kMass = false;
    static constexpr bool kSkipCoincident = true;
    Smoothing<K, D, false> S;
    float vi[3], shift[3], change[3];
    __device__ void operator()(int, const float *d, float r, float, const KernelAt &k, const NeighbourRows &R)
    {
        float dot = __fmul_rn(d[0], shift[0]);
        for (int a = 1; a < D; ++a) dot = __fmaf_rn(d[a], shift[a], dot);
        const float f = __fmul_rn(__fmul_rn(volumeIn<D>(R), kernelGradient<K>(__fmul_rn(r, k.invH), k)), dot);
        float vj[3];
        velocityIn<D>(R.K, vj);
        for (int a = 0; a < D; ++a) change[a] = __fmaf_rn(f, __fsub_rn(vj[a], vi[a]), change[a]);
    }
};

// The shift of a fluid slot off the free surface: -size grad C, along the surface next to a
// surface particle (none where h |grad C| > 0.03 there), with the density change shift . grad rho
// and the velocity change at the new position.  size: CFL Ma (2h)^2 with CFL = c0 dt / h, or
// 2 h |v_i| dt (local).
template <int D, int K, int T, bool FINE>
__global__ void __launch_bounds__(kBlock, 5) shiftKernel(Params P, Frame F, const Control *ctl)
{
    awaitPrevious();
    if (ctl && !ctl->active) return;
    const Group<T> G = groupOf<T>();
    const int i = G.i;
    if (i >= P.n) return;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float hs = signedLength<D>(F, i);
    if (hs <= 0.0f || !(F.shiftPlain[i].w >= P.shiftThreshold)) {
        if (G.t == 0) { F.shift[i] = zero; F.shiftDv[i] = zero; }
        return;
    }
    SurfaceVisit<D, K> surface{P, F, Smoothing<K, D, false>(P, hs)};
    surface.normal[0] = surface.normal[1] = surface.normal[2] = 0.0f;
    surface.vicinity = 0;
    const Row row = openRow<D, FINE>(P, F, i, G.t, hs);
    sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, surface);
    float normal[3];
    for (int a = 0; a < 3; ++a) normal[a] = groupSum<T>(surface.normal[a], G.mask);
    const bool vicinity = groupSum<T>((float)surface.vicinity, G.mask) > 0.0f;
    float vi[3];
    velocityOf<D>(F, i, vi);
    const double dt = ctl ? ctl->dt : P.shiftDt;
    const float size =
        P.shiftLocal ? (float)(2.0 * (double)hs * (double)sqrtf(vi[0] * vi[0] + vi[1] * vi[1] + vi[2] * vi[2]) * dt)
                     : (float)(P.shiftScale * dt);
    const float4 g = F.shiftGrad[i];
    float shift[3] = {-size * g.x, -size * g.y, -size * g.z};
    if (vicinity) {
        if (hs * sqrtf(g.x * g.x + g.y * g.y + g.z * g.z) > 0.03f) {
            shift[0] = shift[1] = shift[2] = 0.0f;
        } else {
            const float weight = sqrtf(normal[0] * normal[0] + normal[1] * normal[1] + normal[2] * normal[2]);
            if (weight > 0.0f) {
                float dot = 0.0f;
                for (int a = 0; a < 3; ++a) { normal[a] /= weight; dot += shift[a] * normal[a]; }
                for (int a = 0; a < 3; ++a) shift[a] -= dot * normal[a];
            }
        }
    }
    if (D == 2) shift[2] = 0.0f;
    const float4 rg = F.shiftRhoGrad[i];
    const float densityChange = shift[0] * rg.x + shift[1] * rg.y + shift[2] * rg.z;
    float change[3] = {0.0f, 0.0f, 0.0f};
    if (shift[0] != 0.0f || shift[1] != 0.0f || shift[2] != 0.0f) {
        ShiftedVelocityVisit<D, K> velocity{Smoothing<K, D, false>(P, hs)};
        for (int a = 0; a < 3; ++a) { velocity.vi[a] = vi[a]; velocity.shift[a] = shift[a]; velocity.change[a] = 0.0f; }
        sumPairs<D, T, FINE, kFluidPair>(P, F, row, true, velocity);
        for (int a = 0; a < D; ++a) change[a] = groupSum<T>(velocity.change[a], G.mask);
    }
    if (G.t != 0) return;
    F.shift[i] = make_float4(shift[0], shift[1], shift[2], densityChange);
    F.shiftDv[i] = make_float4(change[0], change[1], change[2], 0.0f);
}

// The drift of a shifting step (src/pysurf/sphGpu.py:1142-1186): x += u dt + shift, rho and v take
// their changes, then the periodic wrap and the enforcement.  transport: XSPH's F.vec, else v.
template <int D>
__global__ void shiftDriftKernel(Params P, Frame F, Control *ctl, Enforcement E, int useTransport)
{
    awaitPrevious();
    if (!ctl->active) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n || !F.fluid[i]) return;
    const double dt = ctl->dt;
    const float4 s = F.shift[i], dv = F.shiftDv[i];
    const float4 u = F.vec[i];
    const float sh[3] = {s.x, s.y, s.z}, dvel[3] = {dv.x, dv.y, dv.z}, ut[3] = {u.x, u.y, u.z};
    double x[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0}, lift = 0.0, kinetic = 0.0, shiftLift = 0.0;
    for (int a = 0; a < D; ++a) {
        const double velocity = useTransport ? (double)ut[a] : F.v[a][i], start = F.x[a][i];
        x[a] = start + velocity * dt;
        lift += P.gravity64[a] * (x[a] - start);
        x[a] = x[a] + (double)sh[a];
        shiftLift += P.gravity64[a] * (double)sh[a];
        v[a] = F.v[a][i] + (double)dvel[a];
        kinetic += v[a] * v[a] - F.v[a][i] * F.v[a][i];
    }
    const double rhoStart = F.rho[i];
    F.rho[i] = rhoStart + (double)s.w;
    if (P.budget) {
        // the drift's change of potential energy, and the shift's of kinetic, elastic and potential
        // energy (src/pysurf/sphGpu.py:1166-1183)
        const double m = F.m[i];
        addEnergy(P, F, i, kDrift, -m * lift);
        addEnergy(P, F, i, kShifting,
                  m * (0.5 * kinetic + elasticEnergy(P, F.rho[i]) - elasticEnergy(P, rhoStart) - shiftLift));
    }
    if (P.period > 0.0) x[1] = x[1] - P.period * floor(x[1] / P.period);
    enforceTracked(P, F, E, D, i, x, v);
    bool finite = isfinite(F.rho[i]);
    for (int a = 0; a < D; ++a) {
        F.x[a][i] = x[a];
        F.v[a][i] = v[a];
        finite = finite && isfinite(x[a]) && isfinite(v[a]);
    }
    if (!finite) atomicOr(&ctl->error, kErrNonFinite);
}

// ------------------------------------------------------------------------------------------
// Launchers
// ------------------------------------------------------------------------------------------

static inline int blocksFor(long long n, int block) { return (int)((n + block - 1) / block); }

// The table kernel: in 3D a cell holds about 8 particles, and the cell batches build the table a quarter
// faster than lanes a particle (19.8 against 14.4 ms a step on the 16-ppd ridge when both were built);
// a 2D cell holds about 4, too few to pay for a batch's setup (0.149 against 0.112 ms on the 64-ppd
// beach), so 2D keeps the lanes.  The table is the same whatever the batch or the lanes.
template <int D, int SHARE>
static void launchListAs(const LaunchArgs &A)
{
    cudaStream_t st = A.stream;
    if constexpr (D == 3) {
        const int grid = blocksFor((long long)blocksFor(A.P.n, SHARE) * 32, kBlock);
        if (A.P.precise && !A.P.mixedH) launchNext(cellListKernel<D, SHARE, true, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else if (A.P.precise) launchNext(cellListKernel<D, SHARE, true, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else if (!A.P.mixedH) launchNext(cellListKernel<D, SHARE, false, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else launchNext(cellListKernel<D, SHARE, false, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
    } else {
        const int grid = blocksFor((long long)A.P.n * SHARE, kBlock);
        if (A.P.precise && !A.P.mixedH) launchNext(listKernel<D, SHARE, true, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else if (A.P.precise) launchNext(listKernel<D, SHARE, true, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else if (!A.P.mixedH) launchNext(listKernel<D, SHARE, false, false>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
        else launchNext(listKernel<D, SHARE, false, true>, grid, kBlock, st, A.P, A.F, A.ctl, A.maxCount);
    }
}

// Particles too few to fill the chip take more of it each: 4 in place of 8 members a batch in 3D, 16 in place
// of 8 lanes a slot in 2D.  Sort and table, ms:
//   3D   26,866 particles 0.256 at 4 a batch, 0.298 at 8; 46,056 0.344, 0.380; 69,084 0.455, 0.442; 130,492
//        0.734, 0.663
//   2D   10,144 particles 0.0274 at 16 lanes, 0.0358 at 8; 22,701 0.0399, 0.0410; 25,798 0.0404, 0.0412;
//        32,546 0.0467, 0.0490; 59,823 0.0691, 0.0674, all with some 100 neighbours; with 20, whose rows of
//        cells give 16 lanes little, a 35,018-particle dam's span of 16 steps takes 1.583 ms at 16 and 1.521
//        at 8
template <int D>
static void launchList(const LaunchArgs &A)
{
    if constexpr (D == 3) {
        if (A.P.n < 65536) launchListAs<D, 4>(A);
        else launchListAs<D, 8>(A);
    } else {
        if (A.P.n < 24576) launchListAs<D, 16>(A);
        else launchListAs<D, 8>(A);
    }
}

// The plain sums are a form of their own, which carries none of the state of the closure, the budget (its
// parts matter only where the step takes the maxima, or advances the density) or the compensated sums.
template <int D, int K, int T, bool FINE>
static void launchMomentum(const LaunchArgs &A, int grid)
{
    const Params &P = A.P;
    const Frame &F = A.F;
    cudaStream_t st = A.stream;
    if (P.budget && A.maxima) launchNext(momentumKernel<D, K, T, true, FINE, false, true>, grid, kBlock, st, P, F, A.ctl, A.maxima);
    else if (P.compensated) launchNext(momentumKernel<D, K, T, false, FINE, true, true>, grid, kBlock, st, P, F, A.ctl, A.maxima);
    else if (P.closure) launchNext(momentumKernel<D, K, T, false, FINE, false, true>, grid, kBlock, st, P, F, A.ctl, A.maxima);
    else launchNext(momentumKernel<D, K, T, false, FINE, false, false>, grid, kBlock, st, P, F, A.ctl, A.maxima);
}
template <int D, int K, int T, bool FINE, bool TABLED>
static void launchGradients(const LaunchArgs &A, int grid)
{
    auto kernel = A.wantRho ? gradientKernel<D, K, T, FINE, true, TABLED> : gradientKernel<D, K, T, FINE, false, TABLED>;
    launchNext(kernel, grid, kBlock, A.stream, A.P, A.F, A.ctl, A.wantG, A.wantL, A.floorDet);
}
template <int D, int K, int T, bool FINE>
static void launchContinuity(const LaunchArgs &A, int grid)
{
    const Params &P = A.P;
    const Frame &F = A.F;
    cudaStream_t st = A.stream;
    if (P.budget && A.flag != 0) launchNext(continuityKernel<D, K, T, true, FINE, false, true>, grid, kBlock, st, P, F, A.ctl, A.E, A.flag);
    else if (P.compensated) launchNext(continuityKernel<D, K, T, false, FINE, true, true>, grid, kBlock, st, P, F, A.ctl, A.E, A.flag);
    else if (P.closure) launchNext(continuityKernel<D, K, T, false, FINE, false, true>, grid, kBlock, st, P, F, A.ctl, A.E, A.flag);
    else launchNext(continuityKernel<D, K, T, false, FINE, false, false>, grid, kBlock, st, P, F, A.ctl, A.E, A.flag);
}

template <int D, int K, int T, bool FINE>
static void launchT(const LaunchArgs &A, Stage stage)
{
    const Params &P = A.P;
    const Frame &F = A.F;
    const int grid = blocksFor((long long)P.n * T, kBlock), pointwise = blocksFor(P.n, kBlock);
    if (P.n == 0) return;
    cudaStream_t st = A.stream;
    switch (stage) {
    case Stage::ShepardSum: launchNext(shepardKernel<D, K, T, FINE>, grid, kBlock, st, P, F, A.ctl); break;
    case Stage::ShepardApply: launchNext(applyShepardKernel<D>, pointwise, kBlock, st, P, F, A.ctl); break;
    case Stage::Wall: launchNext(wallPressureKernel<D, K, T, FINE>, grid, kBlock, st, P, F, A.ctl, A.flag); break;
    case Stage::Gradients:
        if (D == 3 && !FINE && A.tabled) launchGradients<D, K, T, FINE, D == 3 && !FINE>(A, grid);
        else launchGradients<D, K, T, FINE, false>(A, grid);
        break;
    case Stage::Momentum: launchMomentum<D, K, T, FINE>(A, grid); break;
    case Stage::Kick: launchNext(kickKernel<D>, pointwise, kBlock, st, P, F, A.ctl); break;
    case Stage::Continuity: launchContinuity<D, K, T, FINE>(A, grid); break;
    case Stage::Xsph: launchNext(xsphKernel<D, K, T, FINE>, grid, kBlock, st, P, F, A.ctl, A.E, A.densities, A.flag); break;
    case Stage::List:
        // the table does not depend on the kernel: one unit builds it for both
        if constexpr (K == 1) launchList<D>(A);
        break;
    case Stage::Closure: launchNext(closureKernel<D>, pointwise, kBlock, st, P, F, A.ctl); break;
    case Stage::ShiftFields: launchNext(shiftFieldsKernel<D, K, T, false>, grid, kBlock, st, P, F, A.ctl); break;
    case Stage::Shift: launchNext(shiftKernel<D, K, T, false>, grid, kBlock, st, P, F, A.ctl); break;
    case Stage::ShiftDrift: launchNext(shiftDriftKernel<D>, pointwise, kBlock, st, P, F, A.ctl, A.E, A.flag); break;
    case Stage::FrameDensity: launchNext(frameDensityKernel<D>, pointwise, kBlock, st, P, F, A.ctl); break;
    }
}

template <int D, int K>
static void launchDK(const LaunchArgs &A, Stage stage)
{
    if (A.P.levels > 1 || A.P.mixedH) {
        // the shifting sweeps never see differing lengths (shifting needs one smoothing length)
        if (A.threads >= 8) launchT<D, K, 8, true>(A, stage);
        else if (A.threads == 4) launchT<D, K, 4, true>(A, stage);
        else if (A.threads == 2) launchT<D, K, 2, true>(A, stage);
        else launchT<D, K, 1, true>(A, stage);
    } else {
        if (A.threads >= 8) launchT<D, K, 8, false>(A, stage);
        else if (A.threads == 4) launchT<D, K, 4, false>(A, stage);
        else if (A.threads == 2) launchT<D, K, 2, false>(A, stage);
        else launchT<D, K, 1, false>(A, stage);
    }
}

// This file is compiled once a dimension and kernel (SPH_SWEEP_DIM 2 and 3, SPH_SWEEP_KERNEL 0 and 1), so
// that its units build side by side.
#define SPH_JOIN2(a, b, c) a##b##_##c
#define SPH_JOIN(a, b, c) SPH_JOIN2(a, b, c)
void SPH_JOIN(launchStage, SPH_SWEEP_DIM, SPH_SWEEP_KERNEL)(const LaunchArgs &A, Stage stage)
{
    launchDK<SPH_SWEEP_DIM, SPH_SWEEP_KERNEL>(A, stage);
}

}  // namespace sph

// Neighbour lists per warp-group of 32 SFC-consecutive target particles.
//
// Replaces cstone::findNeighbors / sph::findNeighborsSph (domain/include/cstone/findneighbors.hpp:
// 77-170, sph/include/sph/find_neighbors.hpp:10-56) and the reference GPU's per-pass warp
// traversal (domain/include/cstone/traversal/find_neighbors.cuh:182-489).  The set of neighbours
// of i is exactly the reference CPU set {j != i : d2(i,j) < 4 h_i^2}, with d2 rounded as in
// distanceSq (minimum image by rint when the 2h box of i leaves a periodic box).
//
// Per warp: one depth-first walk of the octree in SFC order against the group's search box, so
// candidate ranges arrive in ascending particle order and every list comes out sorted.  Leaves,
// internal nodes whose box lies inside the search box and internal nodes of few particles each
// give one contiguous particle range (per-node ranges precomputed with the tree); contiguous
// ranges are merged and staged 32 candidates at a time in shared memory.
// Positions are read in the grid form of the mixed passes: a 21-bit cell per axis plus an FP32
// offset inside the cell.  Offsets from the group origin are (cell difference, wrapped exactly
// in integers) x cell edge + (offset difference), so neither staging nor the distance filter
// runs an FP64 instruction.  Only pairs whose FP32 distance lies within a rounding margin of the
// radius are re-tested in FP64 from the original coordinates.  Lists are stored in granules of four
// entries transposed per granule (listSlot), written one 16-byte granule at a time, so that the pair
// passes read them coalesced.
#include <algorithm>
#include <cmath>


#include "pairs.cuh"

namespace sphgb {

namespace {

constexpr int kNbrBlock = 128;
constexpr int kWarpsPerBlock = kNbrBlock / kWarp;
constexpr int kStack = 192;  // 8 children x (21 levels + 3)
// internal nodes of at most this many particles are taken whole: eight leaves of 13-30, the octree's
// last level.  With nodes pruned by their distance from the target box, fewer pops pay for the extra
// staged candidates: 8M search stage 12.9 ms against 13.1 with 128; 64 costs the 27M set 7 ms of 28.
constexpr uint32_t kCoarseNode = 256;
// above the rounding of a squared FP32 distance that is subnormal (lengths below 1e-19 in the caller's units):
// part of every margin on squares.  Below 1e-21 all squares lie inside it and all candidates take the FP64
// test.
constexpr float kTinySq = 0x1p-140f;

struct NbrArgs {
    const double *x, *y, *z;
    const void* h;
    int hIsFloat;
    const u64* cell;      // packed grid cell per particle
    const float4* loc;    // FP32 offset inside the cell (w unused here)
    float u[3];           // cell edge per axis
    int sh[3];            // 32 - 21 on periodic axes, 0 on open ones (wrapShift)
    int64_t first, last;
    const uint32_t* active;  // optional: only targets with active[i - first] != 0 are searched
    const int32_t* childOffsets;
    const float4* nodeBox;
    const uint2* nodeRange;  // particles [start, end) per node
    float pruneUnit;         // power of two: the unit of the squared distances that prune nodes
    DevBox box;
    uint32_t ngmax;
    int64_t stride;
    uint32_t* nbr;
    uint32_t* count;           // [last-first] neighbours excluding self (uncapped)
    int* flags;
    unsigned long long* stats; // [0] candidates [1] fp64 rechecks
};

__device__ __forceinline__ double loadH(const void* h, int isFloat, int64_t i)
{
    return isFloat ? double(static_cast<const float*>(h)[i]) : static_cast<const double*>(h)[i];
}

__device__ __forceinline__ double foldRint(double d, const DevBox& b, int k)
{
    // minimum image of the reference's distanceSq<true> / applyPbc: d - L * rint(d / L)
    return __dsub_rn(d, __dmul_rn(b.L[k], rint(__dmul_rn(d, b.iL[k]))));
}

__device__ __forceinline__ void unpackCell(u64 c, int ic[3])
{
    ic[0] = int(c & kGridMask);
    ic[1] = int((c >> kGridBits) & kGridMask);
    ic[2] = int(c >> (2 * kGridBits));
}

// offset of a particle (cell cj, offset lj) from the origin (cell co, offset lo), FP32
__device__ __forceinline__ void gridOffset(const NbrArgs& a, const int cj[3], float4 lj, const int co[3], float4 lo,
                                           float r[3])
{
    const float lv[3] = {lj.x - lo.x, lj.y - lo.y, lj.z - lo.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = fmaf(float(CoordMixed::wrapShift(cj[k] - co[k], a.sh[k])), a.u[k], lv[k]);
}

// tested candidate blocks whose decision masks wait in registers before the lanes append their neighbours
constexpr int kHeld = 4;

struct WarpSmem {
    int32_t stack[kStack];
    // queue of staged candidates that lie in the group's search box: negated offsets from the
    // group origin, one array per axis so that one 16-byte broadcast load gives four candidates'
    // coordinate for the packed FP32x2 arithmetic, and their particle indices (ascending)
    alignas(16) float nx[2 * kWarp];
    alignas(16) float ny[2 * kWarp];
    alignas(16) float nz[2 * kWarp];
    alignas(16) uint32_t idx[2 * kWarp];
    uint32_t self[kWarp];  // position of each target in the queue, counted from the first candidate
    uint32_t held[kHeld][kWarp];  // indices of the tested blocks whose neighbours are still to be appended
    // the cull: box of the target positions (lo x y z, squared radius, hi x y z)
    alignas(16) float cull[8];
};

// Bound by instruction issue (about 27k warp instructions per group of 32 targets and 620 tests per target).
// At 27M particles the search takes 28.0 ms (37.1 with an append loop per tested block, nodes pruned per
// axis, 6 blocks per SM and nodes of 128 particles taken whole); 8 blocks of 64 registers hide the
// staging loads best (6: 29.6 ms, 7: 28.6, 9: 30.3).
// Fold: groups whose pairs need a fold each do it in FP32; without it they run the FP64 test for every pair,
// and the code of the fold does not cost registers (1 % of the search at 27M).  What decides is geometry, a search
// region beyond half a periodic box, which the launch does not know; below kFoldBelow particles a cubic box
// with ordinary h reaches it (12^3: a sweep of 2.42 ms with the FP64 tests, 1.33 with the fold), and larger
// sets do only in a box that is thin on a periodic axis, where they take the FP64 test as they always did.
constexpr int64_t kFoldBelow = 100000;

template<bool Fold>
__global__ void __launch_bounds__(kNbrBlock, Fold ? 6 : 8) nbrGroupKernel(NbrArgs a)
{
    __shared__ WarpSmem smem[kWarpsPerBlock];
    const int lane = threadIdx.x & (kWarp - 1);
    WarpSmem& sm = smem[threadIdx.x / kWarp];
    const int64_t g0 = a.first + (int64_t(blockIdx.x) * kWarpsPerBlock + threadIdx.x / kWarp) * kWarp;
    if (g0 >= a.last) return;
    const int64_t i = g0 + lane;
    bool valid = i < a.last && (a.active == nullptr || a.active[i - a.first] != 0);
    const unsigned validMask = __ballot_sync(0xffffffffu, valid);
    if (validMask == 0) return;
    const int leader = __ffs(validMask) - 1;
    const DevBox& b = a.box;

    // targets: grid form for the filter, exact FP64 radius and periodic decision
    const int64_t iv = valid ? i : g0 + leader;
    const u64 cellI = a.cell[iv];
    const float4 locI = a.loc[iv];
    const double hi = valid ? loadH(a.h, a.hIsFloat, i) : 0.0;
    const double r2 = __dmul_rn(__dmul_rn(4.0, hi), hi);  // reference radiusSq = 4 h h
    const double twoH = __dmul_rn(2.0, hi);
    bool usePbc = false;
    if (valid && (b.pbc[0] | b.pbc[1] | b.pbc[2])) {
        const double xi = a.x[i], yi = a.y[i], zi = a.z[i];
        const bool inside = __dsub_rn(xi, twoH) >= b.lo[0] && __dsub_rn(yi, twoH) >= b.lo[1] &&
                            __dsub_rn(zi, twoH) >= b.lo[2] && __dadd_rn(xi, twoH) <= b.hi[0] &&
                            __dadd_rn(yi, twoH) <= b.hi[1] && __dadd_rn(zi, twoH) <= b.hi[2];
        usePbc = !inside;
    }

    // group origin = the leader's cell and offset
    int co[3], ci[3];
    unpackCell(__shfl_sync(0xffffffffu, cellI, leader), co);
    unpackCell(cellI, ci);
    float4 lo;
    lo.x = __shfl_sync(0xffffffffu, locI.x, leader);
    lo.y = __shfl_sync(0xffffffffu, locI.y, leader);
    lo.z = __shfl_sync(0xffffffffu, locI.z, leader);
    lo.w = 0.f;
    float reli[3];
    gridOffset(a, ci, locI, co, lo, reli);
    const float dxi = reli[0], dyi = reli[1], dzi = reli[2];
    const float rf = valid ? __double2float_ru(twoH) : 0.f;

    // box of the target positions relative to the origin, and the largest radius: the search region is
    // that box grown by rfm, with rounded edges and corners
    float tmn[3] = {valid ? dxi : INFINITY, valid ? dyi : INFINITY, valid ? dzi : INFINITY};
    float tmx[3] = {valid ? dxi : -INFINITY, valid ? dyi : -INFINITY, valid ? dzi : -INFINITY};
    float rfm = rf;
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            tmn[k] = fminf(tmn[k], __shfl_xor_sync(0xffffffffu, tmn[k], o));
            tmx[k] = fmaxf(tmx[k], __shfl_xor_sync(0xffffffffu, tmx[k], o));
        }
        rfm = fmaxf(rfm, __shfl_xor_sync(0xffffffffu, rfm, o));
    }
    // absolute position of the origin from its cell (FP32 suffices for pruning, see the pad).
    // foldPairs: on some periodic axis the search region reaches half the box from the origin (sets of a
    // few thousand particles).  Below that a neighbour's offset, wrapped against the origin, is also
    // the image nearest to its target (|offset| <= Rg < L/2), so differences of offsets need no fold.
    bool foldPairs = false;
    float gc[3], gt[3], Rg = 0.f;  // center and half size of the target box for the walk, padded
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float reach = fmaxf(fabsf(tmn[k]), fabsf(tmx[k])) + rfm;
        if (b.pbc[k] && reach > 0.49f * b.Lf[k]) foldPairs = true;
        const float lok = (k == 0) ? lo.x : (k == 1 ? lo.y : lo.z);
        float cAbs = float(b.lo[k]) + fmaf(float(co[k]), a.u[k], lok) + 0.5f * (tmn[k] + tmx[k]);
        if (b.pbc[k]) {
            if (cAbs >= float(b.hi[k])) cAbs -= b.Lf[k];
            else if (cAbs < float(b.lo[k])) cAbs += b.Lf[k];
        }
        gc[k] = cAbs;
        const float pad = float((fabs(b.lo[k]) + fabs(b.hi[k])) * 0x1p-19);
        gt[k] = 0.5f * (tmx[k] - tmn[k]) + pad;
        Rg = fmaxf(Rg, reach);
    }
    const float gR = rfm * a.pruneUnit, gR2 = fmaf(gR * gR, 1.f + 0x1p-18f, kTinySq);
    // FP32 decision margin on d2: covers the rounding of cell edge, offsets and the squared sum (and,
    // where pairs are folded, of the box length, L <= 2 Rg / 0.98 there); pairs inside the margin get the
    // exact FP64 test
    const float r2f = float(r2);
    const float margin = 64.f * 0x1p-24f * (Rg + rf) * (Rg + rf) + kTinySq;
    const float inBelow = r2f - margin;   // d2f < inBelow: neighbour
    const float outAbove = r2f + margin;  // d2f > outAbove: not a neighbour

    unsigned cnt = 0;
    unsigned long long tested = 0, rechecked = 0;
    const int64_t ii = i - a.first;
    const uint32_t iu = uint32_t(i);
    GranuleWriter out(a.nbr, ii, a.stride, a.ngmax);

    // the reference's distanceSq decision in FP64 (findneighbors.hpp:33-60)
    auto exactIn = [&](uint32_t j) {
        ++rechecked;
        double dx = __dsub_rn(a.x[j], a.x[i]), dy = __dsub_rn(a.y[j], a.y[i]), dz = __dsub_rn(a.z[j], a.z[i]);
        if (usePbc) {
            if (b.pbc[0]) dx = foldRint(dx, b, 0);
            if (b.pbc[1]) dy = foldRint(dy, b, 1);
            if (b.pbc[2]) dz = foldRint(dz, b, 2);
        }
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        return d2 < r2;
    };
    auto take = [&](uint32_t j) {
        if (j != iu) {
            out.put(cnt, j);
            ++cnt;
        }
    };
    // Appends run for four tested blocks together.  The hits of one block of 32 lie in few lanes (17
    // loop trips for 5 hits on average, the block being a compact cluster near some of the targets); over
    // four blocks the lanes even out (1M particles: 341 -> 150 trips per warp and search).
    uint32_t m0 = 0, m1 = 0, m2 = 0, m3 = 0;
    int nHeld = 0;
    auto appendHeld = [&]() {
        int base = -1;
        while (m0 | m1 | m2 | m3) {
            const bool next = m0 == 0;
            m0 = next ? m1 : m0;
            m1 = next ? m2 : m1;
            m2 = next ? m3 : m2;
            m3 = next ? 0u : m3;
            base += next ? kWarp : 0;
            if (m0 != 0) {
                out.put(cnt, (&sm.held[0][0])[base + __ffs(m0)]);
                ++cnt;
                m0 &= m0 - 1u;
            }
        }
        nHeld = 0;
        __syncwarp();
    };

    // Candidates are staged 32 at a time (one per lane, coalesced loads of cell and offset); those
    // outside the search region by more than the FP32 rounding of the offsets (cullPad) are
    // dropped and the rest appended, in ascending index order, to the warp's queue by ballot
    // compaction.  A dropped candidate is farther than 2h from every target, so the reference's FP64
    // test rejects it too.  Each full queue block of 32 is tested by every target
    // with a fixed trip count; the last, partial block has NaN in its empty slots.
    // Groups that fold their pairs keep every candidate.
    const float cullPad = 32.f * 0x1p-24f * (Rg + fmaxf(a.u[0], fmaxf(a.u[1], a.u[2])));
    // the cull: a candidate farther than max 2h from the target box is farther than 2h_i from every
    // target i; the pad covers the offsets' FP32 rounding, the factor the squared sum's
    const float cullR = rfm + cullPad;
    if (lane == 0) {
        sm.cull[0] = tmn[0];
        sm.cull[1] = tmn[1];
        sm.cull[2] = tmn[2];
        sm.cull[3] = fmaf(cullR * cullR, 1.f + 0x1p-18f, kTinySq);
        sm.cull[4] = tmx[0];
        sm.cull[5] = tmx[1];
        sm.cull[6] = tmx[2];
        sm.cull[7] = 0.f;
    }
    __syncwarp();
    // 1/L of the periodic axes (0 leaves an axis unfolded)
    const float foldL[3] = {b.pbc[0] ? 1.f / b.Lf[0] : 0.f, b.pbc[1] ? 1.f / b.Lf[1] : 0.f, b.pbc[2] ? 1.f / b.Lf[2] : 0.f};
    int qn = 0;          // candidates in the queue
    uint32_t qBase = 0;  // candidates tested before the queue's first
    sm.self[lane] = 0xffffffffu;
    __syncwarp();
    auto testBlock = [&](int filled) {
        if (valid) tested += unsigned(filled);
        if (!Fold && foldPairs) {
            if (valid)
                for (int t = 0; t < filled; ++t) {
                    const uint32_t j = sm.idx[t];
                    if (exactIn(j)) take(j);
                }
        } else {
            uint32_t hit = 0, nearm = 0;
            if (Fold && foldPairs) {
                // offsets of target and candidate may differ by up to L: the nearest image of the
                // difference, in FP32.  Where 2h < L/2 there is one image within the radius; beyond,
                // images at equal distance give the same d2 to rounding.
    #pragma unroll 1
                for (int t = 0; t < filled; t += 4) {
                    const float4 X = *reinterpret_cast<const float4*>(&sm.nx[t]);
                    const float4 Y = *reinterpret_cast<const float4*>(&sm.ny[t]);
                    const float4 Z = *reinterpret_cast<const float4*>(&sm.nz[t]);
                    const float x[4] = {X.x, X.y, X.z, X.w}, y[4] = {Y.x, Y.y, Y.z, Y.w}, z[4] = {Z.x, Z.y, Z.z, Z.w};
    #pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        float ex = dxi + x[s], ey = dyi + y[s], ez = dzi + z[s];
                        ex = fmaf(-b.Lf[0], rintf(ex * foldL[0]), ex);
                        ey = fmaf(-b.Lf[1], rintf(ey * foldL[1]), ey);
                        ez = fmaf(-b.Lf[2], rintf(ez * foldL[2]), ez);
                        const float d2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                        hit |= (d2 < inBelow ? 1u : 0u) << (t + s);
                        nearm |= (d2 <= outAbove ? 1u : 0u) << (t + s);
                    }
                }
            } else {
                // four slots per step on packed FP32x2 operations: e = d_i + (-r_j) rounds as
                // d_i - r_j, and d2 = fma(ex, ex, fma(ey, ey, ez * ez)) per slot as in scalar form.
                // The block's decisions go into two 32-bit masks (d2 below the margin: neighbour; d2
                // within it: exact FP64 test), then each lane appends its neighbours slot by slot in
                // ascending order, one loop trip per neighbour instead of a predicated append per slot.
                const float2 dx2 = make_float2(dxi, dxi), dy2 = make_float2(dyi, dyi), dz2 = make_float2(dzi, dzi);
    #pragma unroll
                for (int t = 0; t < kWarp; t += 4) {
                    const float4 X = *reinterpret_cast<const float4*>(&sm.nx[t]);
                    const float4 Y = *reinterpret_cast<const float4*>(&sm.ny[t]);
                    const float4 Z = *reinterpret_cast<const float4*>(&sm.nz[t]);
                    const float2 ex0 = __fadd2_rn(dx2, make_float2(X.x, X.y));
                    const float2 ex1 = __fadd2_rn(dx2, make_float2(X.z, X.w));
                    const float2 ey0 = __fadd2_rn(dy2, make_float2(Y.x, Y.y));
                    const float2 ey1 = __fadd2_rn(dy2, make_float2(Y.z, Y.w));
                    const float2 ez0 = __fadd2_rn(dz2, make_float2(Z.x, Z.y));
                    const float2 ez1 = __fadd2_rn(dz2, make_float2(Z.z, Z.w));
                    const float2 q0 = __ffma2_rn(ex0, ex0, __ffma2_rn(ey0, ey0, __fmul2_rn(ez0, ez0)));
                    const float2 q1 = __ffma2_rn(ex1, ex1, __ffma2_rn(ey1, ey1, __fmul2_rn(ez1, ez1)));
                    const float d2[4] = {q0.x, q0.y, q1.x, q1.y};
    #pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        hit |= (d2[s] < inBelow ? 1u : 0u) << (t + s);
                        nearm |= (d2[s] <= outAbove ? 1u : 0u) << (t + s);
                    }
                }
            }
            // a target is no neighbour of itself
            const uint32_t own = sm.self[lane] - qBase;
            if (own < unsigned(kWarp)) {
                hit &= ~(1u << own);
                nearm &= ~(1u << own);
            }
            if (valid) {
                // a pair within the FP32 margin of the radius (rare): the exact test
                for (uint32_t band = nearm & ~hit; band != 0; band &= band - 1u) {
                    const int s = __ffs(band) - 1;
                    if (exactIn(sm.idx[s])) hit |= 1u << s;
                }
            } else
                hit = 0;
            sm.held[nHeld][lane] = sm.idx[lane];
            if (nHeld == 0) m0 = hit;
            else if (nHeld == 1) m1 = hit;
            else if (nHeld == 2) m2 = hit;
            else m3 = hit;
            ++nHeld;
            __syncwarp();
            if (nHeld == kHeld) appendHeld();
        }
        qBase += kWarp;
        __syncwarp();
    };
    auto flush = [&](int64_t ja, int m) {
        float rj[3];
        bool keep = false;
        if (lane < m) {
            const int64_t j = ja + lane;
            int cj[3];
            unpackCell(a.cell[j], cj);
            gridOffset(a, cj, a.loc[j], co, lo, rj);
            const float4 cl = *reinterpret_cast<const float4*>(&sm.cull[0]);
            const float4 ch = *reinterpret_cast<const float4*>(&sm.cull[4]);
            const float ex = fmaxf(fmaxf(cl.x - rj[0], rj[0] - ch.x), 0.f);
            const float ey = fmaxf(fmaxf(cl.y - rj[1], rj[1] - ch.y), 0.f);
            const float ez = fmaxf(fmaxf(cl.z - rj[2], rj[2] - ch.z), 0.f);
            keep = foldPairs || fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= cl.w;
        }
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int q = qn + __popc(km & ((1u << lane) - 1u));
            sm.nx[q] = -rj[0];
            sm.ny[q] = -rj[1];
            sm.nz[q] = -rj[2];
            sm.idx[q] = uint32_t(ja + lane);
            const int64_t t = ja + lane - g0;
            if (t >= 0 && t < kWarp) sm.self[t] = qBase + q;
        }
        qn += __popc(km);
        __syncwarp();
        if (qn >= kWarp) {
            testBlock(kWarp);
            qn -= kWarp;
            if (lane < qn) {  // move the queue's tail [32, 32 + qn) to the front
                sm.nx[lane] = sm.nx[kWarp + lane];
                sm.ny[lane] = sm.ny[kWarp + lane];
                sm.nz[lane] = sm.nz[kWarp + lane];
                sm.idx[lane] = sm.idx[kWarp + lane];
            }
            __syncwarp();
        }
    };
    // the partial last block: NaN in the empty slots, so that neither comparison holds (also where r^2
    // overflows FP32 and every pair is within the margin)
    auto drain = [&]() {
        if (qn == 0) return;
        if (lane >= qn) {
            sm.nx[lane] = sm.ny[lane] = sm.nz[lane] = __int_as_float(0x7fffffff);
        }
        __syncwarp();
        testBlock(qn);
        qn = 0;
    };

    int64_t pa = 0, pb = 0;  // pending contiguous candidate range
    auto addRange = [&](int64_t la, int64_t lb) {
        if (la == lb) return;
        if (la != pb) {
            while (pb > pa) {
                const int m = int(pb - pa < kWarp ? pb - pa : int64_t(kWarp));
                flush(pa, m);
                pa += m;
            }
            pa = la;
        }
        pb = lb;
        while (pb - pa >= kWarp) {
            flush(pa, kWarp);
            pa += kWarp;
        }
    };

    // depth-first walk in SFC order: children pushed in reverse so child 0 is popped first
    if (lane == 0) sm.stack[0] = 0;
    int sp = 1;
    __syncwarp();
    bool overflow = false;
    while (sp > 0) {
        // stack entries: node index, sign bit set when the node's box lies inside the search box
        const int32_t e = sm.stack[--sp];
        const int32_t node = e & 0x7fffffff;
        // a leaf, an internal node inside the search box (all its children would be walked) or one
        // of at most kCoarseNode particles: one contiguous range of particles instead of a walk over
        // its leaves.  Extra candidates only cost staging: the culls and the pair test decide.
        const int32_t co8 = a.childOffsets[node];
        const uint2 nr = a.nodeRange[node];
        if (co8 == 0 || e < 0 || nr.y - nr.x <= kCoarseNode) {
            addRange(nr.x, nr.y);
            continue;
        }
        bool ov = false, inside = false;
        const int32_t child = co8 + (lane & 7);
        if (lane < 8) {
            const float4 c4 = a.nodeBox[2 * child], s4 = a.nodeBox[2 * child + 1];
            const float cc[3] = {c4.x, c4.y, c4.z}, ss[3] = {s4.x, s4.y, s4.z};
            inside = true;
            float e2 = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float dd = fabsf(cc[k] - gc[k]);
                if (b.pbc[k]) dd = fminf(dd, b.Lf[k] - dd);
                const float gap = fmaxf(dd - ss[k] - gt[k], 0.f) * a.pruneUnit;
                e2 = fmaf(gap, gap, e2);
                inside = inside && (dd + ss[k] <= gt[k] + rfm);
            }
            ov = e2 <= gR2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, ov);
        const int k = __popc(m);
        if (sp + k > kStack) {
            overflow = true;
            break;
        }
        __syncwarp();
        if (ov) sm.stack[sp + __popc(m >> (lane + 1))] = inside ? int32_t(uint32_t(child) | 0x80000000u) : child;
        sp += k;
        __syncwarp();
    }
    if (overflow) {
        if (lane == 0) atomicOr(a.flags, kFlagStackOverflow);
        return;
    }
    while (pb > pa) {
        const int m = int(pb - pa < kWarp ? pb - pa : int64_t(kWarp));
        flush(pa, m);
        pa += m;
    }
    drain();
    appendHeld();

    if (valid) {
        out.finish(cnt);
        a.count[ii] = cnt;
    }
    // warp-aggregated statistics
    for (int o = 16; o > 0; o >>= 1) {
        tested += __shfl_xor_sync(0xffffffffu, tested, o);
        rechecked += __shfl_xor_sync(0xffffffffu, rechecked, o);
    }
    if (lane == 0 && a.stats) {
        atomicAdd(&a.stats[0], tested);
        atomicAdd(&a.stats[1], rechecked);
    }
}

// h / nc iteration step (sph/include/sph/find_neighbors.hpp:26-37, updateH kernels.hpp:26-32):
// marks targets that leave [ng0/4, ngmax+1] and updates their h; counts active and failed.
template<class Th>
__global__ void hIterKernel(const uint32_t* __restrict__ count, Th* __restrict__ h, uint32_t* __restrict__ active,
                            uint8_t* __restrict__ iters, int64_t first, int64_t nWork, unsigned ng0, unsigned ngmax,
                            unsigned long long* __restrict__ counters)
{
    int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= nWork) return;
    unsigned nc = count[k] + 1;
    unsigned ngmin = ng0 / 4;
    bool bad = (ngmin > nc) || (nc - 1 > ngmax);
    bool go = bad && iters[k] < 10 && (active[k] != 0);
    if (go) {
        Th hv = h[first + k];
        const Th c0 = Th(1023.0);
        const Th ex = Th(1.0) / Th(10.0);
        h[first + k] = hv * Th(0.5) * pow(Th(1) + c0 * ng0 / Th(nc), ex);
        iters[k]++;
        atomicAdd(&counters[2], 1ull);
    }
    active[k] = go ? 1u : 0u;
}

constexpr int kNcOutBlock = 256;

__global__ void __launch_bounds__(kNcOutBlock) ncOutKernel(const uint32_t* __restrict__ count, const uint8_t* __restrict__ iters, int64_t nWork,
                            uint32_t ngmax, uint32_t* __restrict__ nc, int addSelf,
                            unsigned long long* __restrict__ counters)
{
    int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    unsigned long long capped = 0, sum = 0, fails = 0;
    unsigned mx = 0;
    if (k < nWork) {
        uint32_t cnt = count[k];
        if (nc) nc[k] = cnt + (addSelf ? 1u : 0u);
        capped = cnt > ngmax;
        sum = min(cnt, ngmax);
        mx = cnt + 1;
        fails = (iters && iters[k] >= 10) ? 1 : 0;
    }
    for (int o = 16; o > 0; o >>= 1) {
        capped += __shfl_xor_sync(0xffffffffu, capped, o);
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        fails += __shfl_xor_sync(0xffffffffu, fails, o);
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    // one atomic per block and counter: same-address atomics from every warp serialise in L2
    __shared__ unsigned long long sS[kNcOutBlock / kWarp], sC[kNcOutBlock / kWarp], sF[kNcOutBlock / kWarp];
    __shared__ unsigned sM[kNcOutBlock / kWarp];
    const int w = threadIdx.x / kWarp;
    if ((threadIdx.x & 31) == 0) {
        sS[w] = sum;
        sC[w] = capped;
        sF[w] = fails;
        sM[w] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < kNcOutBlock / kWarp; ++q) {
            sum += sS[q];
            capped += sC[q];
            fails += sF[q];
            mx = max(mx, sM[q]);
        }
        atomicAdd(&counters[3], sum);
        atomicAdd(&counters[4], capped);
        atomicMax(&counters[5], (unsigned long long)mx);
        atomicAdd(&counters[6], fails);
    }
}

// lists in the reference layout out[k * ngmax + q], q < min(count, ngmax).  A warp copies 32 lists, 32
// entries at a time: the lanes read granules of their own list (512 contiguous bytes per granule row),
// turn the 32 x 32 entries in shared memory, and write runs of up to 128 bytes of one row.  Written
// straight from the lists' order every lane's 4-byte stores went to a row of its own, 0.75 ms at 1M
// particles (0.4 GB read and written); now 0.23 ms.
constexpr int kExportWarps = 4;

__global__ void __launch_bounds__(32 * kExportWarps) exportKernel(const uint32_t* __restrict__ nbr,
                                                                  const uint32_t* __restrict__ count, int64_t nWork,
                                                                  int64_t stride, uint32_t ngmax,
                                                                  uint32_t* __restrict__ out)
{
    __shared__ uint32_t tile[kExportWarps][32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t k0 = (blockIdx.x * int64_t(kExportWarps) + w) * 32;
    if (k0 >= nWork) return;
    const int64_t k = k0 + lane;
    const uint32_t c = k < nWork ? min(count[k], ngmax) : 0u;
    const uint32_t longest = __reduce_max_sync(0xffffffffu, c);
    const uint4* lists = reinterpret_cast<const uint4*>(nbr) + (k < nWork ? k : k0);
    for (uint32_t q0 = 0; q0 < longest; q0 += 32) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const uint32_t q = q0 + 4 * g;
            if (q < c) {
                const uint4 e = __ldg(lists + int64_t(q / kListGran) * stride);
                tile[w][lane][4 * g] = e.x;
                tile[w][lane][4 * g + 1] = e.y;
                tile[w][lane][4 * g + 2] = e.z;
                tile[w][lane][4 * g + 3] = e.w;
            }
        }
        __syncwarp();
#pragma unroll 4
        for (int r = 0; r < 32; ++r) {
            const uint32_t cr = __shfl_sync(0xffffffffu, c, r);
            if (q0 + lane < cr) out[(k0 + r) * ngmax + q0 + lane] = tile[w][r][lane];
        }
        __syncwarp();
    }
}

// ---- owned pair lists for the pair-once momentum-energy pass ----
// Pair (i, j) is mutual when the k-th neighbour j of i also lists i: j has a list (inside the
// searched range), i lies within j's capped list (the ngmax smallest indices), and |x_i - x_j|^2 <
// 4 h_j^2 in the reference's distanceSq semantics for target j (rint minimum image when the 2h box of
// j leaves the periodic box).  Decided in FP32 on the grid form with a relative margin of 2^-17 (the
// grid-form d2 and the FP32 radius are within a few 2^-24 relative of the exact values); pairs inside
// the margin or crossing a periodic face take the exact FP64 test.
// i owns every non-mutual entry and half of its mutual ones: the mutual pair {i, j} belongs to the
// smaller index when i + j is odd and to the larger when it is even, so each particle owns about
// half of its mutual pairs wherever it sits in the SFC order; pairs within one warp of 32 targets
// (about 25 of a particle's 96) go to whichever end owns fewer (ownWithinWarp).  The owned entries are
// written compacted in the granule layout of the lists, entry = j | mutual << 31, the warp's own
// pairs last, with their count per particle.
struct MutualArgs {
    const double *x, *y, *z;
    const void* h;
    int hIsFloat;
    float u[3];
    DevBox box;
    int64_t first, last, stride;
    uint32_t ngmax;
    const uint32_t* nbr;
    const uint32_t* count;
    // one 32-byte block per particle (packGridBlock), one load per pair: grid position, then (2 h_j)^2 in
    // FP32, negative when the 2h box of j leaves the periodic box (j's search takes the minimum image:
    // no FP64 work per pair outside the rounding margin), then j's neighbour count (0 outside [first, last))
    const Rec8* rec;
    // (L/4)^2 of the smallest periodic box length (INFINITY without periodic axes): pairs whose
    // larger 2h exceeds L/4 are not evaluated once, because the legacy wrap of the pair loops
    // (threshold 2h of the list owner, box.hpp:216-238) may then pick different images at the two ends
    float wrapSafe2;
    uint32_t* owned;
    uint32_t* ownedCount;
    // rows of the pair-geometry cache: each warp's first, handed out from a counter in any order
    uint32_t* rowOff;
    uint32_t* rowCount;
};

__global__ void ownedRecKernel(const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, const void* h, int hIsFloat, int64_t n, DevBox b,
                               const u64* __restrict__ cell, const float4* __restrict__ loc,
                               const uint32_t* __restrict__ count, int64_t first, int64_t last,
                               float4* __restrict__ rec)
{
    const int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    const double hj = loadH(h, hIsFloat, j);
    const float tf = 2.f * float(hj);
    bool usePbc = false;
    if (b.pbc[0] | b.pbc[1] | b.pbc[2]) {  // the search's decision for target j (nbrGroupKernel)
        const double twoH = __dmul_rn(2.0, hj);
        const bool inside = __dsub_rn(x[j], twoH) >= b.lo[0] && __dsub_rn(y[j], twoH) >= b.lo[1] &&
                            __dsub_rn(z[j], twoH) >= b.lo[2] && __dadd_rn(x[j], twoH) <= b.hi[0] &&
                            __dadd_rn(y[j], twoH) <= b.hi[1] && __dadd_rn(z[j], twoH) <= b.hi[2];
        usePbc = !inside;
    }
    const uint32_t nc = j >= first && j < last ? count[j - first] : 0u;
    packGridBlock(rec + 2 * j, cell[j], loc[j], usePbc ? -(tf * tf) : tf * tf, __uint_as_float(nc), 0.f);
}

__device__ bool mutualExact(const MutualArgs& a, int64_t i, int64_t j, double hj)
{
    const DevBox& b = a.box;
    const double r2 = __dmul_rn(__dmul_rn(4.0, hj), hj);
    const double twoH = __dmul_rn(2.0, hj);
    const double xj = a.x[j], yj = a.y[j], zj = a.z[j];
    bool usePbc = false;
    if (b.pbc[0] | b.pbc[1] | b.pbc[2]) {
        const bool inside = __dsub_rn(xj, twoH) >= b.lo[0] && __dsub_rn(yj, twoH) >= b.lo[1] &&
                            __dsub_rn(zj, twoH) >= b.lo[2] && __dadd_rn(xj, twoH) <= b.hi[0] &&
                            __dadd_rn(yj, twoH) <= b.hi[1] && __dadd_rn(zj, twoH) <= b.hi[2];
        usePbc = !inside;
    }
    double dx = __dsub_rn(a.x[i], xj), dy = __dsub_rn(a.y[i], yj), dz = __dsub_rn(a.z[i], zj);
    if (usePbc) {
        if (b.pbc[0]) dx = foldRint(dx, b, 0);
        if (b.pbc[1]) dy = foldRint(dy, b, 1);
        if (b.pbc[2]) dz = foldRint(dz, b, 2);
    }
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return d2 < r2;
}

// i's own block bi, its cell ci unpacked
__device__ __forceinline__ bool mutualPair(const MutualArgs& a, int64_t i, const int ci[3], const Rec8& bi, int64_t j)
{
    if (j < a.first || j >= a.last) return false;
    const Rec8 bj = ldRec8(a.rec + j);
    if (__float_as_uint(bj.v[6]) > a.ngmax &&
        i > int64_t(__ldg(a.nbr + listSlot(j - a.first, a.ngmax - 1, a.stride))))
        return false;
    const float R2s = bj.v[5], R2j = fabsf(R2s);
    if (fmaxf(R2j, fabsf(bi.v[5])) > a.wrapSafe2) return false;
    int cj[3];
    unpackCell(u64(__float_as_uint(bj.v[0])) | (u64(__float_as_uint(bj.v[1])) << 32), cj);
    const float lv[3] = {bi.v[2] - bj.v[2], bi.v[3] - bj.v[3], bi.v[4] - bj.v[4]};
    constexpr int R = 1 << kGridBits;
    bool wrapped = false;
    float r[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int d = ci[k] - cj[k];
        if (a.box.pbc[k]) {
            if (d > R / 2) {
                d -= R;
                wrapped = true;
            } else if (d < -R / 2) {
                d += R;
                wrapped = true;
            }
        }
        r[k] = fmaf(float(d), a.u[k], lv[k]);
    }
    // across a periodic face only a target that takes the minimum image can list i
    if (wrapped && !(R2s < 0.f)) return false;
    const float d2 = fmaf(r[0], r[0], fmaf(r[1], r[1], r[2] * r[2]));
    const float eps = fmaf(0x1p-17f, R2j, kTinySq);
    if (d2 < R2j - eps) return true;
    if (d2 > R2j + eps) return false;
    return mutualExact(a, i, j, loadH(a.h, a.hIsFloat, j));
}

// the lanes among `intra` (the lane's mutual neighbours within its warp) that this lane owns: every
// pair of lanes meets in one of 31 steps and goes to the lane that owns fewer entries so far (on a tie
// by index parity).  The pair-once passes walk a warp's owned lists in step, so they take as long as
// the longest of the 32: with the parity rule alone that was 55 entries against a mean of 48.
__device__ __forceinline__ unsigned ownWithinWarp(unsigned intra, unsigned cnt, int lane)
{
    unsigned own = 0;
#pragma unroll 1
    for (int s = 1; s < kWarp; ++s) {
        const int p = lane ^ s;
        const unsigned theirs = __shfl_xor_sync(0xffffffffu, intra, s), theirCnt = __shfl_xor_sync(0xffffffffu, cnt, s);
        const bool odd = (s & 1) != 0, lower = lane < p;
        if ((intra >> p) & (theirs >> lane) & 1u) {
            const bool take = cnt < theirCnt || (cnt == theirCnt && odd == lower);
            own |= unsigned(take) << p;
            cnt += take;
        }
    }
    return own;
}

// one target's owned list: entries are offered in list order; mutual ones within the warp are kept
// back until the warp has shared them out in finish()
struct OwnedWriter {
    GranuleWriter out;
    int64_t ii, first;
    unsigned cnt = 0, intra = 0;
    __device__ __forceinline__ OwnedWriter(uint32_t* base, int64_t ii_, int64_t first_, int64_t stride, uint32_t ngmax)
        : out(base, ii_, stride, ngmax), ii(ii_), first(first_)
    {
    }
    __device__ __forceinline__ void offer(uint32_t j, bool mutual)
    {
        const int64_t jj = int64_t(j) - first;
        if (mutual && (jj >> 5) == (ii >> 5)) {
            intra |= 1u << (jj & 31);
            return;
        }
        const bool own = !mutual || ((((ii ^ jj) & 1) != 0) == (ii < jj));
        if (own) out.put(cnt++, j | (mutual ? 0x80000000u : 0u));
    }
    // all 32 lanes of the warp together
    __device__ __forceinline__ unsigned finish()
    {
        unsigned own = ownWithinWarp(intra, cnt, int(ii & 31));
        const uint32_t base = uint32_t(first + (ii & ~int64_t(31)));
        for (; own != 0; own &= own - 1u) out.put(cnt++, (base + unsigned(__ffs(own) - 1)) | 0x80000000u);
        out.finish(cnt);
        return cnt;
    }
};

__global__ void __launch_bounds__(128) ownedListKernel(MutualArgs a)
{
    const int64_t i = a.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    const bool valid = i < a.last;
    const int64_t ii = i - a.first;
    OwnedWriter w(a.owned, ii, a.first, a.stride, a.ngmax);
    if (valid) {
        const unsigned nc = min(__ldg(a.count + ii), a.ngmax);
        const Rec8 bi = ldRec8(a.rec + i);
        int ci[3];
        unpackCell(u64(__float_as_uint(bi.v[0])) | (u64(__float_as_uint(bi.v[1])) << 32), ci);
        const uint4* lists = reinterpret_cast<const uint4*>(a.nbr) + ii;
        uint4 G = make_uint4(0u, 0u, 0u, 0u);
        for (unsigned k = 0; k < nc; ++k) {
            if ((k & 3u) == 0u) G = __ldg(lists + int64_t(k / kListGran) * a.stride);
            const uint32_t j = pick(G, k & 3u);
            w.offer(j, mutualPair(a, i, ci, bi, j));
        }
    }
    const unsigned cnt = w.finish();
    if (valid) a.ownedCount[ii] = cnt;
    const unsigned rows = __reduce_max_sync(0xffffffffu, valid ? cnt : 0u);
    if (valid && (ii & 31) == 0) a.rowOff[ii >> 5] = atomicAdd(a.rowCount, rows);
}

// owned lists from list membership alone: (i, j) is mutual when i is in j's (capped, ascending)
// list, found by binary search, so the decision holds whatever the positions are now (frozen lists
// after moved particles).  A mutual pair goes by index parity: balanced lists (ownWithinWarp) gave the
// FP32 adjoint that walks these no time back, and FP32 sums in another order move its gradients by
// 4e-7, three times what two runs differ by.
__global__ void __launch_bounds__(128) ownedByListKernel(const uint32_t* __restrict__ nbr,
                                                         const uint32_t* __restrict__ count, int64_t first, int64_t last,
                                                         int64_t stride, uint32_t ngmax, uint32_t* __restrict__ owned,
                                                         uint32_t* __restrict__ ownedCount)
{
    const int64_t i = first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= last) return;
    const int64_t ii = i - first;
    const unsigned nc = min(__ldg(count + ii), ngmax);
    unsigned cnt = 0;
    GranuleWriter out(owned, ii, stride, ngmax);
    for (unsigned k = 0; k < nc; ++k) {
        const uint32_t j = __ldg(nbr + listSlot(ii, k, stride));
        bool m = false;
        if (int64_t(j) >= first && int64_t(j) < last) {
            const int64_t jj = int64_t(j) - first;
            unsigned lo = 0, hi = min(__ldg(count + jj), ngmax);  // search [lo, hi) of j's sorted list
            while (lo < hi) {
                const unsigned mid = (lo + hi) >> 1;
                const uint32_t e = __ldg(nbr + listSlot(jj, mid, stride));
                if (int64_t(e) < i) lo = mid + 1;
                else hi = mid;
            }
            m = lo < min(__ldg(count + jj), ngmax) && int64_t(__ldg(nbr + listSlot(jj, lo, stride))) == i;
        }
        const bool own = !m || ((((i ^ int64_t(j)) & 1) != 0) == (i < int64_t(j)));
        if (own) out.put(cnt++, j | (m ? 0x80000000u : 0u));
    }
    out.finish(cnt);
    ownedCount[ii] = cnt;
}

// ---- records of the std passes (PairRec) ----
// how many mutual pairs of each particle others own
__global__ void __launch_bounds__(128) inboxCountKernel(OwnedView ov, int64_t n, uint32_t* __restrict__ count)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const unsigned no = ov.size(i);
    for (unsigned k = 0; k < no; ++k) {
        bool mutual;
        const uint32_t j = ov.at(i, k, mutual);
        if (mutual) atomicAdd(count + j, 1u);
    }
}

// owner and record index of each of them, in any order (count runs down to 0)
__global__ void __launch_bounds__(128) inboxFillKernel(OwnedView ov, const uint32_t* __restrict__ rowOff, int64_t n,
                                                       const uint32_t* __restrict__ off, uint32_t* __restrict__ count,
                                                       uint2* __restrict__ entries)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const unsigned no = ov.size(i);
    const uint32_t base = 32u * __ldg(rowOff + (i >> 5)) + unsigned(i & 31);
    for (unsigned k = 0; k < no; ++k) {
        bool mutual;
        const uint32_t j = ov.at(i, k, mutual);
        if (mutual) entries[__ldg(off + j) + atomicSub(count + j, 1u) - 1u] = make_uint2(uint32_t(i), base + 32u * k);
    }
}

// the record indices by owner: one warp per particle, each entry's place is the number of smaller owners
__global__ void __launch_bounds__(128) inboxOrderKernel(int64_t n, const uint32_t* __restrict__ off,
                                                        const uint2* __restrict__ entries, uint32_t* __restrict__ inbox)
{
    const int64_t j = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / kWarp;
    if (j >= n) return;
    const unsigned lane = threadIdx.x % kWarp;
    const uint32_t o = off[j], m = off[j + 1] - o;
    if (m <= 2 * kWarp) {
        const uint2 none = make_uint2(0xffffffffu, 0u);
        const uint2 e0 = lane < m ? entries[o + lane] : none, e1 = lane + kWarp < m ? entries[o + lane + kWarp] : none;
        uint32_t b0 = 0, b1 = 0;
        const int m0 = int(min(m, uint32_t(kWarp))), m1 = int(m) - m0;
#pragma unroll 4
        for (int s = 0; s < m0; ++s) {
            const uint32_t q = __shfl_sync(0xffffffffu, e0.x, s);
            b0 += q < e0.x;
            b1 += q < e1.x;
        }
#pragma unroll 4
        for (int s = 0; s < m1; ++s) {
            const uint32_t q = __shfl_sync(0xffffffffu, e1.x, s);
            b0 += q < e0.x;
            b1 += q < e1.x;
        }
        if (lane < m) inbox[o + b0] = e0.y;
        if (lane + kWarp < m) inbox[o + b1] = e1.y;
        return;
    }
    for (uint32_t a0 = 0; a0 < m; a0 += kWarp) {
        const bool valid = a0 + lane < m;
        const uint2 e = valid ? entries[o + a0 + lane] : make_uint2(0u, 0u);
        uint32_t before = 0;
        for (uint32_t b0 = 0; b0 < m; b0 += kWarp) {
            const uint32_t other = b0 + lane < m ? entries[o + b0 + lane].x : 0xffffffffu;
            const int cnt = int(min(uint32_t(kWarp), m - b0));
            for (int s = 0; s < cnt; ++s) before += __shfl_sync(0xffffffffu, other, s) < e.x;
        }
        if (valid) inbox[o + before] = e.y;
    }
}

// Lanes lanes per particle share its records (g, g + Lanes, ...), their sums combined by shuffles; the lanes then
// add the own partial sums of one sum each.  Reads about 48 records per particle from anywhere: 32 bytes
// each, one sector.  Eight lanes in small sets, whose lists are serial chains; in large ones the adds of the shuffles
// cost more than the chains (1M particles: six sums 1.35 ms with eight lanes, 0.94 with two; four sums 0.75, and
// 0.56 with four).
template<int Sums, int Lanes>
__global__ void __launch_bounds__(256) gatherKernel(PairRec pr, int64_t n, const uint32_t* __restrict__ off,
                                                    const uint32_t* __restrict__ inbox, int slices,
                                                    double* __restrict__ acc)
{
    const int64_t t = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / Lanes;
    const unsigned g = threadIdx.x % Lanes;
    const bool valid = t < n;
    const int64_t j = valid ? t : 0;
    const uint32_t to = valid ? off[j + 1] : 0u;
    double s[Sums];
#pragma unroll
    for (int q = 0; q < Sums; ++q) s[q] = 0.0;
#pragma unroll 2
    for (uint32_t k = (valid ? off[j] : 0u) + g; k < to; k += Lanes) {
        const uint32_t e = __ldg(inbox + k);
        if constexpr (Sums == 1) {
            s[0] += __ldg(reinterpret_cast<const double*>(pr.rec) + e);
        } else {
            const Rec4d r = ldRec4d(pr.rec + e);
            if constexpr (Sums == 4) {
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] += r.v[q];
            } else {
                const double x = r.v[0], y = r.v[1], z = r.v[2], fx = r.v[3] * x, fy = r.v[3] * y, fz = r.v[3] * z;
                s[0] = fma(fx, x, s[0]);
                s[1] = fma(fx, y, s[1]);
                s[2] = fma(fx, z, s[2]);
                s[3] = fma(fy, y, s[3]);
                s[4] = fma(fy, z, s[4]);
                s[5] = fma(fz, z, s[5]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < Sums; ++q)
#pragma unroll
        for (int o = Lanes / 2; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    if (!valid) return;
#pragma unroll
    for (int q = 0; q < Sums; ++q)
        if (g == unsigned(q % Lanes)) {
            double v = 0.0;
            for (int l = 0; l < slices; ++l) v += pr.part[(int64_t(l) * Sums + q) * n + j];
            acc[int64_t(q) * n + j] = v + s[q];
        }
}

__global__ void fillOnes(uint32_t* p, int64_t n)
{
    int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k < n) p[k] = 1u;
}

// grid form of all particles' positions (cells + FP32 offsets), shared with the mixed passes
__global__ void gridFormKernel(const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, int64_t n, DevBox box, u64* __restrict__ cell,
                               float4* __restrict__ loc)
{
    int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const double c[3] = {x[i], y[i], z[i]};
    unsigned ic[3];
    float l[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // cell = floor((x - lo) / u) by a multiply: a cell off by one near a boundary only gives an
        // offset just outside [0, u), which the FP32 offset still holds to 2^-24 of u
        double u = box.L[k] / double(1 << kGridBits);
        double g = floor((c[k] - box.lo[k]) * (double(1 << kGridBits) * box.iL[k]));
        g = fmin(fmax(g, 0.0), double(kGridMask));
        ic[k] = unsigned(g);
        l[k] = float(c[k] - (box.lo[k] + g * u));
    }
    cell[i] = u64(ic[0]) | (u64(ic[1]) << kGridBits) | (u64(ic[2]) << (2 * kGridBits));
    loc[i] = make_float4(l[0], l[1], l[2], 0.f);
}

int runSearch(sphgb_ctx* c, const double* x, const double* y, const double* z, const void* h, int hIsFloat,
              int64_t first, int64_t last, uint32_t ngmax, const uint32_t* active)
{
    NbrArgs a;
    a.x = x;
    a.y = y;
    a.z = z;
    a.h = h;
    a.hIsFloat = hIsFloat;
    a.cell = c->gridKey.as<u64>();
    a.loc = c->gridLoc.as<float4>();
    for (int k = 0; k < 3; ++k) {
        a.u[k] = float(c->box.L[k] / double(1 << kGridBits));
        a.sh[k] = c->box.pbc[k] ? 32 - kGridBits : 0;
    }
    // boxes beyond 2^+-30 are pruned in units of their own size: squares of lengths below 1e-19 or above 1e19
    // would underflow or overflow, and every node would be walked
    const double longest = std::max(c->box.L[0], std::max(c->box.L[1], c->box.L[2]));
    const int e = longest > 0.0 && std::isfinite(longest) ? std::ilogb(longest) : 0;
    a.pruneUnit = std::abs(e) > 30 ? float(std::ldexp(1.0, std::min(126, std::max(-126, -e)))) : 1.f;
    a.first = first;
    a.last = last;
    a.active = active;
    a.childOffsets = c->childOffsets.as<int32_t>();
    a.nodeBox = c->nodeBoxF.as<float4>();
    a.nodeRange = c->nodeRange.as<uint2>();
    a.box = c->box;
    a.ngmax = ngmax;
    a.stride = c->nbrStride;
    a.nbr = c->nbr.as<uint32_t>();
    a.count = c->ncount.as<uint32_t>();
    a.flags = c->dFlags;
    a.stats = c->counters.as<unsigned long long>();
    int64_t groups = (last - first + kWarp - 1) / kWarp;
    unsigned blocks = unsigned((groups + kWarpsPerBlock - 1) / kWarpsPerBlock);
    if (c->n < kFoldBelow) nbrGroupKernel<true><<<blocks, kNbrBlock, 0, c->stream>>>(a);
    else nbrGroupKernel<false><<<blocks, kNbrBlock, 0, c->stream>>>(a);
    return launched(c, "nbrGroupKernel");
}

int buildOwned(sphgb_ctx* c, const double* x, const double* y, const double* z, const void* h, int hIsFloat)
{
    const int64_t nWork = c->nbrLast - c->nbrFirst;
    SPHGB_TRY(c->owned.ensure(sizeof(uint32_t) * listCapacity(c->nbrNgmax) * size_t(c->nbrStride)));
    SPHGB_TRY(c->ownedCount.ensure(sizeof(uint32_t) * size_t(c->nbrStride)));
    SPHGB_TRY(c->pack.ensure(sizeof(Rec8) * size_t(c->n)));  // the pair passes' records: free here
    ownedRecKernel<<<gridFor(c->n, 256), 256, 0, c->stream>>>(x, y, z, h, hIsFloat, c->n, c->box, c->gridKey.as<u64>(),
                                                              c->gridLoc.as<float4>(), c->ncount.as<uint32_t>(),
                                                              c->nbrFirst, c->nbrLast, c->pack.as<float4>());
    SPHGB_TRY(launched(c, "ownedRecKernel"));
    MutualArgs a;
    a.x = x;
    a.y = y;
    a.z = z;
    a.h = h;
    a.hIsFloat = hIsFloat;
    for (int k = 0; k < 3; ++k) a.u[k] = float(c->box.L[k] / double(1 << kGridBits));
    a.box = c->box;
    a.first = c->nbrFirst;
    a.last = c->nbrLast;
    a.stride = c->nbrStride;
    a.ngmax = c->nbrNgmax;
    a.nbr = c->nbr.as<uint32_t>();
    a.count = c->ncount.as<uint32_t>();
    a.rec = c->pack.as<Rec8>();
    a.wrapSafe2 = INFINITY;
    for (int k = 0; k < 3; ++k)
        if (c->box.pbc[k]) a.wrapSafe2 = std::min(a.wrapSafe2, float(0.0625 * c->box.L[k] * c->box.L[k]));
    a.owned = c->owned.as<uint32_t>();
    a.ownedCount = c->ownedCount.as<uint32_t>();
    const int64_t nWarps = (nWork + 31) / 32;
    SPHGB_TRY(c->geoRows.ensure(sizeof(uint32_t) * size_t(nWarps + 1)));
    a.rowOff = c->geoRows.as<uint32_t>();
    a.rowCount = a.rowOff + nWarps;
    SPHGB_CUDA(cudaMemsetAsync(a.rowCount, 0, sizeof(uint32_t), c->stream));
    ownedListKernel<<<gridFor(nWork, 128), 128, 0, c->stream>>>(a);
    SPHGB_TRY(launched(c, "ownedListKernel"));
    uint32_t rows = 0;
    SPHGB_CUDA(cudaMemcpyAsync(&rows, a.rowCount, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
    SPHGB_CUDA(cudaStreamSynchronize(c->stream));
    c->geoRowCount = rows;
    c->ownedEpoch = c->nbrEpoch;
    c->ownedFromLists = false;
    return SPHGB_OK;
}

int prepareLists(sphgb_ctx* c, const double* x, const double* y, const double* z, int64_t first, int64_t last,
                 uint32_t ngmax)
{
    if (!c->haveTree) return SPHGB_ERR_STATE;
    if (first < 0 || last > c->n || first >= last) return SPHGB_ERR_ARG;
    const int64_t nWork = last - first;
    c->nbrStride = (nWork + 31) / 32 * 32;
    // lists larger than the buffers hold: the pair-geometry cache of an earlier sweep gives its
    // memory back first (the next FP64 sweep sizes it again within half of the free memory)
    if (c->nbr.bytes < sizeof(uint32_t) * listCapacity(ngmax) * c->nbrStride) {
        c->dropPairGeo();
        c->dropPairRec();
    }
    SPHGB_TRY(c->nbr.ensure(sizeof(uint32_t) * listCapacity(ngmax) * c->nbrStride));
    SPHGB_TRY(c->ncount.ensure(sizeof(uint32_t) * c->nbrStride));
    SPHGB_TRY(c->active.ensure(sizeof(uint32_t) * c->nbrStride + c->nbrStride));
    SPHGB_TRY(c->counters.ensure(sizeof(unsigned long long) * 8));
    SPHGB_CUDA(cudaMemsetAsync(c->counters.p, 0, sizeof(unsigned long long) * 8, c->stream));
    SPHGB_CUDA(cudaMemsetAsync(c->dFlags, 0, sizeof(int), c->stream));
    // grid form of every particle (neighbours may be anywhere in [0, n))
    SPHGB_TRY(c->gridKey.ensure(sizeof(u64) * c->n));
    SPHGB_TRY(c->gridLoc.ensure(sizeof(float4) * c->n));
    gridFormKernel<<<gridFor(c->n, 256), 256, 0, c->stream>>>(x, y, z, c->n, c->box, c->gridKey.as<u64>(),
                                                             c->gridLoc.as<float4>());
    SPHGB_TRY(launched(c, "gridFormKernel"));
    c->nbrFirst = first;
    c->nbrLast = last;
    c->nbrNgmax = ngmax;
    return SPHGB_OK;
}

int finishStats(sphgb_ctx* c, int64_t hIters)
{
    unsigned long long h[8];
    int flags = 0;
    SPHGB_CUDA(cudaMemcpyAsync(h, c->counters.p, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    SPHGB_CUDA(cudaMemcpyAsync(&flags, c->dFlags, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SPHGB_CUDA(cudaStreamSynchronize(c->stream));
    c->stats.candidates = int64_t(h[0]);
    c->stats.fp64_rechecks = int64_t(h[1]);
    c->stats.nc_sum = int64_t(h[3]);
    c->stats.capped = int64_t(h[4]);
    c->stats.nc_max = uint32_t(h[5]);
    c->stats.h_fails = int64_t(h[6]);
    c->stats.h_iterations = hIters;
    if (flags & kFlagStackOverflow) return SPHGB_ERR_TRAVERSAL;
    return SPHGB_OK;
}

}  // namespace

int pairGeoStore(sphgb_ctx* c, const sphgb_particles* p, PairGeo* out)
{
    *out = PairGeo{};
    c->geoValid = false;
    c->geoSnapEpoch = -1;
    c->geoArrays = 0;
    // a caller that repeats the first pass alone (densities of many sets, a search for h) pays for the store and
    // has nothing from it (512k particles: xmass 1.57 ms with it, 1.23 without): after two stores that no pass
    // read there are no more until one asks
    if (!c->inSweep && c->geoUnread >= 2) return SPHGB_OK;
    if (c->ownedEpoch != c->nbrEpoch || c->ownedFromLists || !p->vx || !p->vy || !p->vz) return SPHGB_OK;
    const size_t rows = c->geoRowCount;
    if (rows == 0 || c->geoLimit == 0) return SPHGB_OK;
    if (!c->inSweep) {
        if (c->geoSnap.ensure(sizeof(double) * kGeoInputs * size_t(p->n)) != SPHGB_OK ||
            c->geoStale.ensure(sizeof(int)) != SPHGB_OK) {
            (void)cudaGetLastError();
            return SPHGB_OK;
        }
    }
    // five arrays (|r| and w_ij, the two kernel values, r and dv) or the first two, whichever fits
    // in the buffer already held, in half of the free device memory inside a sweep, or in an eighth of it
    // outside (a caller that makes the passes one by one allocates more of its own between them; 8M particles
    // take 33 GB, an eighth of an empty device)
    const size_t share = c->inSweep ? 2 : 8;
    int arrays = 0;
    for (int a : {5, 2}) {
        if (a > c->geoLimit) continue;
        const size_t need = size_t(a) * 32 * sizeof(double2) * rows;
        if (c->pairGeo.bytes >= need) {
            arrays = a;
            break;
        }
        // the rows change a little with every search of a moving set: 3 % more than asked for, where that fits
        size_t freeB = 0, totalB = 0;
        if (cudaMemGetInfo(&freeB, &totalB) != cudaSuccess) continue;
        const size_t most = (freeB + c->pairGeo.bytes) / share, padded = need + need / 32;
        if (need > most) continue;
        const bool got = (padded <= most && c->pairGeo.ensure(padded) == SPHGB_OK) || c->pairGeo.ensure(need) == SPHGB_OK;
        (void)cudaGetLastError();  // of an attempt that failed
        if (!got) continue;
        ++c->geoAllocs;
        arrays = a;
        break;
    }
    if (arrays == 0) return SPHGB_OK;
    c->geoArrays = arrays;
    if (c->inSweep) c->geoValid = true;
    else {
        ++c->geoUnread;
        c->geoSnapEpoch = c->nbrEpoch;
        c->geoSnapN = p->n;
    }
    *out = pairGeoView(c, nullptr);
    return SPHGB_OK;
}

int pairRecords(sphgb_ctx* c, double* part, PairRec* out)
{
    *out = PairRec{};
    const size_t rows = c->geoRowCount, slots = 32 * rows;
    const int64_t n = c->nbrLast - c->nbrFirst;
    if (rows == 0 || rows >= (size_t(1) << 27)) return SPHGB_OK;
    if (c->inboxEpoch != c->nbrEpoch) {
        SPHGB_TRY(c->inboxCount.ensure(sizeof(uint32_t) * size_t(n + 1)));
        SPHGB_TRY(c->inboxOff.ensure(sizeof(uint32_t) * size_t(n + 1)));
        uint32_t *count = c->inboxCount.as<uint32_t>(), *off = c->inboxOff.as<uint32_t>();
        SPHGB_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t) * size_t(n + 1), c->stream));
        const OwnedView ov = ownedView(c);
        inboxCountKernel<<<gridFor(n, 128), 128, 0, c->stream>>>(ov, n, count);
        SPHGB_TRY(launched(c, "inboxCountKernel"));
        SPHGB_TRY(exclusiveScan(c, count, off, n + 1));
        // the space after everything that may take it back; 3 % more than asked for, as for the cache
        if (c->pairRec.bytes < sizeof(Rec4d) * slots || c->inbox.bytes < sizeof(uint32_t) * slots) {
            const size_t padded = slots + slots / 32, need = (sizeof(Rec4d) + sizeof(uint32_t)) * padded;
            size_t freeB = 0, totalB = 0;
            if (cudaMemGetInfo(&freeB, &totalB) != cudaSuccess ||
                need > (freeB + c->pairRec.bytes + c->inbox.bytes) / (c->inSweep ? 2 : 8) ||
                c->pairRec.ensure(sizeof(Rec4d) * padded) != SPHGB_OK ||
                c->inbox.ensure(sizeof(uint32_t) * padded) != SPHGB_OK) {
                (void)cudaGetLastError();
                c->dropPairRec();
                return SPHGB_OK;
            }
        }
        inboxFillKernel<<<gridFor(n, 128), 128, 0, c->stream>>>(ov, c->geoRows.as<uint32_t>(), n, off, count,
                                                                c->pairRec.as<uint2>());
        SPHGB_TRY(launched(c, "inboxFillKernel"));
        inboxOrderKernel<<<gridFor(n * kWarp, 128), 128, 0, c->stream>>>(n, off, c->pairRec.as<uint2>(),
                                                                         c->inbox.as<uint32_t>());
        SPHGB_TRY(launched(c, "inboxOrderKernel"));
        c->inboxEpoch = c->nbrEpoch;
    }
    *out = PairRec{c->geoRows.as<uint32_t>(), c->pairRec.as<Rec4d>(), part};
    return SPHGB_OK;
}

int gatherRecords(sphgb_ctx* c, const PairRec& pr, int64_t n, int sums, int slices, double* acc)
{
    const uint32_t *off = c->inboxOff.as<uint32_t>(), *inbox = c->inbox.as<uint32_t>();
    auto run = [&](auto kernel, int lanes) {
        kernel<<<gridFor(n * lanes, 256), 256, 0, c->stream>>>(pr, n, off, inbox, slices, acc);
    };
    const bool small = slices > 1;
    if (sums == 1) small ? run(gatherKernel<1, 8>, 8) : run(gatherKernel<1, 4>, 4);
    else if (sums == 4) small ? run(gatherKernel<4, 8>, 8) : run(gatherKernel<4, 4>, 4);
    else small ? run(gatherKernel<6, 8>, 8) : run(gatherKernel<6, 2>, 2);
    return launched(c, "gatherKernel");
}

int buildOwnedFromLists(sphgb_ctx* c)
{
    const int64_t nWork = c->nbrLast - c->nbrFirst;
    SPHGB_TRY(c->owned.ensure(sizeof(uint32_t) * listCapacity(c->nbrNgmax) * size_t(c->nbrStride)));
    SPHGB_TRY(c->ownedCount.ensure(sizeof(uint32_t) * size_t(c->nbrStride)));
    ownedByListKernel<<<gridFor(nWork, 128), 128, 0, c->stream>>>(c->nbr.as<uint32_t>(), c->ncount.as<uint32_t>(),
                                                                 c->nbrFirst, c->nbrLast, c->nbrStride, c->nbrNgmax,
                                                                 c->owned.as<uint32_t>(), c->ownedCount.as<uint32_t>());
    SPHGB_TRY(launched(c, "ownedByListKernel"));
    c->ownedEpoch = c->nbrEpoch;
    c->ownedFromLists = true;
    return SPHGB_OK;
}

int findNeighborsSph(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    if (!p->x || !p->y || !p->z || !p->h) return SPHGB_ERR_ARG;
    const uint32_t ngmax = c->prm.ngmax;
    if (c->prm.ng0 > ngmax) return SPHGB_ERR_ARG;  // reference: "ng0 should be smaller than ngmax"
    if (!c->haveTree) return SPHGB_ERR_STATE;
    if (!c->inputsChecked)
        SPHGB_TRY(validateParticles(c, p->x, p->y, p->z, p->h, p->precision == SPHGB_MIXED, c->n));
    SPHGB_TRY(prepareLists(c, p->x, p->y, p->z, first, last, ngmax));
    const int64_t nWork = last - first;
    const int hf = p->precision == SPHGB_MIXED;
    uint32_t* active = c->active.as<uint32_t>();
    uint8_t* iters = reinterpret_cast<uint8_t*>(active + c->nbrStride);
    SPHGB_CUDA(cudaMemsetAsync(iters, 0, c->nbrStride, c->stream));
    SPHGB_TRY(runSearch(c, p->x, p->y, p->z, p->h, hf, first, last, ngmax, nullptr));

    unsigned long long* ctr = c->counters.as<unsigned long long>();
    fillOnes<<<gridFor(nWork, 256), 256, 0, c->stream>>>(active, nWork);
    SPHGB_TRY(launched(c, "fillOnes"));
    int64_t rounds = 0;
    for (int it = 0; it < 10; ++it) {
        SPHGB_CUDA(cudaMemsetAsync(ctr + 2, 0, sizeof(unsigned long long), c->stream));
        if (hf)
            hIterKernel<float><<<gridFor(nWork, 256), 256, 0, c->stream>>>(
                c->ncount.as<uint32_t>(), static_cast<float*>(p->h), active, iters, first, nWork, c->prm.ng0, ngmax,
                ctr);
        else
            hIterKernel<double><<<gridFor(nWork, 256), 256, 0, c->stream>>>(
                c->ncount.as<uint32_t>(), static_cast<double*>(p->h), active, iters, first, nWork, c->prm.ng0, ngmax,
                ctr);
        SPHGB_TRY(launched(c, "hIterKernel"));
        unsigned long long nact = 0;
        SPHGB_CUDA(cudaMemcpyAsync(&nact, ctr + 2, sizeof(nact), cudaMemcpyDeviceToHost, c->stream));
        SPHGB_CUDA(cudaStreamSynchronize(c->stream));
        if (nact == 0) break;
        ++rounds;
        SPHGB_TRY(runSearch(c, p->x, p->y, p->z, p->h, hf, first, last, ngmax, active));
    }
    ncOutKernel<<<gridFor(nWork, kNcOutBlock), kNcOutBlock, 0, c->stream>>>(c->ncount.as<uint32_t>(), iters, nWork, ngmax,
                                                             p->nc ? p->nc + first : nullptr, 1, ctr);
    SPHGB_TRY(launched(c, "ncOutKernel"));
    SPHGB_TRY(finishStats(c, rounds));
    c->nbrEpoch++;
    c->haveNbr = true;
    c->precisionBuilt = p->precision;
    c->xBuilt = p->x;
    // the pair-once FP64 momentum-energy pass reads the owned lists; the mixed passes do not
    if (p->precision == SPHGB_FP64) SPHGB_TRY(buildOwned(c, p->x, p->y, p->z, p->h, hf));
    return c->stats.h_fails > 0 ? SPHGB_ERR_NOCONV : SPHGB_OK;
}

int findNeighborsFixed(sphgb_ctx* c, const double* x, const double* y, const double* z, const void* h, int32_t hPrec,
                       int64_t first, int64_t last, uint32_t ngmax, uint32_t* nbrOut, uint32_t* ncOut)
{
    if (!x || !y || !z || !h || ngmax == 0) return SPHGB_ERR_ARG;
    if (!c->haveTree) return SPHGB_ERR_STATE;
    SPHGB_TRY(validateParticles(c, x, y, z, h, hPrec == SPHGB_MIXED, c->n));
    SPHGB_TRY(prepareLists(c, x, y, z, first, last, ngmax));
    const int64_t nWork = last - first;
    SPHGB_TRY(runSearch(c, x, y, z, h, hPrec == SPHGB_MIXED, first, last, ngmax, nullptr));
    ncOutKernel<<<gridFor(nWork, kNcOutBlock), kNcOutBlock, 0, c->stream>>>(c->ncount.as<uint32_t>(), nullptr, nWork, ngmax, ncOut, 0,
                                                             c->counters.as<unsigned long long>());
    SPHGB_TRY(launched(c, "ncOutKernel"));
    if (nbrOut) {
        exportKernel<<<gridFor(nWork, 32 * kExportWarps), 32 * kExportWarps, 0, c->stream>>>(c->nbr.as<uint32_t>(), c->ncount.as<uint32_t>(),
                                                                  nWork, c->nbrStride, ngmax, nbrOut);
        SPHGB_TRY(launched(c, "exportKernel"));
    }
    SPHGB_TRY(finishStats(c, 0));
    c->nbrEpoch++;
    c->haveNbr = true;
    c->precisionBuilt = hPrec;
    c->xBuilt = x;
    if (hPrec == SPHGB_FP64) SPHGB_TRY(buildOwned(c, x, y, z, h, 0));
    return SPHGB_OK;
}

int exportNeighbors(sphgb_ctx* c, uint32_t* out)
{
    if (!c->haveNbr) return SPHGB_ERR_STATE;
    if (!out) return SPHGB_ERR_ARG;
    const int64_t nWork = c->nbrLast - c->nbrFirst;
    exportKernel<<<gridFor(nWork, 32 * kExportWarps), 32 * kExportWarps, 0, c->stream>>>(c->nbr.as<uint32_t>(), c->ncount.as<uint32_t>(), nWork,
                                                              c->nbrStride, c->nbrNgmax, out);
    SPHGB_TRY(launched(c, "exportKernel"));
    SPHGB_CUDA(cudaStreamSynchronize(c->stream));
    return SPHGB_OK;
}

}  // namespace sphgb

// Neighbour build, mesh contact collection, friction-history merge, contact
// law and the deterministic force gather.
//
// Contact order is canonical and equal to the reference CPU collector's
// (cpu_scheduling.slang:53-91): pair index, then direction, then leaf cluster
// in preorder, then node in meshSampleIndices order.  The collector keeps it
// with no atomics on contact slots: a flat leaf cull per directed pair, an
// exclusive scan to (directed pair, leaf) work items, a filter per item (a
// ballot mask of its nodes), a scan to surviving nodes and a scan to the stored
// exact-query slots, which are therefore in contact order.  A step queries the
// slots that are awake and marks its hits as bits; a hit's contact index is the
// number of hit bits before it.  The history merge and the gather then walk
// sorted runs instead of a hash table and linked lists, so every run is
// reproducible bit for bit.
//
// Every phase is a device function: kernels_contacts.cu launches each as a
// kernel, run_device.cuh runs them all in one.
#pragma once
#include <cuda_runtime.h>
#include "culler.cuh"
#include "launch.h"
#include "state_device.cuh"

namespace sdg {

constexpr uint32_t WARP = 32;
__device__ __forceinline__ uint32_t laneId() { return threadIdx.x & 31u; }
__device__ __forceinline__ uint32_t warpGlobal() { return warpIndex(); }
__device__ __forceinline__ uint32_t warpStride() { return (gridDim.x * blockDim.x) >> 5; }
__device__ __forceinline__ uint32_t lanesBelow() { return (1u << laneId()) - 1u; }

// ------------------------------------------------------------------- scan
__device__ __forceinline__ uint32_t scanCount(const ScanCount& c) {
    if (!c.ptr) return c.constant;
    uint32_t v = *c.ptr;
    return (v < c.cap ? v : c.cap) * c.mul;
}
__device__ __forceinline__ uint32_t blockInclusive(uint32_t v, uint32_t* shared) {
    // 256 threads: warp scans, then a scan of the 8 warp totals.
    uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) shared[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (blockDim.x >> 5) ? shared[lane] : 0;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < (blockDim.x >> 5)) shared[lane] = w;
    }
    __syncthreads();
    uint32_t add = warp ? shared[warp - 1] : 0;
    __syncthreads();
    return v + add;
}

// ------------------------------------------------------------ neighbours
// solver.slang:184-186
// Bin grid of a specimen: sb = (bins x, y, z, first bin of the specimen).
__device__ __forceinline__ void binIndex(const Res& r, uint32_t i, uint4 sb, float4 box, uint32_t b[3]) {
    float4 p = r.position[i];
    uint32_t bins[3] = {sb.x, sb.y, sb.z};
    float g[3] = {floorf(__fmul_rn(__fdiv_rn(p.x, box.x), float(sb.x))),
                  floorf(__fmul_rn(__fdiv_rn(p.y, box.y), float(sb.y))),
                  floorf(__fmul_rn(__fdiv_rn(p.z, box.z), float(sb.z)))};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        uint32_t v = uint32_t(g[k]);
        b[k] = v < bins[k] - 1 ? v : bins[k] - 1;
    }
}
__device__ __forceinline__ uint32_t binFlat(uint4 sb, const uint32_t b[3]) {
    return sb.w + (b[0] * sb.y + b[1]) * sb.z + b[2];
}
__device__ __forceinline__ uint32_t modIndex(int a, uint32_t n) { return uint32_t((a % int(n) + int(n)) % int(n)); }

__device__ __forceinline__ void binsClear(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    for (uint32_t b = gtid(); b < P.c.binCount; b += gstride()) r.binCounts[b] = 0;
}
// solver.slang:350-359
__device__ __forceinline__ void binGrain(const Params& P, uint32_t id) {
    const Res& r = P.r;
    const Config& c = P.c;
    f3 p = xyz(r.position[id]), pl = xyz(r.positionRemainder[id]);
    if (!finite3(p) || !finite3(pl)) { fail(r, F_NONFINITE); return; }
    uint32_t sp = specimenOf(r, id);
    float4 cell = r.cell[3 * sp];
    if (c.periodic == 0) {
        f3 box = xyz(cell);
        if (__fadd_rn(p.x, pl.x) < 0 || __fadd_rn(p.y, pl.y) < 0 || __fadd_rn(p.z, pl.z) < 0 ||
            __fadd_rn(__fsub_rn(p.x, box.x), pl.x) >= 0 || __fadd_rn(__fsub_rn(p.y, box.y), pl.y) >= 0 ||
            __fadd_rn(__fsub_rn(p.z, box.z), pl.z) >= 0) { fail(r, F_ESCAPE); return; }
    }
    uint32_t b[3];
    uint4 sb = r.specimenBins[sp];
    binIndex(r, id, sb, cell, b);
    uint32_t bin = binFlat(sb, b);
    uint32_t slot = atomicAdd(&r.binCounts[bin], 1u);
    if (slot < c.binCapacity) r.binParticles[bin * c.binCapacity + slot] = id;
    else fail(r, F_BIN);
}
__device__ __forceinline__ void binsFill(const Params& P) {
    if (P.r.control[4] == 0) return;
    for (uint32_t id = gtid(); id < P.c.N; id += gstride()) binGrain(P, id);
}
// Ascending bitonic sort of n words in place, by a warp.  Every merge starts
// with mirrored places and then only takes the smaller word down: places past
// an n that is no power of two stand for words above all others and are left
// out.
__device__ __forceinline__ void sortWarp(uint32_t* v, uint32_t n) {
    for (uint32_t size = 2; size < 2 * n; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t k = laneId();; k += WARP) {
                const uint32_t low = 2 * k - (k & (stride - 1));
                if (low >= n) break;
                const uint32_t high = stride == size >> 1 ? low ^ (size - 1) : low + stride;
                if (high >= n) continue;
                const uint32_t a = v[low], b = v[high];
                if (a > b) {
                    v[low] = b;
                    v[high] = a;
                }
            }
            __syncwarp();
        }
    }
}
// The same order by a warp per bin without shared memory (the persistent
// step's small bins): each lane ranks its grains among the bin's, all read
// before any is written.  Up to four grains a lane keep their ranks in
// registers; larger bins (few and full: a wide range of sizes) are sorted in
// place.  A step that builds bins of 460 takes 0.35 ms (launched: 0.53), of 1,281
// 0.92 (0.93); with one lane's insertion instead, quadratic, 2.9 and 16.4.
__device__ __forceinline__ void binsOrder(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    for (uint32_t bin = warpGlobal(); bin < c.binCount; bin += warpStride()) {
        const uint32_t occ = min(r.binCounts[bin], c.binCapacity);
        uint32_t* slots = r.binParticles + size_t(bin) * c.binCapacity;
        if (occ > 128) {
            sortWarp(slots, occ);
            continue;
        }
        uint32_t id[4], rank[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            id[j] = laneId() + 32 * j < occ ? slots[laneId() + 32 * j] : EMPTY;
            rank[j] = 0;
        }
        for (uint32_t k = 0; k < occ; ++k) {
            const uint32_t v = slots[k];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) rank[j] += v < id[j];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (id[j] != EMPTY) slots[rank[j]] = id[j];
        __syncwarp();
    }
}
// ---- radix-sorted cell list (solver.slang:345-359 fills the bins serially,
// in grain order; a stable sort of the grains by bin gives the same slots).
// Keys are the flat bin indices (a grain that fails the checks gets
// binCount, past every bin); an LSD radix sort of 8-bit digits (stable:
// each pass keeps the order of equal digits) orders (bin, grain) pairs, and
// each bin's run is then copied into the reference's fixed-capacity slots.
// The scratch lives in byJPairs (pair ids by second grain), which the
// neighbour build rewrites only after the pairs exist: keys and grains twice
// (ping-pong) and the per-(digit, tile) counts.
constexpr uint32_t RADIX = 256, RADIX_ITEMS = 8, RADIX_TILE = 256 * RADIX_ITEMS;
struct RadixScratch {
    uint32_t *keys[2], *vals[2], *counts;
    uint32_t tiles;
};
__host__ __device__ __forceinline__ uint32_t radixTiles(uint32_t n) { return (n + RADIX_TILE - 1) / RADIX_TILE; }
// Words of byJPairs the sort needs (the radix path runs only where they fit).
__host__ __device__ __forceinline__ uint64_t radixWords(uint32_t n) {
    return 4ull * n + uint64_t(RADIX) * radixTiles(n) + 1;
}
__host__ __device__ __forceinline__ RadixScratch radixScratch(const Res& r, const Config& c) {
    uint32_t* base = r.byJPairs;
    RadixScratch x;
    x.keys[0] = base;
    x.vals[0] = base + c.N;
    x.keys[1] = base + 2 * size_t(c.N);
    x.vals[1] = base + 3 * size_t(c.N);
    x.counts = base + 4 * size_t(c.N);
    x.tiles = radixTiles(c.N);
    return x;
}
// solver.slang:360-392: the pair search, a warp per grain with ballot
// compaction.  An FP32 minimum-image estimate settles the grains clearly
// beyond or within range; the exact FP64 branch decides the rest.  The grain's
// stencil bins (the reference's x, y, z order) are taken 32 at a time, one
// per lane with its occupancy; their slots form one candidate sequence in
// the reference's order (bin, then slot), which the lanes test 32 at a time
// (the FP32 estimate, then the exact FP64 branch).  A ballot of the passing
// candidates counts them or, in the emit pass, gives each its place in
// order: the pair list is the serial search's, pair for pair.  The counting
// pass keeps a grain's first pairRoom partners in its row of byJPairs (free until
// the pairs exist), so the emit pass copies them and searches again only for a
// grain with more: 50,000 grains of uneven size, search and emit 1,081 -> 324 us.
__device__ __forceinline__ uint32_t pairRoom(const Config& c) { return c.pairCapacity / c.N; }
template <bool Emit>
__device__ __forceinline__ void findPairsWarp(const Res& r, const Config& c, uint32_t id) {
    const uint32_t lane = laneId();
    uint32_t sp = specimenOf(r, id);
    uint4 sb = r.specimenBins[sp];
    uint32_t bins[3] = {sb.x, sb.y, sb.z};
    float4 cell = r.cell[3 * sp];
    uint32_t b[3];
    binIndex(r, id, sb, cell, b);
    float cutoff = r.referenceCell[2 * sp + 1].w;
    float box[3] = {cell.x, cell.y, cell.z};
    const float perBox[3] = {1.0f / cell.x, 1.0f / cell.y, 1.0f / cell.z};
    int reach[3], low[3];
    uint32_t width[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        reach[k] = int(ceilf(__fmul_rn(__fdiv_rn(cutoff, box[k]), float(bins[k]))));
        low[k] = max(int(b[k]) - reach[k], 0);
        int high = min(int(b[k]) + reach[k], int(bins[k]) - 1);
        uint32_t w = uint32_t(2 * reach[k] + 1);
        width[k] = c.periodic != 0 ? min(w, bins[k]) : uint32_t(high - low[k] + 1);
    }
    float4 pi = r.position[id], li = r.positionRemainder[id];
    float ri = r.body[id].z;
    uint32_t stencil = width[0] * width[1] * width[2];
    const uint32_t room = pairRoom(c);
    uint32_t count = 0, base = Emit ? r.pairOffsets[id] : 0u;
    for (uint32_t q0 = 0; q0 < stencil; q0 += 32) {
        // Lane q: stencil bin q0 + q (x slowest, z fastest) and its occupancy.
        uint32_t q = q0 + lane, bin = 0, occ = 0;
        if (q < stencil) {
            uint32_t z = q % width[2], y = (q / width[2]) % width[1], x = q / (width[2] * width[1]);
            uint32_t cc[3];
            if (c.periodic != 0) {
                cc[0] = modIndex(int(b[0]) - reach[0] + int(x), bins[0]);
                cc[1] = modIndex(int(b[1]) - reach[1] + int(y), bins[1]);
                cc[2] = modIndex(int(b[2]) - reach[2] + int(z), bins[2]);
            } else {
                cc[0] = uint32_t(low[0] + int(x));
                cc[1] = uint32_t(low[1] + int(y));
                cc[2] = uint32_t(low[2] + int(z));
            }
            bin = binFlat(sb, cc) * c.binCapacity;
            const uint32_t end = min(r.binCounts[binFlat(sb, cc)], c.binCapacity);
            // Grains above this one only: the end of the bin, which is in id order.
            uint32_t lo = 0, hi = end;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (r.binParticles[bin + mid] > id) hi = mid; else lo = mid + 1;
            }
            bin += lo;
            occ = end - lo;
        }
        uint32_t inclusive = occ;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, inclusive, o);
            if (lane >= o) inclusive += t;
        }
        uint32_t total = __shfl_sync(0xffffffffu, inclusive, 31);
        for (uint32_t c0 = 0; c0 < total; c0 += 32) {
            uint32_t k = c0 + lane;
            // The stencil bin holding candidate k: the first lane whose
            // inclusive count exceeds k (every lane searches, past the end
            // with the last candidate, so that each shuffle has the warp).
            uint32_t kk = min(k, total - 1), lo = 0, hi = 31;
#pragma unroll
            for (uint32_t step = 0; step < 5; ++step) {
                uint32_t mid = (lo + hi) >> 1;
                if (__shfl_sync(0xffffffffu, inclusive, mid) > kk) hi = mid; else lo = mid + 1;
            }
            const uint32_t from = __shfl_sync(0xffffffffu, bin - (inclusive - occ), lo);
            bool pass = false;
            uint32_t j = 0;
            if (k < total) {
                j = r.binParticles[from + k];
                {
                    float range = __fadd_rn(__fadd_rn(ri, r.body[j].z), c.skin);
                    float rr = __fmul_rn(range, range);
                    bool near = true, inside = false;
                    if (c.sourceSurfaceNormal == 0) {
                        float4 pj = r.position[j], lj = r.positionRemainder[j];
                        float e[3] = {(pj.x - pi.x) + (lj.x - li.x), (pj.y - pi.y) + (lj.y - li.y),
                                      (pj.z - pi.z) + (lj.z - li.z)};
                        if (c.periodic != 0) {
#pragma unroll
                            for (int a = 0; a < 3; ++a) e[a] -= floorf(e[a] * perBox[a] + 0.5f) * box[a];
                        }
                        // An estimate: only the pairs near the range need the FP64 branch.  A
                        // component is off by a few roundings of a box length (the raw
                        // separation across the boundary, its remainder: below 2.5e-7 of it),
                        // which counts in boxes of thousands of ranges.
                        const float ee = e[0] * e[0] + e[1] * e[1] + e[2] * e[2];
                        const float unsure = 0.002f * rr + 1e-6f * (box[0] + box[1] + box[2]) *
                                                               (range + 5e-7f * (box[0] + box[1] + box[2]));
                        near = ee <= rr + unsure;
                        inside = ee <= rr - unsure;
                    }
                    if (inside) {
                        pass = true;
                    } else if (near) {
                        f3 d = centerBranch64(r, c, id, j);
                        float dd = dot(d, d);
                        if (c.sourceSurfaceNormal != 0 && dd < 1e-12f) fail(r, F_COINCIDENT);
                        else pass = dd <= rr;
                    }
                }
            }
            uint32_t ballot = __ballot_sync(0xffffffffu, pass);
            if (Emit && pass) {
                uint32_t index = base + count + __popc(ballot & lanesBelow());
                if (index < c.pairCapacity) r.pairs[index] = make_uint2(id, j);
                else fail(r, F_PAIR);
            }
            if (!Emit && pass) {
                uint32_t index = count + __popc(ballot & lanesBelow());
                if (index < room) r.byJPairs[size_t(id) * room + index] = j;
            }
            count += __popc(ballot);
        }
    }
    if (!Emit && lane == 0) r.pairCounts[id] = count;
}
__device__ __forceinline__ void pairsCountWarp(const Params& P) {
    if (P.r.control[4] == 0) return;
    for (uint32_t id = warpGlobal(); id < P.c.N; id += warpStride()) findPairsWarp<false>(P.r, P.c, id);
}
// solver.slang:388-392 (the pair total is written by the scan)
__device__ __forceinline__ void pairsEmitWarp(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    if (gtid() == 0) r.work[W_REBUILDS] += 1u;
    const uint32_t room = pairRoom(P.c);
    for (uint32_t id = warpGlobal(); id < P.c.N; id += warpStride()) {
        const uint32_t count = r.pairCounts[id], base = r.pairOffsets[id];
        if (count > room) {
            findPairsWarp<true>(r, P.c, id);
            continue;
        }
        for (uint32_t k = laneId(); k < count; k += WARP) {
            if (base + k < P.c.pairCapacity) r.pairs[base + k] = make_uint2(id, r.byJPairs[size_t(id) * room + k]);
            else fail(r, F_PAIR);
        }
    }
    for (uint32_t id = gtid(); id < P.c.N; id += gstride()) {
        r.referencePosition[id] = r.position[id];
        r.referencePositionRemainder[id] = r.positionRemainder[id];
        uint32_t sp = specimenOf(r, id);
        r.referenceCell[2 * sp] = r.cell[3 * sp];
    }
}
// Pairs grouped by their second grain, ascending pair id per grain.
__device__ __forceinline__ void byJReset(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    for (uint32_t g = gtid(); g <= P.c.N; g += gstride()) {
        r.byJCounts[g] = 0;
        if (g < P.c.N) r.byJCursor[g] = 0;
    }
}
__device__ __forceinline__ void byJCount(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    uint32_t n = activePairs(r, P.c);
    for (uint32_t p = gtid(); p < n; p += gstride()) atomicAdd(&r.byJCounts[r.pairs[p].y], 1u);
}
__device__ __forceinline__ void byJFill(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    uint32_t n = activePairs(r, P.c);
    for (uint32_t p = gtid(); p < n; p += gstride()) {
        uint32_t j = r.pairs[p].y;
        uint32_t slot = atomicAdd(&r.byJCursor[j], 1u);
        r.byJPairs[r.byJOffsets[j] + slot] = p;
    }
}
__device__ __forceinline__ void byJSort(const Params& P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    for (uint32_t g = gtid(); g < P.c.N; g += gstride()) {
        uint32_t begin = r.byJOffsets[g], end = r.byJOffsets[g + 1];
        for (uint32_t a = begin + 1; a < end; ++a) {
            uint32_t v = r.byJPairs[a], k = a;
            while (k > begin && r.byJPairs[k - 1] > v) { r.byJPairs[k] = r.byJPairs[k - 1]; --k; }
            r.byJPairs[k] = v;
        }
    }
}

// ------------------------------------------------------------ collection
// Per pair: FP64 branches of both directions, root cull mask and 3x4
// source-to-target transforms (prepareMeshPairs, solver.slang:468-489), and
// the pair table of the history side being written.
// Upper bound of |R(a) v - R(b) v| / |v| for the rotations of quaternions a
// and b: with 2 alpha the angle between them (or between a and -b), the chord
// 2 sin(2 alpha / 2) <= 4 sin(alpha / 2) = 2 |a -/+ b|.
__device__ __forceinline__ float rotationChord(float4 a, float4 b) {
    float4 d = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
    float4 s = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    float dd = d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w;
    float ss = s.x * s.x + s.y * s.y + s.z * s.z + s.w * s.w;
    return 2.0f * sqrtf(fminf(dd, ss));
}
// Whether the filter results stored for pair p no longer cover it.  They were
// built with every test grown by `margin` (target frame, unscaled).  A node x
// of grain i lies at local = R_j^T (R_i s_i x - b) / s_j in grain j's frame;
// between the build (0) and now (1), for any node that can touch j now
// (|R_i s_i x - b| <= r_j, the bounding radius),
//   s_j |local1 - local0| <= chord_i r_i + |b1 - b0| + chord_j r_j,
// and symmetrically for the other direction.  While that stays below
// margin x min(s_i, s_j), every node that passes the tests now passed the
// grown tests then, so the stored survivors contain every node the filters
// would keep now.  The factor 1.001 and the 1e-5 term cover the FP32
// rounding of the bound and of quaternions that are not exactly unit.
__device__ __forceinline__ bool filterStale(const Res& r, float margin, uint32_t p, uint2 ij, f3 branch) {
    uint2 ref = r.filterRefPairs[p];
    if (ref.x != ij.x || ref.y != ij.y) return true;
    float4 bi = r.body[ij.x], bj = r.body[ij.y];
    float drift = rotationChord(r.rotation[ij.x], r.filterRefRotation[ij.x]) * bi.z +
                  length(branch - xyz(r.filterRefBranch[p])) +
                  rotationChord(r.rotation[ij.y], r.filterRefRotation[ij.y]) * bj.z;
    float slack = 1e-5f * (1.0f + bi.z + bj.z + length(branch));
    return 1.001f * drift + slack > margin * fminf(bi.x, bj.x);
}
__device__ __forceinline__ void pairSetup(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0) return;
    uint32_t n = activePairs(r, c);
    float margin = __uint_as_float(r.work[W_FILTER_MARGIN]);  // the margin the stored results were built with
    bool check = r.work[W_FILTER] == 0;
    for (uint32_t p = gtid(); p < n; p += gstride()) {
        uint2 ij = r.pairs[p];
        f3 branch[2];
        centerBranches64(r, c, ij.x, ij.y, branch[0], branch[1]);
        r.dpairBranch[2 * p] = w4(branch[0], 0.f);
        r.dpairBranch[2 * p + 1] = w4(branch[1], 0.f);
        if (check && filterStale(r, margin, p, ij, branch[0])) atomicOr(&r.work[W_FILTER], 1u);
        r.sidePairB[p] = ij.y;
    }
    uint32_t grains = c.N;
    for (uint32_t g = gtid(); g <= grains; g += gstride())
        r.sidePairOffsets[g] = g < grains ? min(r.pairOffsets[g], n) : n;
    if (storedKeep(c)) {
        // The step's hit counts (groups and sets) start from zero.
        const uint32_t counts = slotHitGroups(c.survivorCapacity) + slotHitSets(c.survivorCapacity);
        for (uint32_t g = gtid(); g < counts; g += gstride()) r.walkHits[g] = 0;
    }
}
// Root cull mask and source-to-target transform of directed pair d
// (prepareMeshPairs, solver.slang:468-489), by its warp: the box corners a
// lane each, the hull group's planes 32 at a time, the transform's columns a
// lane each.  With the test grown by the margin on steps that build the
// filter results.  A thread a pair, one corner and one plane after the other,
// was the longest chain of a build (20 to 30 us whatever the size).
__device__ __forceinline__ bool rootMayContact(const Res& r, uint32_t d, uint32_t i, uint32_t j, f3 branch, float margin) {
    const uint32_t lane = laneId(), cluster = r.meshClusterInfo[r.shapeId[i]].x, shape = r.shapeId[j];
    const f3 sl = xyz(r.meshClusterMin[cluster]), sh = xyz(r.meshClusterMax[cluster]);
    const float4 qs = r.rotation[i], qd = r.rotation[j];
    const float ss = r.body[i].x, sd = r.body[j].x;
    // solver.slang:290-305 (meshClusterMayContact): the transformed corners' box.
    f3 p = mk((lane & 1) ? sh.x : sl.x, (lane & 2) ? sh.y : sl.y, (lane & 4) ? sh.z : sl.z);
    p = qinv(qd, qrot(qs, p * ss) - branch) / sd;
    f3 low = p, high = p;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        low = mn3(low, mk(__shfl_xor_sync(0xffffffffu, low.x, o), __shfl_xor_sync(0xffffffffu, low.y, o),
                          __shfl_xor_sync(0xffffffffu, low.z, o)));
        high = mx3(high, mk(__shfl_xor_sync(0xffffffffu, high.x, o), __shfl_xor_sync(0xffffffffu, high.y, o),
                            __shfl_xor_sync(0xffffffffu, high.z, o)));
    }
    float pad = __fmul_rn(0.00000762939453125f,
        __fadd_rn(__fadd_rn(__fadd_rn(1.0f, mx(mx(fabsf(low.x), fabsf(low.y)), fabsf(low.z))),
                            mx(mx(fabsf(high.x), fabsf(high.y)), fabsf(high.z))), __fdiv_rn(length(branch), sd)));
    if (margin > 0.0f) pad = __fadd_rn(pad, margin);
    low = low - mk(pad, pad, pad);
    high = high + mk(pad, pad, pad);
    f3 centre, half;
    uint32_t group;
    bool open = meshBoxGroup(r, shape, low, high, centre, half, group);
    if (open) {  // (the same on every lane)
        uint4 info = __ldg(&r.meshHullInfo[6 * shape + group]);
        bool outside = false;
        for (uint32_t q = lane; q < info.y; q += WARP) {
            float4 plane = __ldg(&r.meshPlanes[info.x + q]);
            outside |= __fsub_rn(__fadd_rn(dot(xyz(plane), centre), plane.w), dot(abs3(xyz(plane)), half)) > 0;
        }
        open = !__any_sync(0xffffffffu, outside);
    }
    if (open) {
        // Lanes 0-2 the rotated axes, lane 3 the offset; row k from them.
        const float ratio = __fdiv_rn(ss, sd);
        f3 column;
        if (lane < 3) column = qinv(qd, qrot(qs, mk(lane == 0 ? ratio : 0.f, lane == 1 ? ratio : 0.f, lane == 2 ? ratio : 0.f)));
        else column = qinv(qd, -branch) / sd;
        float row[3][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            row[0][k] = __shfl_sync(0xffffffffu, column.x, k);
            row[1][k] = __shfl_sync(0xffffffffu, column.y, k);
            row[2][k] = __shfl_sync(0xffffffffu, column.z, k);
        }
        float4* out = r.meshPairTransform + 4 * size_t(d);
        if (lane == 0) {
            out[0] = make_float4(row[0][0], row[0][1], row[0][2], row[0][3]);
            out[1] = make_float4(row[1][0], row[1][1], row[1][2], row[1][3]);
            out[2] = make_float4(row[2][0], row[2][1], row[2][2], row[2][3]);
            out[3] = make_float4(__fdiv_rn(length(branch), sd), 0.f, 0.f, 0.f);
        }
    }
    __syncwarp();
    return open;
}
// resetMeshContacts (solver.slang:396-403)
// The stored filter results (items, survivor masks and list) serve this step
// if they are complete and were built under this configured margin on a
// pair list of the same length; k_pairSetup then checks each pair and how
// far its grains have moved, and asks for a build if any pair is no longer
// covered.  The margin adapts to the motion, between the configured margin m
// and 16 m: a build within 8 collector runs of the last one doubles it, a
// build after more than 64 halves it (a larger margin keeps a few more nodes
// in the stored lists; it never changes a result).
__device__ __forceinline__ void resetContacts(const Res& r, const Config& c, bool pairsKnown) {
    // Loads first: a store would make each of them wait for the one before.
    const uint32_t complete = r.work[W_FILTER_VALID], configured = r.work[W_FILTER_BASE], pairs = r.work[W_FILTER_PAIRS];
    const uint32_t runs = r.work[W_FILTER_STEPS], age = r.work[W_FILTER_AGE] + 1u, current = r.control[1];
    const float margin = __uint_as_float(r.work[W_FILTER_MARGIN]);
    bool on = c.filterMargin > 0.0f;
    // Steps with the learned culler keep the survivors but no slots (1, not 2).
    bool valid = complete >= (storedKeep(c) ? 2u : 1u) && configured == __float_as_uint(c.filterMargin);
    bool build = !on || !valid || (pairsKnown && pairs != current);
    r.control[2] = 0;
    r.control[6] = 0;
    r.work[W_SLOW] = 0;
    r.work[W_LAPSED] = 0;
    r.work[W_WALL_HITS] = 0;
    if (c.meshGeometry == 0) r.work[W_SURVIVORS] = 0;  // the SDF contacts' scratch slots
    r.work[W_FILTER] = build ? 1u : 0u;
    r.work[W_FILTER_STEPS] = runs + 1u;
    if (on) {
        r.work[W_FILTER_AGE] = age;
        float next = c.filterMargin;
        if (valid)
            next = age <= 8u ? fminf(2.0f * margin, 16.0f * c.filterMargin)
                             : (age > 64u ? fmaxf(0.5f * margin, c.filterMargin) : margin);
        r.work[W_FILTER_NEXT] = __float_as_uint(next);
    }
    if (build) r.work[W_CANDIDATES] = 0;
}
// Flat leaf cull: one warp per directed pair; meshPairBounds (solver.slang:
// 404-417) + meshBoxMayContact (:274-288) on every leaf, gated by the root
// mask.  Equivalent in contacts to the reference's hierarchical walks since
// every test is conservative and each node's decision is exact.
// The enclosure plane test in the source grain's own frame.  With m the
// target-frame normal n rotated to the world, the plane value of a node at
// x (source shape frame, unscaled) is n.local + w = n'.x + w' with
// n' = (s_src/s_dst) qinv(q_src, m) and w' = w - m.branch/s_dst, so one
// 3-term dot per node replaces the two quaternion rotations.  A node (or a
// whole leaf box) is rejected only when n'.x + w' exceeds an upper bound of
// the reference pad 2^-17 (1 + max|local|) -- |local| <= (s_src |x| +
// |branch|) / s_dst -- plus a slack 1e-5 x the magnitudes involved, far
// above the FP32 rounding of either evaluation order.  Such a node would be
// rejected by the reference's own plane test: no contact changes.
struct SourcePlane {
    float4 plane;  // n', w'
    float4 scale;  // s_src/s_dst, |branch|_1/s_dst, |w|, |n'|_1
};
__device__ __forceinline__ SourcePlane sourcePlane(float4 plane, float4 qs, float4 qd, float ss, float sd, f3 branch) {
    SourcePlane sp;
    f3 m = qrot(qd, xyz(plane));
    float k = __fdiv_rn(ss, sd);
    f3 n = qinv(qs, m) * k;
    float w = __fsub_rn(plane.w, __fdiv_rn(dot(m, branch), sd));
    float bn = __fdiv_rn(__fadd_rn(__fadd_rn(fabsf(branch.x), fabsf(branch.y)), fabsf(branch.z)), sd);
    sp.plane = w4(n, w);
    sp.scale = make_float4(k, bn, fabsf(plane.w), __fadd_rn(__fadd_rn(fabsf(n.x), fabsf(n.y)), fabsf(n.z)));
    return sp;
}
// Rejection bound for points with |x|_1 <= extent.
__device__ __forceinline__ float sourcePlaneBound(const SourcePlane& sp, float extent) {
    float reach = __fadd_rn(__fmul_rn(sp.scale.x, extent), sp.scale.y);
    float pad = __fmul_rn(0.00000762939453125f, __fadd_rn(1.0f, reach));
    float slack = __fmul_rn(1e-5f, __fadd_rn(__fadd_rn(__fadd_rn(1.0f, sp.scale.z), reach),
                                            __fmul_rn(sp.scale.w, extent)));
    return __fadd_rn(pad, slack);
}
// `grow` widens a test for the stored filter results: the plane value moves
// by at most |n| = 1 times a node's displacement in the target frame, so
// `grow` = margin x 1.001 (FP32 unit normals) covers every placement within
// the margin.
__device__ __forceinline__ bool nodeBeyondSourcePlane(const SourcePlane& sp, f3 x, float grow = 0.0f) {
    float extent = __fadd_rn(__fadd_rn(fabsf(x.x), fabsf(x.y)), fabsf(x.z));
    return __fadd_rn(dot(xyz(sp.plane), x), sp.plane.w) > __fadd_rn(sourcePlaneBound(sp, extent), grow);
}
__device__ __forceinline__ bool leafBeyondSourcePlane(const SourcePlane& sp, f3 low, f3 high, float grow = 0.0f) {
    f3 c = 0.5f * (low + high), h = 0.5f * (high - low);
    float nearest = __fsub_rn(__fadd_rn(dot(xyz(sp.plane), c), sp.plane.w), dot(abs3(xyz(sp.plane)), h));
    float extent = __fadd_rn(__fadd_rn(__fadd_rn(fabsf(c.x), fabsf(c.y)), fabsf(c.z)),
                             __fadd_rn(__fadd_rn(h.x, h.y), h.z));
    return nearest > __fadd_rn(sourcePlaneBound(sp, extent), grow);
}
// Enclosure plane of the target most violated by the source centre
// (cpu_scheduling.slang:58-71): warp arg-max, lowest index on ties.  Every
// lane returns the plane.
__device__ __forceinline__ float4 enclosurePlane(const Res& r, uint32_t j, uint32_t targetShape, f3 branch) {
    f3 centre = (-qinv(r.rotation[j], branch)) / r.body[j].x;
    uint4 first = __ldg(&r.meshHullInfo[6 * targetShape]);
    uint4 last = __ldg(&r.meshHullInfo[6 * targetShape + 5]);
    uint32_t begin = first.x, end = last.x + last.y;
    float best = -1e30f;
    uint32_t bestIndex = EMPTY;
    for (uint32_t k = begin + laneId(); k < end; k += WARP) {
        float4 candidate = __ldg(&r.meshPlanes[k]);
        float violation = __fadd_rn(dot(xyz(candidate), centre), candidate.w);
        if (violation > best) { best = violation; bestIndex = k; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(0xffffffffu, best, o);
        uint32_t oi = __shfl_xor_sync(0xffffffffu, bestIndex, o);
        if (ob > best || (ob == best && oi < bestIndex)) { best = ob; bestIndex = oi; }
    }
    return bestIndex == EMPTY ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(&r.meshPlanes[bestIndex]);
}
// Runs on steps that build the filter results: with a margin every test is
// grown by it and the pose the results are built at is recorded.
__device__ __forceinline__ void leafCull(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.work[W_FILTER] == 0) return;
    uint32_t n = 2 * activePairs(r, c);
    float margin = buildMargin(r, c);
    float grow = __fmul_rn(1.001f, margin);
    if (gtid() == 0) r.work[W_FILTER_VALID] = 0;  // (also where this build stores nothing: it overwrites the lists)
    if (margin > 0.0f) {
        for (uint32_t g = gtid(); g < c.N; g += gstride()) r.filterRefRotation[g] = r.rotation[g];
        if (gtid() == 0) {
            r.work[W_FILTER_PAIRS] = r.control[1];
            r.work[W_FILTER_MARGIN] = __float_as_uint(margin);
            r.work[W_FILTER_BASE] = __float_as_uint(c.filterMargin);
            r.work[W_FILTER_AGE] = 0;
            r.work[W_FILTER_BUILDS] += 1u;
        }
    }
    for (uint32_t d = warpGlobal(); d < n; d += warpStride()) {
        uint32_t p = d >> 1, pass = d & 1;
        uint2 ij = r.pairs[p];
        uint32_t i = pass ? ij.y : ij.x, j = pass ? ij.x : ij.y;
        if (margin > 0.0f && pass == 0 && laneId() == 0) {
            r.filterRefPairs[p] = ij;
            r.filterRefBranch[p] = r.dpairBranch[d];
        }
        uint32_t count = 0;
        if (live && rootMayContact(r, d, i, j, xyz(r.dpairBranch[d]), margin)) {
            uint4 li = __ldg(&r.meshLeafInfo[r.shapeId[i]]);
            uint32_t targetShape = r.shapeId[j];
            float4 plane;
            SourcePlane source;
            {
                f3 branch = xyz(r.dpairBranch[d]);
                plane = enclosurePlane(r, j, targetShape, branch);
                source = sourcePlane(plane, r.rotation[i], r.rotation[j], r.body[i].x, r.body[j].x, branch);
                if (laneId() == 0) {
                    r.dpairPlane[d] = plane;
                    r.dpairSourcePlane[2 * d] = source.plane;
                    r.dpairSourcePlane[2 * d + 1] = source.scale;
                }
            }
            for (uint32_t k0 = 0; k0 < li.y; k0 += WARP) {
                // Lane per leaf: the cheap tests (target root box, source-frame
                // plane); then, for each leaf still in, the whole warp tests the
                // hull group's planes in parallel.  Every test is a conservative
                // "may contact", so their order does not matter.
                uint32_t k = k0 + laneId();
                bool open = false;
                f3 centre = mk(0.f, 0.f, 0.f), half = centre;
                uint32_t group = 0;
                if (k < li.y) {
                    uint32_t leaf = __ldg(&r.meshLeaves[li.x + k]);
                    f3 low, high;
                    meshPairBounds(r, d, leaf, low, high, margin);
                    open = meshBoxGroup(r, targetShape, low, high, centre, half, group) &&
                           !leafBeyondSourcePlane(source, xyz(__ldg(&r.meshClusterMin[leaf])),
                                                  xyz(__ldg(&r.meshClusterMax[leaf])), grow);
                }
                uint32_t pending = __ballot_sync(0xffffffffu, open), m = 0;
                while (pending) {
                    uint32_t lane = __ffs(pending) - 1;
                    pending &= pending - 1;
                    f3 cl = mk(__shfl_sync(0xffffffffu, centre.x, lane), __shfl_sync(0xffffffffu, centre.y, lane),
                               __shfl_sync(0xffffffffu, centre.z, lane));
                    f3 hl = mk(__shfl_sync(0xffffffffu, half.x, lane), __shfl_sync(0xffffffffu, half.y, lane),
                               __shfl_sync(0xffffffffu, half.z, lane));
                    uint4 info = __ldg(&r.meshHullInfo[6 * targetShape + __shfl_sync(0xffffffffu, group, lane)]);
                    bool outside = false;
                    for (uint32_t q = laneId(); q < info.y; q += WARP) {
                        float4 plane = __ldg(&r.meshPlanes[info.x + q]);
                        outside |= __fsub_rn(__fadd_rn(dot(xyz(plane), cl), plane.w), dot(abs3(xyz(plane)), hl)) > 0;
                    }
                    if (!__any_sync(0xffffffffu, outside)) m |= 1u << lane;
                }
                if (laneId() == 0) r.leafMask[size_t(d) * c.leafWords + k0 / WARP] = m;
                count += __popc(m);
            }
        }
        if (laneId() == 0) r.dpairLeafCount[d] = count;
    }
}
__device__ __forceinline__ void leafEmit(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0 || r.work[W_FILTER] == 0) return;
    uint32_t n = 2 * activePairs(r, c);
    for (uint32_t d = warpGlobal(); d < n; d += warpStride()) {
        if (r.dpairLeafCount[d] == 0) continue;
        uint32_t p = d >> 1, pass = d & 1;
        uint2 ij = r.pairs[p];
        uint32_t i = pass ? ij.y : ij.x;
        uint4 li = __ldg(&r.meshLeafInfo[r.shapeId[i]]);
        uint32_t base = r.dpairCandOffset[d];
        for (uint32_t k0 = 0; k0 < li.y; k0 += WARP) {
            uint32_t m = r.leafMask[size_t(d) * c.leafWords + k0 / WARP];
            uint32_t k = k0 + laneId();
            if ((m >> laneId()) & 1u) {
                uint32_t slot = base + __popc(m & lanesBelow());
                if (slot < c.candidateCapacity) r.candidates[slot] = make_uint2(d, __ldg(&r.meshLeaves[li.x + k]));
            }
            base += __popc(m);
        }
    }
}
// Node query in stages.  The filter stage (one warp per (directed pair,
// leaf) item, two nodes per lane) applies the one-dot enclosure-plane test
// in the source frame and records each item's surviving nodes as a 64-bit
// mask.  A scan turns the survivor counts into offsets and the survivors are
// listed in canonical order.  A dense pass (one thread per survivor) places
// each in the target frame and applies the target-frame plane and the hull;
// with the learned culler on, a second pass evaluates the target's network
// for 64 survivors per warp on tensor cores.  A scan keeps the survivors no
// test ruled out and the exact stage runs one thread per kept survivor: full
// warps of BVH walks instead of warps in which most lanes were rejected and
// idle.  Each hit sets its bit in
// the item's hit mask (integer atomics: the result does not depend on their
// order) and keeps its record in the survivor's scratch slot; the emit pass
// copies hits to their canonical offsets.
__device__ __forceinline__ void nodeFilter(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t n = min(r.work[W_CANDIDATES], c.candidateCapacity);
    // Stored survivors serve this step (their hit masks were cleared by the
    // previous step's emit).
    if (r.work[W_FILTER] == 0) return;
    float grow = __fmul_rn(1.001f, buildMargin(r, c));
    // Two items per warp, one per half-warp, four node slots per lane
    // (slot = lane in half + 16 j): twice the loads in flight per instruction.
    uint32_t half = laneId() >> 4, hl = laneId() & 15u;
    for (uint32_t pair0 = 2 * warpGlobal(); pair0 < n; pair0 += 2 * warpStride()) {
        uint32_t item = pair0 + half;
        bool keep[4] = {false, false, false, false};
        if (item < n && r.control[0] == 0) {
            uint2 cd = r.candidates[item];
            uint32_t d = cd.x, p = d >> 1, pass = d & 1;
            uint2 ij = r.pairs[p];
            uint32_t src = pass ? ij.y : ij.x;
            SourcePlane source{r.dpairSourcePlane[2 * d], r.dpairSourcePlane[2 * d + 1]};
            uint4 range = __ldg(&r.meshClusterRanges[cd.y]);
            const float4* samples = r.sample + __ldg(&r.sampleInfo[r.shapeId[src]].x);
            // One dot per node against the source-frame plane; the exact
            // placement, target-frame plane and hull follow in a dense pass.
            float4 x[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                uint32_t k = hl + 16 * j;
                x[j] = k < range.y ? __ldg(&samples[__ldg(&r.meshSampleIndices[range.x + k])])
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                keep[j] = hl + 16 * j < range.y && !nodeBeyondSourcePlane(source, xyz(x[j]), grow);
        }
        uint32_t b[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) b[j] = __ballot_sync(0xffffffffu, keep[j]);
        if (hl == 0 && item < n) {
            uint32_t sh = 16 * half;
            uint32_t m0 = ((b[0] >> sh) & 0xFFFFu) | (((b[1] >> sh) & 0xFFFFu) << 16);
            uint32_t m1 = ((b[2] >> sh) & 0xFFFFu) | (((b[3] >> sh) & 0xFFFFu) << 16);
            r.candSurvMask[item] = make_uint2(m0, m1);
            r.candSurvCount[item] = __popc(m0) + __popc(m1);
            r.candHitMask[item] = make_uint2(0u, 0u);
            r.candHitCount[item] = 0;
        }
    }
}
// Source node, partner and target-frame position of survivor s.
struct SurvivorNode {
    uint32_t item, slot, src, dst, node;
    f3 arm, local;
};
__device__ __forceinline__ SurvivorNode survivorNode(const Res& r, uint32_t s) {
    SurvivorNode v;
    uint2 sv = r.survivors[s];
    v.item = sv.x;
    v.slot = sv.y;
    uint2 cd = r.candidates[sv.x];
    uint32_t d = cd.x, p = d >> 1, pass = d & 1;
    uint2 ij = r.pairs[p];
    v.src = pass ? ij.y : ij.x;
    v.dst = pass ? ij.x : ij.y;
    v.node = __ldg(&r.meshSampleIndices[__ldg(&r.meshClusterRanges[cd.y]).x + sv.y]);
    float4 sp = __ldg(&r.sample[__ldg(&r.sampleInfo[r.shapeId[v.src]].x) + v.node]);
    v.arm = qrot(r.rotation[v.src], xyz(sp) * r.body[v.src].x);
    v.local = qinv(r.rotation[v.dst], v.arm - xyz(r.dpairBranch[d])) / r.body[v.dst].x;
    return v;
}
// Exact placement, distance grid, target-frame enclosure plane and hull of
// every survivor of the one-dot test, a thread each: survKeep[s] = 1 for
// the nodes that go on to the exact query.
// When the exact-query list is stored with the filter results, this pass
// runs only on build steps, with the plane, hull and grid tests grown by the
// margin (a node the grid bounds farther than the margin from the surface
// cannot reach it while the results serve).
__device__ __forceinline__ void survivorPrefilter(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    bool stored = storedKeep(c);
    if (r.control[0] != 0 || (stored && r.work[W_FILTER] == 0)) return;
    float grow = stored ? __fmul_rn(1.001f, buildMargin(r, c)) : 0.0f;
    uint32_t n = min(r.work[W_SURVIVORS], c.survivorCapacity);
    for (uint32_t s = gtid(); s < n; s += gstride()) {
        uint2 sv = r.survivors[s];
        uint2 cd = r.candidates[sv.x];
        uint32_t d = cd.x, p = d >> 1, pass = d & 1;
        uint2 ij = r.pairs[p];
        uint32_t src = pass ? ij.y : ij.x, dst = pass ? ij.x : ij.y;
        uint32_t node = __ldg(&r.meshSampleIndices[__ldg(&r.meshClusterRanges[cd.y]).x + sv.y]);
        // Placed with survivorNode's expressions; a node certified outside the target by
        // the distance-bound grid cannot be a contact (the exact query would
        // find phi > 0).  Each test only rejects, so the order is free: the
        // grid first, one load that drops most, then the plane and the hull,
        // a load a plane.
        f3 arm = qrot(r.rotation[src], xyz(__ldg(&r.sample[__ldg(&r.sampleInfo[r.shapeId[src]].x) + node])) * r.body[src].x);
        f3 local = qinv(r.rotation[dst], arm - xyz(r.dpairBranch[d])) / r.body[dst].x;
        const uint32_t shape = r.shapeId[dst];
        bool keep = !(c.distanceGridEnabled && distanceBound(r, shape, local) > grow);
        if (keep) {
            float4 plane = r.dpairPlane[d];
            keep = nodeTests(r, shape, &plane, local, grow);
        }
        r.survKeep[s] = keep ? 1u : 0u;
    }
}
// Learned culler over the kept survivors, on the tensor cores (culler.cuh).
// The survivors are first sorted by target shape (a counting sort into
// walkKey: per-shape counts, their scan, then placement -- the walk-bucket
// arrays and walkKey serve the stored exact-query list only, which the
// culler does not use), so that a 128-row tile holds one shape, or a few at
// its ends.  The culler clears keep[s] when the target's network places a
// kept survivor s beyond the shape's calibrated margin; the exact query
// decides every other one.  The order of the sorted list within a shape is
// immaterial: each row's prediction depends on its own point only.
__device__ __forceinline__ uint32_t survivorTargetShape(const Res& r, const Config& c, uint32_t s) {
    uint2 sv = r.survivors[s];
    uint32_t d = r.candidates[sv.x].x;
    uint2 ij = r.pairs[d >> 1];
    uint32_t shape = r.shapeId[(d & 1) ? ij.x : ij.y];
    return shape < c.shapes ? shape : EMPTY;
}
// Survivors kept for the exact query, in survivor order, which is contact
// order (pair, direction, leaf, node): their indices, or, when the list is
// stored with the filter results, a slot each with what its exact query reads
// every step (one load instead of the survivor -> item -> pair -> sample
// chain).  In this order a warp's slots share their two grains and branch,
// and the step's contacts leave it in place (k_emitSlots).
__device__ __forceinline__ void walkList(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    bool stored = storedKeep(c);
    if (r.control[0] != 0 || (stored && r.work[W_FILTER] == 0)) return;
    uint32_t n = min(r.work[W_SURVIVORS], c.survivorCapacity);
    if (stored && gtid() == 0) r.work[W_DORMANT] = 0;  // a new list: no slot sleeps yet
    for (uint32_t s = gtid(); s < n; s += gstride()) {
        if (!r.survKeep[s]) continue;
        uint32_t slot = r.keepOffset[s];
        if (!stored) {
            r.walkList[slot] = s;
            continue;
        }
        uint2 sv = r.survivors[s];
        uint2 cd = r.candidates[sv.x];
        uint2 ij = r.pairs[cd.x >> 1];
        uint32_t src = (cd.x & 1) ? ij.y : ij.x, dst = (cd.x & 1) ? ij.x : ij.y;
        uint32_t node = __ldg(&r.meshSampleIndices[__ldg(&r.meshClusterRanges[cd.y]).x + sv.y]);
        r.walkNode[slot] = make_uint4(src, dst, cd.x, __ldg(&r.sampleInfo[r.shapeId[src]].x) + node);
        r.walkState[slot] = EMPTY;
        r.walkContact[slot] = EMPTY;
    }
}
// Survivor list in canonical (item, node slot) order.
// On a build step with a margin, it also marks the stored results complete
// when no list overflowed.
__device__ __forceinline__ void survivorList(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0 || r.work[W_FILTER] == 0) return;
    uint32_t n = min(r.work[W_CANDIDATES], c.candidateCapacity);
    if (gtid() == 0 && c.filterMargin > 0.0f) {
        const bool complete = r.work[W_CANDIDATES] <= c.candidateCapacity && r.work[W_SURVIVORS] <= c.survivorCapacity;
        r.work[W_FILTER_VALID] = complete ? (storedKeep(c) ? 2u : 1u) : 0u;
    }
    for (uint32_t item = warpGlobal(); item < n; item += warpStride()) {
        uint2 m = r.candSurvMask[item];
        if ((m.x | m.y) == 0) continue;
        uint32_t base = r.candSurvOffset[item];
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
            uint32_t word = half ? m.y : m.x;
            if (!((word >> laneId()) & 1u)) continue;
            uint32_t s = base + (half ? __popc(m.x) : 0) + __popc(word & lanesBelow());
            if (s < c.survivorCapacity) r.survivors[s] = make_uint2(item, laneId() + half * WARP);
            else fail(r, F_CONTACT);
        }
    }
}
// Exact query, one thread per kept survivor.
__device__ __forceinline__ void recordHitAt(const Res& r, uint32_t s, uint32_t item, uint32_t slot, float4 pd,
                                            float4 na) {
    r.hitScratch[2 * s] = pd;
    r.hitScratch[2 * s + 1] = na;
    atomicOr(slot < WARP ? &r.candHitMask[item].x : &r.candHitMask[item].y, 1u << (slot & 31u));
    atomicAdd(&r.candHitCount[item], 1u);
}
__device__ __forceinline__ void recordHit(const Res& r, uint32_t s, const SurvivorNode& v, float4 pd, float4 na) {
    recordHitAt(r, s, v.item, v.slot, pd, na);
}
// A stored walk slot's node, placed in the target frame from its record:
// the same expressions as survivorNode (the same arm and local bits).
struct WalkNode {
    uint4 rec;  // source, target, directed pair, packed sample
    float4 sp, bs, bd, qd;
    f3 arm, local;
};
__device__ __forceinline__ WalkNode walkNode(const Res& r, uint32_t t) {
    WalkNode w;
    w.rec = r.walkNode[t];
    w.sp = __ldg(&r.sample[w.rec.w]);
    w.bs = r.body[w.rec.x];
    w.bd = r.body[w.rec.y];
    w.qd = r.rotation[w.rec.y];
    float4 qs = r.rotation[w.rec.x];
    f3 branch = xyz(r.dpairBranch[w.rec.z]);
    w.arm = qrot(qs, xyz(w.sp) * w.bs.x);
    w.local = qinv(w.qd, w.arm - branch) / w.bd.x;
    return w;
}
// Exact queries of a stored list.  A stored list keeps its slots from step
// to step, and each slot keeps a certificate: the triangles nearest to the
// point p0 it was taken at and a gap g, every other triangle lying at least g
// farther from p0 than the nearest.  Distances are 1-Lipschitz in the point,
// so while 2 |p - p0| + slack < g the triangle the walk would record at p is
// among the listed ones: the step evaluates those (one for most slots; the
// faces of an edge or a vertex where that is the nearest feature) and takes
// the smallest distance, as the walk does (considerTriangle).  The slack,
// 4e-6 (1 + |p|_1), covers the FP32 rounding of the distances: with e the
// largest difference between a computed triangle distance and the exact one
// (a few units in the last place of |p|, about 3e-7 (1 + |p|) here), the
// other triangles stay strictly farther while 2 |p - p0| + 4e < g; the slack
// is above 4e.  Slots whose certificate lapsed and new slots are listed
// and answered and certified again from their grid
// cell's triangle list in a kernel of their own, in full warps
// (k_nodeCertify); what a list cannot decide is walked (k_nodeWalkSlow).
// Bound by the latency of dependent loads (under 30% of issue slots used),
// so: few of them, and many warps.  One triangle a certificate left 2% of a
// resting packing's slots and 15 to 25% of a relaxing one's to BVH walks every
// step, whose chains of dependent node loads were the step's critical path;
// with the faces of edges and vertices in the certificate, cell lists for the
// lapsed ones and the fused emit and law below, a step went from 185 to 120 us
// (10,000 grains at rest), 640 to 361 (50,000) and 1,848 to 914 (15,625
// relaxing, 3.3 M live slots).
//
// Dormant slots.  Until the next build, the motion check of k_pairSetup
// bounds chord_i r_i + |d branch| + chord_j r_j by m s_j (chord: of a
// grain's rotation since the build; r: bounding radius; s: scale), so a node
// inside the target's bounding sphere -- as every node touching it is --
// lies within m (target frame, unscaled) of where it was at the build, and
// a node at distance |v| from the target's centre now lies within
// m max(1, |v| / r_j) of it.  A node farther outside than the sum (times
// 1.001, plus the distance rounding slack) cannot touch the target before
// the next build, and its slot sleeps: it is skipped with one 8-byte load.
__device__ __forceinline__ bool fallsAsleep(const WalkNode& w, float phi, float margin) {
    float slack = __fmul_rn(2e-5f, __fadd_rn(1.0f, __fadd_rn(__fadd_rn(fabsf(w.local.x), fabsf(w.local.y)),
                                                             fabsf(w.local.z))));
    float reachNow = fmaxf(1.0f, __fdiv_rn(__fmul_rn(length(w.local), w.bd.x), w.bd.z));
    float sleep = __fmul_rn(__fmul_rn(1.001f, margin), __fadd_rn(1.0f, reachNow));
    return phi > __fadd_rn(sleep, slack);
}
__device__ __forceinline__ float certificateReach(float margin) { return __fadd_rn(__fmul_rn(2.01f, margin), 1e-4f); }
// Appends the warp's flagged lanes' values to a list of `room` words (called by
// whole warps); the count goes on past them, the stores do not.
// Few slots lapse, so few warps append: a block's one atomic for all of its
// warps cost every block a barrier a round (a quarter of the query's stalls).
__device__ __forceinline__ void appendWarp(bool flagged, uint32_t value, uint32_t* list, uint32_t room,
                                           uint32_t* count) {
    const uint32_t ballot = __ballot_sync(0xffffffffu, flagged);
    if (ballot == 0) return;
    uint32_t base = 0;
    if (laneId() == 0) base = atomicAdd(count, uint32_t(__popc(ballot)));
    base = __shfl_sync(0xffffffffu, base, 0);
    base += __popc(ballot & lanesBelow());
    if (flagged && base < room) list[base] = value;
}
// The slot's contact record, in its scratch slot; whether it is a contact.
__device__ __forceinline__ bool recordSlot(const Res& r, const Config& c, uint32_t t, const WalkNode& w, float4 f) {
    float4 pd, na;
    if (!nodeContactWith(r, c, w.rec.x, w.sp, w.bs, w.bd, w.qd, w.arm, f, pd, na)) return false;
    r.hitScratch[2 * size_t(t)] = pd;
    r.hitScratch[2 * size_t(t) + 1] = na;
    return true;
}
// A hit of active slot i found after k_nodeQuery.
__device__ __forceinline__ void lateHit(const SlotHits& hits, uint32_t i) {
    atomicOr(&hits.words[i >> 5], 1u << (i & 31u));
    atomicAdd(&hits.groups[i / (32 * HIT_WORDS)], 1u);
    atomicAdd(&hits.sets[i / (32 * HIT_WORDS * HIT_GROUPS)], 1u);
}
// The active slots whose certificates hold: their hit bits and counts.  The
// others are listed in walkList (which lists built every step use; survKeep holds
// keep flags and nothing else).  Only the slots their build left awake are
// visited (walkActive): 185 of 449 thousand on a dense packing of 10,000
// grains, and warps full of them instead of a third full.
__device__ __forceinline__ void nodeQuery(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    const SlotHits hits = slotHits(r, c);
    uint32_t n = min(r.work[W_ACTIVE], c.survivorCapacity);
    for (uint32_t w0 = warpGlobal(); WARP * w0 < n; w0 += warpStride()) {
        uint32_t i = WARP * w0 + laneId(), t = i < n ? r.walkActive[i] : 0u;
        uint32_t state = i < n ? r.walkState[t] : DORMANT;
        bool lapsed = state == EMPTY, hit = false;
        if (state == CERTIFIED) {
            WalkNode w = walkNode(r, t);
            float4 f;
            if (certificateQuery(r, r.walkCert + size_t(CERT_ROWS) * t, r.shapeId[w.rec.y], w.local, f))
                hit = recordSlot(r, c, t, w, f);
            else
                lapsed = true;
        }
        uint32_t ballot = __ballot_sync(0xffffffffu, hit);
        if (laneId() == 0 && i < n) {
            hits.words[i >> 5] = ballot;
            if (ballot) {
                atomicAdd(&hits.groups[i / (32 * HIT_WORDS)], uint32_t(__popc(ballot)));
                atomicAdd(&hits.sets[i / (32 * HIT_WORDS * HIT_GROUPS)], uint32_t(__popc(ballot)));
            }
        }
        appendWarp(lapsed, i, r.walkList, c.survivorCapacity, &r.work[W_LAPSED]);
    }
}
// A new list's slots, certified from their grid cells' triangle lists (in the
// filter build): the slots that fall asleep at once are left out of the
// active list (survKeep, then its scan).
__device__ __forceinline__ void certifyBuild(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live || r.work[W_FILTER] == 0) return;
    uint32_t n = min(r.work[W_KEPT], c.survivorCapacity);
    const float margin = __uint_as_float(r.work[W_FILTER_MARGIN]), reach = certificateReach(margin);
    uint32_t slept = 0;
    for (uint32_t t = gtid(); t < n; t += gstride()) {
        bool asleep = false;
        if (c.cellListsEnabled) {
            WalkNode w = walkNode(r, t);
            float4 f;
            if (cellQuery(r, r.shapeId[w.rec.y], w.local, reach, r.walkCert + size_t(CERT_ROWS) * t, f)) {
                asleep = fallsAsleep(w, f.w, margin);
                r.walkState[t] = asleep ? DORMANT : CERTIFIED;
            }
        }
        r.survKeep[t] = asleep ? 0u : 1u;
        slept += asleep;
    }
    slept = __reduce_add_sync(0xffffffffu, slept);
    if (laneId() == 0 && slept) atomicAdd(&r.work[W_DORMANT], slept);
}
// The listed active slots, from their grid cells' triangle lists: a warp a
// slot where there are few (cellQueryWarp), a lane a slot where many lapsed at
// once.  The undecided ones (all of them without the lists) are listed in
// walkKey.
__device__ __forceinline__ void nodeCertify(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    const uint32_t n = min(r.work[W_LAPSED], c.survivorCapacity);
    const SlotHits hits = slotHits(r, c);
    const float margin = __uint_as_float(r.work[W_FILTER_MARGIN]), reach = certificateReach(margin);
    const bool single = c.cellListsEnabled && n <= 8 * warpStride();
    const uint32_t each = single ? 1u : WARP;
    for (uint32_t k0 = each * warpGlobal(); k0 < n; k0 += each * warpStride()) {
        const uint32_t k = single ? k0 : k0 + laneId();
        uint32_t i = 0;
        bool slow = false;
        if (k < n) {
            i = r.walkList[k];
            slow = !single || laneId() == 0;
            if (c.cellListsEnabled) {
                const uint32_t t = r.walkActive[i];
                WalkNode w = walkNode(r, t);
                uint4* record = r.walkCert + size_t(CERT_ROWS) * t;
                float4 f;
                const bool decided = single ? cellQueryWarp(r, r.shapeId[w.rec.y], w.local, record, f)
                                            : cellQuery(r, r.shapeId[w.rec.y], w.local, reach, record, f);
                if (decided && slow) {
                    slow = false;
                    const bool asleep = fallsAsleep(w, f.w, margin);
                    if (asleep) atomicAdd(&r.work[W_DORMANT], 1u);
                    r.walkState[t] = asleep ? DORMANT : CERTIFIED;
                    if (recordSlot(r, c, t, w, f)) lateHit(hits, i);
                }
            }
        }
        __syncwarp();
        appendWarp(slow, i, r.walkKey, c.survivorCapacity, &r.work[W_SLOW]);
    }
}
// Records a slot's query: its certificate from the triangles at the nearest
// distance (`ids`, EMPTY-padded) with every other one farther by `gap`.
__device__ __forceinline__ void certifySlot(const Res& r, const Config& c, uint32_t i, uint32_t t, const WalkNode& w,
                                            float4 f, uint32_t id0, uint32_t id1, uint32_t id2, float gap,
                                            float margin) {
    bool found = id0 != EMPTY, dormant = found && fallsAsleep(w, f.w, margin);
    if (dormant) {
        // One count per group of lanes marking slots together.
        uint32_t group = __activemask();
        if (laneId() == uint32_t(__ffs(group) - 1)) atomicAdd(&r.work[W_DORMANT], uint32_t(__popc(group)));
    }
    r.walkState[t] = dormant ? DORMANT : (found ? CERTIFIED : EMPTY);
    if (found && !dormant) {
        uint4* record = r.walkCert + size_t(CERT_ROWS) * t;
        record[0] = make_uint4(__float_as_uint(w.local.x), __float_as_uint(w.local.y), __float_as_uint(w.local.z),
                               __float_as_uint(gap));
        record[1] = make_uint4(id0, id1, id2, 0u);
        record[2] = make_uint4(EMPTY, EMPTY, EMPTY, EMPTY);
    }
    if (recordSlot(r, c, t, w, f)) lateHit(slotHits(r, c), i);
}
// One slot's query by a whole block, without a walk: the threads test the
// boxes of every BVH leaf of the shape (independent loads: no chain of
// dependent visits) and evaluate the triangles of those within the reach of
// the seed; the smallest distance over the threads is the one a walk records,
// exact ties ordered as it visits them.  A few such slots a step are on its
// critical path: a warp's certifying walk of one took 40 to 140 us of
// dependent loads (the nodes near a 5,120-triangle shape's medial axis).
__device__ __forceinline__ void scanSlot(const Res& r, const Config& c, uint32_t i, float margin, float reach) {
    __shared__ float warpBest[32], warpOther[32];
    __shared__ uint32_t warpTriangle[32];
    const uint32_t t = r.walkActive[i];
    WalkNode w = walkNode(r, t);
    const uint32_t shape = r.shapeId[w.rec.y];
    f3 centre;
    uint32_t cell = nearestCell(__ldg(&r.distanceGridInfo[shape]), w.local, centre);
    uint32_t seed = __ldg(&r.distanceGridTriangle[size_t(shape) * GRID * GRID * GRID + cell]);
    NearestTriangle n{1e30f, mk(0.f, 0.f, 0.f), 0, EMPTY, false, false};
    float cap = 1e30f;
    if (seed != EMPTY) {
        float root = __fadd_rn(__fsqrt_rn(considerTriangle(r, shape, w.local, seed, n)), reach);
        cap = nextafterf(__fmul_rn(__fmul_rn(root, root), 1.0000019073486328f), 1e30f);
        n.best = 1e30f;
        n.triangle = EMPTY;
    }
    float other = cap;
    uint4 nodes = __ldg(&r.meshRoots[shape]);
#pragma unroll 2
    for (uint32_t node = nodes.x + threadIdx.x; node < nodes.y; node += blockDim.x) {
        uint4 link = __ldg(&r.meshLinks[node]);
        float away = meshBoxDistance(r, node, w.local);
        if (link.z == 0 || away > cap) continue;
        for (uint32_t k = 0; k < link.z; ++k) {
            float before = n.best;
            float d = considerTriangle<true>(r, shape, w.local, link.y + k, n);
            other = fminf(other, d < before ? before : d);
        }
    }
    // The smallest, its triangle (the first a walk visits among ties, which
    // lie in different leaves), and the smallest of the other distances.
    auto merge = [&](float& best, uint32_t& triangle, float& rest, float theirs, uint32_t next, float theirRest) {
        rest = fminf(rest, theirRest);
        if (next == EMPTY) return;
        if (triangle == EMPTY || theirs < best ||
            (theirs == best && leafVisitedFirst(r, shape, w.local, __ldg(&r.triangleLeaf[next]),
                                                __ldg(&r.triangleLeaf[triangle])))) {
            if (triangle != EMPTY) rest = fminf(rest, best);
            best = theirs;
            triangle = next;
        } else {
            rest = fminf(rest, theirs);
        }
    };
    float best = n.best;
    uint32_t triangle = n.triangle;
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        float theirs = __shfl_down_sync(0xffffffffu, best, o), theirRest = __shfl_down_sync(0xffffffffu, other, o);
        uint32_t next = __shfl_down_sync(0xffffffffu, triangle, o);
        if (laneId() < uint32_t(o)) merge(best, triangle, other, theirs, next, theirRest);
    }
    if (laneId() == 0) {
        warpBest[threadIdx.x >> 5] = best;
        warpTriangle[threadIdx.x >> 5] = triangle;
        warpOther[threadIdx.x >> 5] = other;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t k = 1; k < blockDim.x >> 5; ++k) merge(best, triangle, other, warpBest[k], warpTriangle[k], warpOther[k]);
        NearestTriangle found{1e30f, mk(0.f, 0.f, 0.f), 0, EMPTY, false, false};
        if (triangle != EMPTY) considerTriangle(r, shape, w.local, triangle, found);
        float gap = triangle != EMPTY ? __fsub_rn(__fsqrt_rn(other), __fsqrt_rn(best)) : 0.0f;
        float4 f = distanceResult(r, w.local, triangle != EMPTY ? found.best : cap, found.point, found.normal,
                                  triangle != EMPTY, false);
        certifySlot(r, c, i, t, w, f, triangle, EMPTY, EMPTY, gap, margin);
    }
    __syncthreads();  // before the next slot writes the shared rows
}
// The slots the triangle lists left undecided (all that lapsed, without the
// lists).  Few run a block each (scanSlot; up to four per block of the grid);
// more run a lane each, a certifying walk in 32-slot runs of the list
// (coherent walks) dealt to the blocks in turn, so that either way they
// spread over every SM.
__device__ __forceinline__ void nodeWalkSlow(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    uint32_t n = min(r.work[W_SLOW], c.survivorCapacity);
    if (gtid() == 0) r.work[W_CERTIFIED] += min(r.work[W_KEPT], c.survivorCapacity) - n;
    float margin = __uint_as_float(r.work[W_FILTER_MARGIN]);
    float reach = certificateReach(margin);
    uint32_t warps = warpStride(), warp = warpGlobal();
    if (n <= 4 * gridDim.x) {
        // A slot a list left undecided has many triangles at about its
        // nearest distance: no certificate is worth the ones within reach.
        if (c.cellListsEnabled) reach = 0.0f;
        for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) scanSlot(r, c, r.walkKey[k], margin, reach);
        return;
    }
    for (uint32_t k = 32 * warp + laneId(); k < n; k += 32 * warps) {
        uint32_t i = r.walkKey[k], t = r.walkActive[i], triangle, tie;
        float gap;
        WalkNode w = walkNode(r, t);
        uint32_t shape = r.shapeId[w.rec.y];
        float4 f = meshDistanceCertified(r, shape, w.local, gridSeed(r, shape, w.local), reach, triangle, tie, gap);
        // The triangle with its same-leaf partner and its tie, all at its
        // distance; every other one is farther by the gap.
        uint32_t at = triangle & 0x3FFFFFFFu, partner = triangle >> 30;
        if (triangle == EMPTY) at = EMPTY, partner = 0;
        certifySlot(r, c, i, t, w, f, at, partner ? at + partner : tie, partner ? tie : EMPTY, gap, margin);
    }
}
// Emits one item's hits (the warp, lane per node slot of each 32-slot half).
__device__ __forceinline__ void emitItem(const Res& r, const Config& c, uint32_t item, uint2 m) {
    uint2 cd = r.candidates[item];
    uint32_t d = cd.x, p = d >> 1, pass = d & 1;
    uint2 ij = r.pairs[p];
    uint32_t src = pass ? ij.y : ij.x, dst = pass ? ij.x : ij.y;
    uint4 range = __ldg(&r.meshClusterRanges[cd.y]);
    uint2 sm = r.candSurvMask[item];
    uint32_t out = r.candHitOffset[item], in = r.candSurvOffset[item];
#pragma unroll
    for (uint32_t half = 0; half < 2; ++half) {
        uint32_t word = half ? m.y : m.x;
        if (!((word >> laneId()) & 1u)) continue;
        uint32_t rank = (half ? __popc(m.x) : 0) + __popc(word & lanesBelow());
        uint32_t survivorRank = (half ? __popc(sm.x) : 0) + __popc((half ? sm.y : sm.x) & lanesBelow());
        uint32_t slot = out + rank, from = in + survivorRank;
        if (slot >= c.contactCapacity || from >= c.survivorCapacity) { fail(r, F_CONTACT); continue; }
        uint32_t node = __ldg(&r.meshSampleIndices[range.x + laneId() + half * WARP]);
        r.meta[slot] = make_uint4(src, dst, node, 0);
        r.pointDepth[slot] = r.hitScratch[2 * from];
        r.normalArea[slot] = r.hitScratch[2 * from + 1];
        r.contactPair[slot] = p;
    }
}
// ------------------------------------------------------------ SDF geometry
// solver.slang:188-200: trilinear signed distance and gradient from the
// target shape's grid, in the FP32 order of the reference's generated CPU
// code (lerp(x, y, s) = x + (y - x) * s, products left to right).
__device__ __forceinline__ float4 sdfQuery(const Res& r, uint32_t shape, f3 p) {
    uint4 meta = __ldg(&r.grids[shape]);
    float4 o = __ldg(&r.gridOrigin[shape]);
    f3 g = (p - xyz(o)) / o.w;
    int ax = int(floorf(g.x)), ay = int(floorf(g.y)), az = int(floorf(g.z));
    if (ax < 0 || ay < 0 || az < 0 || ax >= int(meta.y) - 1 || ay >= int(meta.z) - 1 || az >= int(meta.w) - 1)
        return make_float4(0.f, 0.f, 0.f, 1.00000002004087734e+20f);
    f3 t = g - mk(float(ax), float(ay), float(az));
    f3 u = mk(1.f, 1.f, 1.f) - t;
    float value = 0.f;
    f3 grad = mk(0.f, 0.f, 0.f);
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i)
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k) {
                f3 w = u + (t - u) * mk(float(i), float(j), float(k));
                float f = __ldg(&r.distance[meta.x + ((uint32_t(ax) + i) * meta.z + (uint32_t(ay) + j)) * meta.w +
                                            (uint32_t(az) + k)]);
                value = __fadd_rn(value, __fmul_rn(__fmul_rn(__fmul_rn(f, w.x), w.y), w.z));
                f3 v = mk(__fmul_rn(__fmul_rn(__fsub_rn(__fmul_rn(2.0f, float(i)), 1.0f), w.y), w.z),
                          __fmul_rn(__fmul_rn(__fsub_rn(__fmul_rn(2.0f, float(j)), 1.0f), w.x), w.z),
                          __fmul_rn(__fmul_rn(__fsub_rn(__fmul_rn(2.0f, float(k)), 1.0f), w.x), w.y));
                grad = grad + (f * v) / o.w;
            }
    return w4(grad, value);
}
// solver.slang:319-343 with the SDF geometry; the directed-pair branch is
// the FP64 one k_pairSetup stored (the same bits as the per-call reference).
__device__ __forceinline__ bool sdfNodeContact(const Res& r, const Config& c, uint32_t src, uint32_t dst,
                                               uint32_t node, f3 branch, float4& pd, float4& na) {
    uint32_t sid = r.shapeId[src];
    float4 sp = __ldg(&r.sample[__ldg(&r.sampleInfo[sid].x) + node]);
    float4 bs = r.body[src], bd = r.body[dst];
    f3 arm = qrot(r.rotation[src], xyz(sp) * bs.x);
    f3 local = qinv(r.rotation[dst], arm - branch) / bd.x;
    // Beyond the target's bounding radius by more than a grid-cell diagonal,
    // all eight grid values around the node are distances of points outside
    // the shape (positive), so the interpolated distance is positive: no
    // contact, as the full query would find; skip its grid loads.
    float reach = __fadd_rn(__fdiv_rn(bd.z, bd.x), __fmul_rn(1.7339f, __ldg(&r.gridOrigin[r.shapeId[dst]].w)));
    if (dot(local, local) > __fmul_rn(reach, reach)) return false;
    float4 f = sdfQuery(r, r.shapeId[dst], local);
    pd = w4(arm, __fmul_rn(-f.w, bd.x));
    if (pd.w <= 0.0f) return false;
    f3 grad = qrot(r.rotation[dst], xyz(f));
    float len = length(grad);
    if (len < 1.00000001168609742e-07f || !isfinite(pd.w)) { fail(r, F_DEGENERATE); return false; }
    na = w4(grad / len, __fmul_rn(__fmul_rn(sp.w, bs.x), bs.x));
    if (pd.w > __fmul_rn(c.maxOverlap, mn(bs.w, bd.w))) fail(r, F_PENETRATION);
    return true;
}
// One direction of a pair for the reach test of its source's nodes: a node at
// x (source frame) lies at squared distance s^2 |x|^2 - 2 s x.b' + |b|^2 from
// the target's centre, b' the branch in the source frame and s the source's
// scale.  `limit` is the squared reach of sdfNodeContact's own test in world
// units, grown by 1e-4 of the magnitudes involved -- far above the FP32
// rounding of either form -- so a node beyond it fails that test too.
struct SdfReach {
    f3 branch;  // 2 s b'
    float scale, square, limit;
    const float4* samples;
};
__device__ __forceinline__ SdfReach sdfReach(const Res& r, uint32_t src, uint32_t dst, f3 branch) {
    SdfReach k;
    float4 bs = r.body[src], bd = r.body[dst];
    const uint32_t shape = r.shapeId[src];
    k.branch = (2.0f * bs.x) * qinv(r.rotation[src], branch);
    k.scale = bs.x * bs.x;
    k.square = dot(branch, branch);
    float reach = bd.z + 1.7339f * __ldg(&r.gridOrigin[r.shapeId[dst]].w) * bd.x;
    float size = bs.z + sqrtf(k.square) + reach;
    k.limit = reach * reach + 1e-4f * size * size;
    k.samples = r.sample + __ldg(&r.sampleInfo[shape].x);
    return k;
}
__device__ __forceinline__ bool sdfBeyond(const SdfReach& k, float4 x) {
    float xx = x.x * x.x + x.y * x.y + x.z * x.z;
    return k.scale * xx - (x.x * k.branch.x + x.y * k.branch.y + x.z * k.branch.z) + k.square > k.limit;
}
// The contacts of every pair (countContacts and emitContacts' evaluation,
// solver.slang:536-565), a warp a pair: the nodes s of both grains in order,
// the second's after the first's.  Nearly all lie beyond the other grain's
// reach: one pass over the samples (one load and a dozen operations a node)
// lists those that do not in shared memory, and the lanes evaluate the listed
// ones together, once each.  A contact goes to a scratch slot with its pair,
// s and its rank among the earlier contacts of its virtual lane (s mod 64) of
// the reference's 64-thread group; the lanes' counts are kept for
// k_sdfEmit, which puts the pair's contacts in the reference's order (lane,
// then node).  Evaluating every node in a counting and in an emitting pass,
// a lane each in turn, took 104 of a step's 147 us for 1,000 spheres of 512
// nodes; a step takes 68 us now (180 -> 98 for 2,197 rough grains).
constexpr uint32_t SDF_LIST = 64;  // listed nodes at most: a batch of 32 and a round's addition
__device__ __forceinline__ void sdfQueryPairs(const Params& P, uint32_t* list, uint32_t* counts, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    const uint32_t pairs = activePairs(r, c), lane = laneId();
    for (uint32_t p = warpGlobal(); p < pairs; p += warpStride()) {
        const uint2 ij = r.pairs[p];
        const f3 b0 = xyz(r.dpairBranch[2 * p]), b1 = xyz(r.dpairBranch[2 * p + 1]);
        const SdfReach reach[2] = {sdfReach(r, ij.x, ij.y, b0), sdfReach(r, ij.y, ij.x, b1)};
        const uint32_t first = __ldg(&r.sampleInfo[r.shapeId[ij.x]].y);
        const uint32_t nodes[2] = {first, __ldg(&r.sampleInfo[r.shapeId[ij.y]].y)};
        __syncwarp();
        counts[lane] = counts[lane + WARP] = 0;
        uint32_t listed = 0, total = 0;
        // The first `n` listed nodes (at most 32), in order.
        auto evaluate = [&](uint32_t n) {
            __syncwarp();
            const uint32_t s = lane < n ? list[lane] : 0u;
            float4 pd, na;
            bool hit = false;
            if (lane < n) {
                const bool second = s >= first;
                hit = sdfNodeContact(r, c, second ? ij.y : ij.x, second ? ij.x : ij.y, second ? s - first : s,
                                     second ? b1 : b0, pd, na);
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, hit);
            if (hits == 0) return;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&r.work[W_SURVIVORS], uint32_t(__popc(hits)));
            base = __shfl_sync(0xffffffffu, base, 0);
            total += __popc(hits);
            const uint32_t v = hit ? s & 63u : 64u + lane;
            const uint32_t same = __match_any_sync(0xffffffffu, v);
            const uint32_t rank = hit ? counts[v] + __popc(same & lanesBelow()) : 0u;
            __syncwarp();
            if (hit && (same & ~lanesBelow()) >> lane == 1u) counts[v] = rank + 1;  // the last of its lane
            __syncwarp();
            if (hit) {
                const uint32_t slot = base + __popc(hits & lanesBelow());
                if (slot >= c.survivorCapacity) {
                    fail(r, F_CONTACT);
                } else {
                    r.walkNode[slot] = make_uint4(p, s, rank, 0u);
                    r.hitScratch[2 * size_t(slot)] = pd;
                    r.hitScratch[2 * size_t(slot) + 1] = na;
                }
            }
        };
        for (uint32_t side = 0; side < 2; ++side) {
            const SdfReach& k = reach[side];
            const uint32_t n = nodes[side], offset = side ? first : 0u;
            for (uint32_t k0 = 0; k0 < n; k0 += 4 * WARP) {
                float4 x[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t node = k0 + WARP * j + lane;
                    x[j] = node < n ? __ldg(&k.samples[node]) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t node = k0 + WARP * j + lane;
                    const bool near = node < n && !sdfBeyond(k, x[j]);
                    const uint32_t ballot = __ballot_sync(0xffffffffu, near);
                    if (ballot == 0) continue;
                    if (near) list[listed + __popc(ballot & lanesBelow())] = offset + node;
                    listed += __popc(ballot);
                    if (listed >= WARP) {
                        evaluate(WARP);
                        listed -= WARP;
                        __syncwarp();
                        const uint32_t rest = lane < listed ? list[WARP + lane] : 0u;
                        __syncwarp();
                        if (lane < listed) list[lane] = rest;
                    }
                }
            }
        }
        if (listed) evaluate(listed);
        __syncwarp();
        r.sdfLaneCounts[size_t(WARP) * p + lane] = counts[lane] | (counts[lane + WARP] << 16);  // each below 65,536 (the host checks)
        if (lane == 0) r.contactCounts[p] = total;
    }
}

// ---------------------------------------------------------------- friction
// solver.slang:691-696
__device__ __forceinline__ f3 transported(f3 x, f3 a, f3 b, float spin) {
    float cc = mn(mx(dot(a, b), -1.0f), 1.0f);
    if (cc < -0.999999f) return mk(0.f, 0.f, 0.f);
    f3 v = cross(a, b);
    f3 out = (x + cross(v, x)) + cross(v, cross(v, x)) / __fadd_rn(1.0f, cc);
    float cs = cosf(spin), sn = sinf(spin);
    out = (out * cs + cross(b, out) * sn) + (b * dot(b, out)) * __fsub_rn(1.0f, cs);
    return out - b * dot(out, b);
}
// normal.slang:2-11
__device__ __forceinline__ void normalResponse(float depth, float area, float vn, float stiffness, float viscosity,
                                               float weight, float& force, float& lossPower) {
    force = 0.f;
    lossPower = 0.f;
    if (depth <= 0) return;
    float elastic = __fmul_rn(__fmul_rn(__fmul_rn(weight, stiffness), area), depth);
    force = viscosity == 0 ? elastic
                           : mx(0.0f, __fsub_rn(elastic, __fmul_rn(__fmul_rn(__fmul_rn(weight, viscosity), area), vn)));
    lossPower = mx(0.0f, __fmul_rn(__fsub_rn(elastic, force), vn));
}
// History key within a pair: direction (source > target) then the node's
// position in its shape's cluster order; runs of one pair are sorted by it.
// With the SDF geometry a pair's contacts are in the reference emit order:
// s = node (first grain) or V_first + node (second grain), taken by virtual
// lane s mod 64, then s / 64.
__device__ __forceinline__ uint32_t pairKey(const Res& r, const Config& c, uint32_t src, uint32_t dst,
                                            uint32_t node) {
    if (c.meshGeometry == 0) {
        uint32_t s = src > dst ? __ldg(&r.sampleInfo[r.shapeId[dst]].y) + node : node;
        return ((s & 63u) << 24) | (s >> 6);
    }
    return (src > dst ? 0x80000000u : 0u) | __ldg(&r.meshSampleRank[__ldg(&r.sampleInfo[r.shapeId[src]].x) + node]);
}
// Slot of key (src, dst, node) among the committed contacts, or EMPTY.
// The committed side stores, per grain a, the run of its pairs (a, b) with
// b > a and, per pair, its contacts sorted by pairKey: a sorted merge done as
// a run lookup plus a binary search.
__device__ __forceinline__ uint32_t historySlot(const Res& r, const Config& c, uint32_t src, uint32_t dst,
                                                uint32_t node) {
    uint32_t a = min(src, dst), b = max(src, dst);
    uint32_t begin = r.oldPairOffsets[a], end = r.oldPairOffsets[a + 1];
    uint32_t q = EMPTY;
    for (uint32_t k = begin; k < end; ++k)
        if (r.oldPairB[k] == b) { q = k; break; }
    if (q == EMPTY) return EMPTY;
    uint32_t lo = r.oldContactStart[q], hi = r.oldContactStart[q + 1];
    uint32_t key = pairKey(r, c, src, dst, node);
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        uint4 m = r.oldMeta[mid];
        uint32_t mk2 = pairKey(r, c, m.x, m.y, m.z);
        if (mk2 < key) lo = mid + 1;
        else hi = mid;
    }
    if (lo < r.oldContactStart[q + 1]) {
        uint4 m = r.oldMeta[lo];
        if (m.x == src && m.y == dst && m.z == node) return lo;
    }
    return EMPTY;
}
// ------------------------------------------------------------------ planes
// Signed distance of a grain surface point (centre + arm) from the plane
// (solver.slang:605-610), from the centre's two-sum.
__device__ __forceinline__ float localWallDistance(const Res& r, uint32_t wall, Sum2 centre, f3 arm) {
    Sum2 sum = wallAddDot(centre, xyz(r.wallPlane[wall]), arm);
    sum = wallAddDot(sum, xyz(r.wallRemainder[wall]), arm);
    return __fadd_rn(sum.hi, sum.lo);
}
// The per-(wall, grain) terms of the cluster bound (solver.slang:613-624):
// the plane normal in the grain's scaled frame, the centre distance and the
// grain-independent part of the FP32 pad.
struct WallFrame {
    f3 normal;
    float normalLength, base, padBase;
};
__device__ __forceinline__ WallFrame wallFrame(const Res& r, uint32_t body, uint32_t wall, float base) {
    float4 plane = r.wallPlane[wall];
    WallFrame f;
    f.normal = qinv(r.rotation[body], xyz(plane)) * r.body[body].x;
    f.normalLength = length(f.normal);
    f.base = base;
    f.padBase = __fadd_rn(__fadd_rn(1.0f, fabsf(plane.w)), length(xyz(r.position[body])));
    return f;
}
// solver.slang:613-624: whether any node of a sample cluster can reach
// behind the plane (fixed-normal support bound with an FP32 pad).
__device__ __forceinline__ bool wallClusterMayContact(const Res& r, const WallFrame& f, uint32_t cluster) {
    f3 low = xyz(__ldg(&r.meshClusterMin[cluster])), high = xyz(__ldg(&r.meshClusterMax[cluster]));
    f3 center = 0.5f * (low + high), half = 0.5f * (high - low);
    float support = __fsub_rn(dot(f.normal, center), dot(abs3(f.normal), half));
    float pad = __fmul_rn(__fmul_rn(64.0f, 1.1920928955078125e-7f),
                          __fadd_rn(f.padBase, __fmul_rn(f.normalLength, __fadd_rn(length(center), length(half)))));
    return __fadd_rn(f.base, support) <= pad;
}
// solver.slang:625-638: node `node` of grain `body` behind the plane, with
// its record (arm and depth; plane normal and node area).  `flag` raises the
// non-finite and penetration flags (once per step: in the counting pass).
__device__ __forceinline__ bool wallNode(const Res& r, const Config& c, uint32_t body, uint32_t wall, Sum2 centre,
                                        uint32_t node, bool flag, float4& pd, float4& na) {
    float4 point = __ldg(&r.sample[__ldg(&r.sampleInfo[r.shapeId[body]].x) + node]);
    float4 b = r.body[body];
    f3 arm = qrot(r.rotation[body], xyz(point) * b.x);
    float phi = localWallDistance(r, wall, centre, arm);
    if (!isfinite(phi)) {
        if (flag) fail(r, F_NONFINITE);
        return false;
    }
    if (phi >= 0) return false;
    if (flag && -phi > __fmul_rn(c.maxOverlap, b.w)) fail(r, F_PENETRATION);
    pd = w4(arm, -phi);
    na = w4(xyz(r.wallPlane[wall]), __fmul_rn(__fmul_rn(point.w, b.x), b.x));
    return true;
}
// Whether grain `body` may reach behind plane `wall`: the centre-distance
// early-out of collectWallContacts (solver.slang:642-653), one lane per item.
__device__ __forceinline__ bool wallReach(const Res& r, uint32_t body, uint32_t wall, Sum2& centre) {
    float4 plane = r.wallPlane[wall];
    centre = wallCentreDistance(r, body, wall);
    float phi = __fadd_rn(centre.hi, centre.lo);
    float pad = __fmul_rn(__fmul_rn(64.0f, 1.1920928955078125e-7f),
                          __fadd_rn(__fadd_rn(1.0f, length(xyz(r.position[body]))), fabsf(plane.w)));
    return !(phi > __fadd_rn(r.body[body].z, pad));
}
// The plane contacts of one (wall, grain) item that passed the early-out, in
// the reference CPU collector's order (cpu_scheduling.slang:133-154): the
// grain's nodes in order (SDF geometry), or its sample clusters in preorder
// -- a cluster the plane cannot reach skips its subtree -- and each visited
// cluster's nodes in order (mesh geometry).  One warp: the 32 clusters from
// the walk's cursor are bounded at once (one per lane), then the walk
// advances through them with the lanes' results; nodes are tested 32 per
// round, order kept by ballot ranks.  Each contact is listed in hitScratch (its
// rows are free once the grain contacts are written) as item, node and rank
// within the item, in any order of the items: lane v keeps round v's hits until
// 32 rounds are full or the item ends, so that an item costs one atomic and not
// one a round.  Returns the count.
inline __device__ uint32_t wallItem(const Res& r, const Config& c, uint32_t item, Sum2 centre) {
    uint32_t body = item % c.N, wall = item / c.N, lane = laneId();
    float phi = __fadd_rn(centre.hi, centre.lo);
    uint32_t shape = r.shapeId[body], count = 0, listed = 0, rounds = 0, heldMask = 0, heldFrom = 0;
    uint4* list = reinterpret_cast<uint4*>(r.hitScratch);
    auto flush = [&]() {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&r.work[W_WALL_HITS], count - listed);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (uint32_t v = 0; v < rounds; ++v) {
            const uint32_t mask = __shfl_sync(0xffffffffu, heldMask, int(v)), from = __shfl_sync(0xffffffffu, heldFrom, int(v));
            if ((mask >> lane) & 1u) {
                const uint32_t e = at + __popc(mask & lanesBelow()), rank = listed + __popc(mask & lanesBelow());
                const uint32_t node = c.meshGeometry == 0 ? from + lane : __ldg(&r.meshSampleIndices[from + lane]);
                if (e < 2 * c.survivorCapacity) list[e] = make_uint4(item, node, rank, 0u);
                else fail(r, F_CONTACT);
            }
            at += __popc(mask);
            listed += __popc(mask);
        }
        rounds = 0;
    };
    // A round: the nodes of places from + lane.
    auto visit = [&](uint32_t from, bool valid, uint32_t node) {
        float4 pd, na;
        bool hit = valid && wallNode(r, c, body, wall, centre, node, true, pd, na);
        uint32_t mask = __ballot_sync(0xffffffffu, hit);
        if (mask == 0) return;
        if (lane == rounds) {
            heldMask = mask;
            heldFrom = from;
        }
        count += __popc(mask);
        if (++rounds == WARP) flush();
    };
    if (c.meshGeometry == 0) {
        uint32_t nodes = __ldg(&r.sampleInfo[shape].y);
        for (uint32_t base = 0; base < nodes; base += WARP) visit(base, base + lane < nodes, base + lane);
        if (rounds) flush();
        return count;
    }
    WallFrame frame = wallFrame(r, body, wall, phi);
    uint4 info = __ldg(&r.meshClusterInfo[shape]);
    uint32_t end = info.x + info.y, cursor = info.x;
    // Every window moves the cursor forward (escape links point forward; a
    // link that does not ends the walk).
    for (uint32_t guard = 0; cursor < end && guard < info.y; ++guard) {
        uint32_t window = cursor, cl = window + lane;
        bool candidate = cl < end && wallClusterMayContact(r, frame, cl);
        uint4 range = cl < end ? __ldg(&r.meshClusterRanges[cl]) : make_uint4(0u, 0u, 0u, 0u);
        uint32_t mask = __ballot_sync(0xffffffffu, candidate);
        while (cursor < end && cursor - window < WARP) {
            uint32_t k = cursor - window;
            uint32_t x = __shfl_sync(0xffffffffu, range.x, int(k)), y = __shfl_sync(0xffffffffu, range.y, int(k));
            uint32_t z = __shfl_sync(0xffffffffu, range.z, int(k));
            if ((mask >> k) & 1u) {
                for (uint32_t base = 0; base < y; base += WARP) {
                    uint32_t n = base + lane;
                    visit(x + base, n < y, n < y ? __ldg(&r.meshSampleIndices[x + n]) : 0u);
                }
                ++cursor;
            } else {
                cursor = z > cursor ? z : end;
            }
        }
    }
    if (rounds) flush();
    return count;
}
// Plane contacts per (wall, grain), wall-major: each lane runs the early-out
// of one item, then the warp collects its items that pass, one after the
// other.  A warp's 32 items are a grid of warps apart: the grains near a wall
// are runs of consecutive items, spread this way over many warps.  Records
// where the plane contacts start.
__device__ __forceinline__ void wallCount(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    if (gtid() == 0) r.work[W_WALL_BASE] = r.control[2];
    uint32_t items = c.N * c.wallCount, lane = laneId(), stride = warpStride(), first = warpGlobal();
    for (uint32_t base = 0; base < items; base += stride * WARP) {
        uint32_t item = base + lane * stride + first;
        Sum2 centre{0.f, 0.f};
        bool reach = item < items && wallReach(r, item % c.N, item / c.N, centre);
        if (item < items && !reach) r.wallCounts[item] = 0;
        for (uint32_t mask = __ballot_sync(0xffffffffu, reach); mask; mask &= mask - 1u) {
            uint32_t k = __ffs(mask) - 1u, it = base + k * stride + first;
            Sum2 ck{__shfl_sync(0xffffffffu, centre.hi, int(k)), __shfl_sync(0xffffffffu, centre.lo, int(k))};
            uint32_t n = wallItem(r, c, it, ck);
            if (lane == 0) r.wallCounts[it] = n;
        }
    }
}
// The plane contacts appended after the grain-grain ones (gpu.py:544-545),
// per-(wall, grain) starts and the new contact total.
__device__ __forceinline__ void wallEmit(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    uint32_t items = c.N * c.wallCount, base0 = r.work[W_WALL_BASE];
    for (uint32_t i = gtid(); i <= items; i += gstride()) r.sideWallStart[i] = base0 + r.wallOffsets[i];
    if (gtid() == 0) {
        uint32_t total = base0 + r.wallOffsets[items];
        r.control[2] = total;
        if (total > c.contactCapacity) fail(r, F_CONTACT);
    }
    // A lane a listed contact; the items' walks a second time took 41 us for
    // 4,913 grains in a box.
    const uint4* list = reinterpret_cast<const uint4*>(r.hitScratch);
    const uint32_t n = min(r.work[W_WALL_HITS], 2 * c.survivorCapacity);
    for (uint32_t e = gtid(); e < n; e += gstride()) {
        const uint4 x = list[e];
        const uint32_t body = x.x % c.N, wall = x.x / c.N, out = base0 + r.wallOffsets[x.x] + x.z;
        if (out >= c.contactCapacity) continue;
        float4 pd, na;
        wallNode(r, c, body, wall, wallCentreDistance(r, body, wall), x.y, false, pd, na);
        r.meta[out] = make_uint4(body, c.N + wall, x.y, 1u);
        r.pointDepth[out] = pd;
        r.normalArea[out] = na;
    }
}
// Within one (wall, grain) run, the order of a node's contact: its position in
// the grain's cluster order (mesh) or its index (SDF).
__device__ __forceinline__ uint32_t wallKey(const Res& r, const Config& c, uint32_t body, uint32_t node) {
    return c.meshGeometry == 0 ? node : __ldg(&r.meshSampleRank[__ldg(&r.sampleInfo[r.shapeId[body]].x) + node]);
}
// Slot of the committed plane contact (body, wall, node), or EMPTY: binary
// search of the committed (wall, grain) run.
__device__ __forceinline__ uint32_t wallHistorySlot(const Res& r, const Config& c, uint32_t body, uint32_t wall,
                                                    uint32_t node) {
    uint32_t item = wall * c.N + body;
    uint32_t lo = r.oldWallStart[item], end = r.oldWallStart[item + 1], hi = end;
    uint32_t key = wallKey(r, c, body, node);
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (wallKey(r, c, body, r.oldMeta[mid].z) < key) lo = mid + 1;
        else hi = mid;
    }
    if (lo < end) {
        uint4 m = r.oldMeta[lo];
        if (m.x == body && m.y == c.N + wall && m.z == node) return lo;
    }
    return EMPTY;
}
// solver.slang:702-733 with plane.slang:13-36: a plane contact.
__device__ __forceinline__ void resolveWall(const Res& r, const Config& c, uint32_t id, uint4 key) {
    uint32_t i = key.x, w = key.y - c.N;
    float4 m = r.wallMaterial[w];
    float viscosity = m.w;
    f3 nrm = xyz(r.normalArea[id]);
    f3 wi = viscosity > 0 ? xyz(r.forceOmega[i]) : omegaOf(r, i);
    f3 elastic = mk(0.f, 0.f, 0.f);
    if (c.historyStep != 0) {
        uint32_t old = wallHistorySlot(r, c, i, w, key.z);
        if (old != EMPTY)
            elastic = transported(xyz(r.oldSlip[old]), xyz(r.oldNormal[old]), nrm,
                                  __fmul_rn(__fmul_rn(0.5f, dot(wi + mk(0.f, 0.f, 0.f), nrm)), c.dt));
    }
    f3 arm = xyz(r.pointDepth[id]);
    f3 v = viscosity > 0 ? xyz(r.forceVelocity[i]) : xyz(r.velocity[i]) + xyz(r.velocityRemainder[i]);
    f3 rv = (v + cross(wi, arm)) - xyz(r.wallVelocity[w]);
    float4 forceEnergy = make_float4(0.f, 0.f, 0.f, 0.f), slipLoss = forceEnergy;
    float lossPower = 0.f;
    bool sliding = false;
    float signedDistance = -r.pointDepth[id].w, area = r.normalArea[id].w;
    if (signedDistance < 0) {
        float depth = -signedDistance;
        f3 tangent = rv - nrm * dot(rv, nrm);
        f3 trial = (elastic - nrm * dot(elastic, nrm)) + c.dt * tangent;
        f3 slip = trial;
        float fn;
        normalResponse(depth, area, dot(rv, nrm), m.x, viscosity, 1.0f, fn, lossPower);
        f3 ft = __fmul_rn(-m.y, area) * slip;
        float magnitude = length(ft);
        if (magnitude > __fmul_rn(m.z, fn) && magnitude > 0) {
            sliding = true;
            ft = ft * __fdiv_rn(__fmul_rn(m.z, fn), magnitude);
            slip = (-ft) / __fmul_rn(m.y, area);
        }
        forceEnergy = w4(fn * nrm + ft, __fmul_rn(__fmul_rn(0.5f, area), __fadd_rn(__fmul_rn(__fmul_rn(m.x, depth), depth),
                                                                               __fmul_rn(m.y, dot(slip, slip)))));
        slipLoss = w4(slip, mx(0.0f, -dot(ft, trial - slip)));
    }
    r.slip[id] = slipLoss;
    r.contactForce[id] = forceEnergy;
    r.normalLossPower[id] = lossPower;
    if (!isfinite(forceEnergy.x) || !isfinite(forceEnergy.y) || !isfinite(forceEnergy.z) || !isfinite(forceEnergy.w) ||
        !isfinite(lossPower)) {
        fail(r, F_NONFINITE);
        return;
    }
    if (sliding) atomicAdd(&r.control[6], 1u);
}
// solver.slang:834-856: per (wall, grain), the reaction, its moment about
// the origin and the wall power over the grain's contacts with that wall, in
// its linked-list order (descending contact id), and the accumulated work.
__device__ __forceinline__ void gatherWallRows(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0) return;
    uint32_t items = c.N * c.wallCount;
    for (uint32_t item = gtid(); item < items; item += gstride()) {
        uint32_t body = item % c.N, wall = item / c.N;
        uint32_t lo = r.sideWallStart[item], hi = r.sideWallStart[item + 1];
        f3 centre = mk(0.f, 0.f, 0.f), velocity = centre;
        if (hi > lo) {
            centre = xyz(r.position[body]) + xyz(r.positionRemainder[body]);
            velocity = xyz(r.wallVelocity[wall]);
        }
        f3 reaction = mk(0.f, 0.f, 0.f), moment = reaction;
        float power = 0.f;
        // From the last contact; four loaded before the first is added (one at
        // a time: 23 us for 4,913 grains in a box, a load's latency a contact).
        for (uint32_t k = hi; k > lo;) {
            const uint32_t n = min(k - lo, 4u);
            float4 f[4], p[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (u >= n) break;
                f[u] = r.contactForce[k - 1 - u];
                p[u] = r.pointDepth[k - 1 - u];
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (u >= n) break;
                f3 force = xyz(f[u]);
                f3 point = centre + xyz(p[u]);
                reaction = reaction - force;
                moment = moment - cross(point, force);
                power = __fadd_rn(power, dot(force, velocity));
            }
            k -= n;
        }
        float4 work = r.wallAccumulated[item];
        r.wallRows[3 * item] = w4(reaction, __uint_as_float(hi - lo));
        r.wallRows[3 * item + 1] = w4(moment, power);
        r.wallRows[3 * item + 2] = make_float4(__fadd_rn(work.x, work.y), 0.f, 0.f, 0.f);
    }
}

// solver.slang:702-733: the plane contacts, after the grain-grain ones.
__device__ __forceinline__ void resolveWalls(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0) return;
    uint32_t n = activeContacts(r, c);
    for (uint32_t id = min(r.work[W_WALL_BASE], n) + gtid(); id < n; id += gstride()) resolveWall(r, c, id, r.meta[id]);
}
// solver.slang:702-749: the law of grain-grain contact `id` (source i, target
// j, normal and area, arm and depth, branch), with the slip of its committed
// slot `old` (EMPTY: none).  Returns whether it slides.
__device__ __forceinline__ bool resolveGrain(const Res& r, const Config& c, uint32_t id, uint32_t i, uint32_t j,
                                             float4 na, float4 pd, f3 branch, uint32_t old) {
    f3 nrm = xyz(na), arm = xyz(pd);
    float viscosity = c.normalViscosity;
    f3 wi = viscosity > 0 ? xyz(r.forceOmega[i]) : omegaOf(r, i);
    f3 wj = viscosity > 0 ? xyz(r.forceOmega[j]) : omegaOf(r, j);
    f3 elastic = mk(0.f, 0.f, 0.f);
    if (old != EMPTY)
        elastic = transported(xyz(r.oldSlip[old]), xyz(r.oldNormal[old]), nrm,
                              __fmul_rn(__fmul_rn(0.5f, dot(wi + wj, nrm)), c.dt));
    f3 translation = viscosity > 0 ? xyz(r.forceVelocity[i]) - xyz(r.forceVelocity[j])
                                   : xyz(r.velocity[i]) - xyz(r.velocity[j]);
    f3 rv = ((translation - xyz(r.cell[3 * specimenOf(r, i) + 1]) * branch) + cross(wi, arm)) - cross(wj, arm - branch);
    elastic = elastic + (rv - nrm * dot(rv, nrm)) * c.dt;
    f3 trial = elastic;
    float area = na.w, depth = pd.w;
    float fn, lossPower;
    normalResponse(depth, area, dot(rv, nrm), c.kn, viscosity, 0.5f, fn, lossPower);
    r.normalLossPower[id] = lossPower;
    float ktA = __fmul_rn(__fmul_rn(-0.5f, c.kt), area);
    f3 ft = ktA * elastic;
    float magnitude = length(ft);
    bool sliding = magnitude > __fmul_rn(c.mu, fn) && magnitude > 0;
    if (sliding) {
        ft = ft * __fdiv_rn(__fmul_rn(c.mu, fn), magnitude);
        elastic = (-ft) / __fmul_rn(__fmul_rn(0.5f, c.kt), area);
    }
    r.slip[id] = w4(elastic, mx(0.0f, -dot(ft, trial - elastic)));
    float4 cf = w4(fn * nrm + ft,
                   __fmul_rn(__fmul_rn(0.25f, area), __fadd_rn(__fmul_rn(__fmul_rn(c.kn, depth), depth),
                                                               __fmul_rn(c.kt, dot(elastic, elastic)))));
    r.contactForce[id] = cf;
    if (!isfinite(cf.x) || !isfinite(cf.y) || !isfinite(cf.z) || !isfinite(cf.w) || !isfinite(lossPower))
        fail(r, F_NONFINITE);
    return sliding;
}
// The contact records of a stored exact-query list, and with `Law` the
// contact law of each in the same pass (the step; the named phases of a
// dispatch run them apart).  The active slots are in contact order, so this
// is a stream compaction: a warp takes 32 slots, adds up the hits before them
// (hitsBefore), and the slots that hit write their contacts in place,
// consecutive lanes to consecutive contacts.  The first slot of each pair
// also writes the pair's first contact (for the pairs before it without
// slots too).  A slot keeps the contact it became (walkContact): on the next
// step that contact's committed key is its own, which spares the search of
// the pair's committed run; where the key does not match (another step's
// contacts were committed) or the slot was no contact, the search decides.
template <bool Law>
__device__ __forceinline__ void emitSlots(const Params& P, bool live) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    const SlotHits hits = slotHits(r, c);
    const uint32_t n = min(r.work[W_ACTIVE], c.survivorCapacity), pairs = activePairs(r, c), lane = laneId();
    if (n == 0) {
        for (uint32_t p = gtid(); p <= pairs; p += gstride()) r.sideContactStart[p] = 0;
        return;
    }
    // Contacts on the committed side: a hint must lie below them.
    const uint32_t committed = Law && c.historyStep != 0 ? r.oldContactStart[r.oldPairOffsets[c.N]] : 0u;
    for (uint32_t w = warpGlobal(); 32 * w < n; w += warpStride()) {
        const uint32_t i = 32 * w + lane;
        const bool valid = i < n;
        const uint32_t t = valid ? r.walkActive[i] : 0u;
        const uint4 rec = valid ? r.walkNode[t] : make_uint4(0u, 0u, 2 * pairs, 0u);
        const uint32_t word = hits.words[w], pair = rec.z >> 1;
        const bool hit = (word >> lane) & 1u;
        // This slot's contact index, or the next one's.
        const uint32_t contact = hitsBefore(hits, w) + __popc(word & lanesBelow());
        uint32_t from = __shfl_up_sync(0xffffffffu, pair, 1) + 1;
        if (lane == 0) from = i == 0 ? 0u : (r.walkNode[r.walkActive[i - 1]].z >> 1) + 1;
        // First contacts of the pairs up to this slot's; of the rest after the last slot.
        const uint32_t upTo = valid ? pair + 1 : from;
        if (valid && upTo - from <= 4)
            for (; from < upTo; ++from) r.sideContactStart[from] = contact;
        const bool last = i == n - 1;
        for (uint32_t wide = __ballot_sync(0xffffffffu, from < upTo || last); wide; wide &= wide - 1) {
            uint32_t k = __ffs(wide) - 1, first = __shfl_sync(0xffffffffu, from, k), end = __shfl_sync(0xffffffffu, upTo, k);
            uint32_t value = __shfl_sync(0xffffffffu, contact, k);
            for (uint32_t q = first + lane; q < end; q += WARP) r.sideContactStart[q] = value;
            if (__shfl_sync(0xffffffffu, uint32_t(last), k)) {
                uint32_t total = value + __shfl_sync(0xffffffffu, uint32_t(hit), k);
                for (uint32_t q = end + lane; q <= pairs; q += WARP) r.sideContactStart[q] = total;
                if (lane == 0) {
                    r.control[2] = total;
                    if (total > c.contactCapacity) fail(r, F_CONTACT);
                }
            }
        }
        bool sliding = false;
        if (hit && contact < c.contactCapacity) {
            const float4 pd = r.hitScratch[2 * size_t(t)], na = r.hitScratch[2 * size_t(t) + 1];
            const uint32_t node = rec.w - __ldg(&r.sampleInfo[r.shapeId[rec.x]].x);
            r.meta[contact] = make_uint4(rec.x, rec.y, node, 0);
            r.pointDepth[contact] = pd;
            r.normalArea[contact] = na;
            if (Law) {
                uint32_t old = EMPTY;
                if (c.historyStep != 0) {
                    uint32_t hint = r.walkContact[t];
                    if (hint < committed) {
                        uint4 m = r.oldMeta[hint];
                        if (m.x == rec.x && m.y == rec.y && m.z == node) old = hint;
                    }
                    if (old == EMPTY) old = historySlot(r, c, rec.x, rec.y, node);
                }
                sliding = resolveGrain(r, c, contact, rec.x, rec.y, na, pd, xyz(r.dpairBranch[rec.z]), old);
            } else {
                r.contactPair[contact] = pair;
            }
            r.walkContact[t] = contact;
        }
        uint32_t slides = __popc(__ballot_sync(0xffffffffu, sliding));
        if (lane == 0 && slides) atomicAdd(&r.control[6], slides);
    }
}

// The SDF contacts from their scratch slots to their places -- the pair's
// first contact, the contacts of its lower virtual lanes, the rank in the
// lane -- with the contact law of each where `Law` (see emitSlots), and the
// per-pair contact starts of the history side being written.
template <bool Law>
__device__ __forceinline__ void sdfEmit(const Params& P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t pairs = activePairs(r, c);
    uint32_t total = r.control[2];
    if (total > c.contactCapacity) fail(r, F_CONTACT);
    if (r.control[0] != 0) return;
    const uint32_t n = min(r.work[W_SURVIVORS], c.survivorCapacity);
    for (uint32_t slot = gtid(); slot < n; slot += gstride()) {
        const uint4 rec = r.walkNode[slot];
        const uint32_t p = rec.x, v = rec.y & 63u;
        const uint4* lanes = reinterpret_cast<const uint4*>(r.sdfLaneCounts + size_t(WARP) * p);
        uint32_t contact = r.contactOffsets[p] + rec.z;
        // Lanes below 32 in the low halves, the others in the high halves.
#pragma unroll
        for (uint32_t q = 0; q < WARP / 4; ++q) {
            const uint4 w = lanes[q];
            const uint32_t word[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t l = 4 * q + j;
                if (l < v) contact += word[j] & 0xFFFFu;
                if (l + WARP < v) contact += word[j] >> 16;
            }
        }
        const uint2 ij = r.pairs[p];
        const uint32_t first = __ldg(&r.sampleInfo[r.shapeId[ij.x]].y);
        const bool second = rec.y >= first;
        const uint32_t i = second ? ij.y : ij.x, j = second ? ij.x : ij.y, node = second ? rec.y - first : rec.y;
        const float4 pd = r.hitScratch[2 * size_t(slot)], na = r.hitScratch[2 * size_t(slot) + 1];
        r.meta[contact] = make_uint4(i, j, node, 0);
        r.pointDepth[contact] = pd;
        r.normalArea[contact] = na;
        if (Law) {
            const uint32_t old = c.historyStep != 0 ? historySlot(r, c, i, j, node) : EMPTY;
            if (resolveGrain(r, c, contact, i, j, na, pd, xyz(r.dpairBranch[2 * p + (second ? 1 : 0)]), old))
                atomicAdd(&r.control[6], 1u);
        } else {
            r.contactPair[contact] = p;
        }
    }
    for (uint32_t p = gtid(); p <= pairs; p += gstride()) r.sideContactStart[p] = p < pairs ? r.contactOffsets[p] : total;
}

// -------------------------------------------------------------------- gather
// solver.slang:760-811, one warp per grain.  Contacts of grain g are taken in
// the order the reference's linked lists hold them (descending contact id):
// pairs where g is first (a contiguous run) and second (the byJ run) merged
// from the highest pair id down, each pair's contacts from the last.  Lanes
// load and evaluate 32 contacts at a time and store their terms in shared
// memory; every accumulator component is an independent sequential chain
// (the compensated force and torque sums are componentwise), so lane j then
// replays chain j over the 32 terms in that order: the sums are
// bit-identical to the serial loop, with 22 chains advancing in parallel.
struct GatherTerms {
    f3 force, torque, s0, s1, s2;
    float energy, denom, depth, dissipation, normalPower, stiffness, viscous;
};
// Accumulator chains: 0-2 force and 3-5 torque (compensated), 6-14 the three
// stress rows (stored negated), 15 energy, 16 denominator, 17 deepest overlap
// (maximum), 18 dissipation, 19 normal loss power, 20-21 timestep rates.
constexpr uint32_t GATHER_CHAINS = 22;
// Row stride: 16-byte rows for the replay's float4 reads; at 36 words a
// quarter warp's reads (and a warp's word stores) touch every bank once.
constexpr uint32_t GATHER_STRIDE = WARP + 4;
// Lane `chain` replays its accumulator chain over the `count` terms of one
// round, in order.  Every chain runs the same instructions: the compensated
// step (y = t + low, next = acc + y, low = y - (next - acc)), whose residual
// only the force and torque chains keep.  With low = +0 the step is the plain
// sum acc + t bit for bit (acc starts at +0 and is never -0, so a -0 term
// read as +0 changes nothing); the stress rows are stored negated (a - b is
// a + (-b)), and the maximum chain selects.  One loop for the warp, fed by
// float4 shared loads, instead of one per kind of chain: those four diverged
// and ran one after the other.  The gather went from 205 to 164 us for
// 15,625 grains with 2.0 M contacts, 129 to 113 us for 50,000 with 950 k.
__device__ __forceinline__ void replayChain(const float (*terms)[GATHER_STRIDE], uint32_t count, uint32_t chain,
                                            float& acc, float& accLow) {
    const float* row = terms[min(chain, GATHER_CHAINS - 1)];
    const bool compensated = chain < 6, maximum = chain == 17;
    auto step = [&](float t) {
        float y = __fadd_rn(t, accLow);
        float nx = __fadd_rn(acc, y);
        float low = __fsub_rn(y, __fsub_rn(nx, acc));
        accLow = compensated ? low : 0.0f;
        acc = maximum ? mx(acc, t) : nx;
    };
    uint32_t k = 0;
    for (; k + 4 <= count; k += 4) {
        float4 t = *reinterpret_cast<const float4*>(row + k);
        step(t.x);
        step(t.y);
        step(t.z);
        step(t.w);
    }
    for (; k < count; ++k) step(row[k]);
}
__device__ __forceinline__ void storeTerms(float (*terms)[GATHER_STRIDE], uint32_t lane, const GatherTerms& g) {
    const float v[GATHER_CHAINS] = {g.force.x, g.force.y, g.force.z, g.torque.x, g.torque.y, g.torque.z,
                                    -g.s0.x, -g.s0.y, -g.s0.z, -g.s1.x, -g.s1.y, -g.s1.z,
                                    -g.s2.x, -g.s2.y, -g.s2.z, g.energy, g.denom, g.depth,
                                    g.dissipation, g.normalPower, g.stiffness, g.viscous};
#pragma unroll
    for (uint32_t j = 0; j < GATHER_CHAINS; ++j) terms[j][lane] = v[j];
}
// solver.slang:773-791, the plane branch: full force, moment about the
// grain centre, virial with the arm, full energy and losses; the wall's own
// material in the timestep rates with coupling 1.
__device__ __forceinline__ GatherTerms wallTerms(const Res& r, const Config& c, uint32_t contact, uint32_t wall,
                                                 float mass, float bw, float inverseInertia) {
    GatherTerms g{};
    float4 cf = r.contactForce[contact], pdv = r.pointDepth[contact];
    f3 force = xyz(cf), arm = xyz(pdv);
    if (c.activeTimestep != 0) {
        float mobility = __fadd_rn(__fdiv_rn(1.0f, mass), __fmul_rn(dot(arm, arm), inverseInertia));
        float4 m = r.wallMaterial[wall];
        float area = __fmul_rn(1.0f, r.normalArea[contact].w);
        float friction = __fadd_rn(1.0f, m.z);
        g.stiffness = __fmul_rn(__fmul_rn(area, __fadd_rn(__fmul_rn(m.x, friction), m.y)), mobility);
        g.viscous = __fmul_rn(__fmul_rn(__fmul_rn(area, m.w), friction), mobility);
    }
    g.force = force;
    g.torque = cross(arm, force);
    g.s0 = force.x * arm;
    g.s1 = force.y * arm;
    g.s2 = force.z * arm;
    g.energy = cf.w;
    g.denom = length(force);
    g.depth = __fdiv_rn(pdv.w, bw);
    g.dissipation = r.slip[contact].w;
    g.normalPower = r.normalLossPower[contact];
    return g;
}
// A warp's scratch: B candidates, merged pairs, offsets and range ends of a
// window of pairs, and the terms of a round.
struct GatherScratch {
    uint32_t window[4][WARP];
    float terms[GATHER_CHAINS][GATHER_STRIDE];
};
// What follows a grain's sums: its diagnostic, loss and accumulator rows, and
// with `finish` (no plane, no timestep guard in between) the closing half kick.
__device__ __forceinline__ void gatherTail(const Res& r, const Config& c, uint32_t id, bool finish) {
    KickRows k = kickRows(r, id);
    float4 diagnostic = r.particleDiagnostic[id];
    f3 rate = xyz(r.cell[3 * specimenOf(r, id) + 1]);
    f3 v = xyz(k.v), w = omegaRows(k.inertia, k.q, xyz(k.l) + xyz(k.ll));
    float kinetic = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(k.mass, dot(v, v)), dot(xyz(k.l), w)));
    k.damping.z = diagnostic.x;
    compensated4(k.high, k.low, make_float4(k.torque.w, 0.f, 0.f, 0.f));
    r.particleDiagnostic[id] = make_float4(kinetic, diagnostic.y, length(xyz(k.force)), diagnostic.w);
    if (finish) {
        finishRows(r, c, id, k, rate);
    } else {
        r.normalDamping[id] = k.damping;
        r.accumulated[id] = k.high;
        r.accumulatedRemainder[id] = k.low;
    }
}
// With `tail` each warp also runs the tail of the grains it gathered, a lane
// a grain: one round of latency less than a kernel of its own, where the
// warps gather several grains each (the persistent step).
__device__ __forceinline__ void gather(const Params& P, GatherScratch& scratch, bool live, bool tail, bool finish) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (!live) return;
    uint32_t pairs = activePairs(r, c);
    uint32_t *wb = scratch.window[0], *wp = scratch.window[1], *wo = scratch.window[2], *we = scratch.window[3];
    float (*terms)[GATHER_STRIDE] = scratch.terms;
    const uint32_t chain = laneId();
    for (uint32_t p = gtid(); p < pairs; p += gstride())
        r.contactCounts[p] = r.sideContactStart[p + 1] - r.sideContactStart[p];
    for (uint32_t id = warpGlobal(); id < c.N; id += warpStride()) {
        // This lane's chain: running value and compensation residual.
        float acc = 0.f, accLow = 0.f;
        f3 one = mk(1.f, 1.f, 1.f);
        float inverseInertia = mx(mx(dot(abs3(xyz(r.invI[3 * id])), one), dot(abs3(xyz(r.invI[3 * id + 1])), one)),
                                  dot(abs3(xyz(r.invI[3 * id + 2])), one));
        float m_ = r.body[id].y, bw = r.body[id].w;
        // Plane contacts come first in the grain's list: they were appended
        // last (highest wall first, each run from its last contact).
        for (uint32_t w = c.wallCount; w-- > 0;) {
            uint32_t lo = r.sideWallStart[w * c.N + id], hi = r.sideWallStart[w * c.N + id + 1];
            while (hi > lo) {
                uint32_t count = min(hi - lo, WARP);
                if (laneId() < count) storeTerms(terms, laneId(), wallTerms(r, c, hi - 1 - laneId(), w, m_, bw, inverseInertia));
                __syncwarp();
                replayChain(terms, count, chain, acc, accLow);
                __syncwarp();
                hi -= count;
            }
        }
        uint32_t aBegin = min(r.pairOffsets[id], pairs), aEnd = min(aBegin + r.pairCounts[id], pairs);
        uint32_t bBegin = r.byJOffsets[id], bEnd = r.byJOffsets[id + 1];
        // The grain's pairs in descending pair id (the first-grain run
        // aBegin..aEnd-1 and the second-grain run byJPairs[bBegin..bEnd),
        // both ascending, merged from the top), taken 32 at a time: each
        // window is merged by ranks, its pairs' contact ranges are scanned,
        // and its contacts -- each pair's from the last -- are processed 32
        // per round in that flattened order, the reference's LIFO order.
        uint32_t ia = aEnd, ib = bEnd;
        while (ia > aBegin || ib > bBegin) {
            uint32_t na = min(ia - aBegin, WARP), nb = min(ib - bBegin, WARP), lane = laneId();
            uint32_t bv = lane < nb ? r.byJPairs[ib - 1 - lane] : 0u;  // descending
            wb[lane] = bv;
            __syncwarp();
            // Rank of each candidate among the union of both windows.
            uint32_t av = ia - 1 - lane;                                // descending, valid for lane < na
            uint32_t rankA = WARP, rankB = WARP;
            if (lane < na) {
                uint32_t lo = 0, hi = nb;                               // B candidates greater than av
                while (lo < hi) { uint32_t mid = (lo + hi) >> 1; if (wb[mid] > av) lo = mid + 1; else hi = mid; }
                rankA = lane + lo;
            }
            if (lane < nb) {
                uint32_t greater = bv >= ia - 1 ? 0u : min(na, ia - 1 - bv);  // A candidates greater than bv
                rankB = lane + greater;
            }
            uint32_t takeA = __popc(__ballot_sync(0xffffffffu, rankA < WARP));
            uint32_t takeB = __popc(__ballot_sync(0xffffffffu, rankB < WARP));
            __syncwarp();
            if (rankA < WARP) wp[rankA] = av;
            if (rankB < WARP) wp[rankB] = bv;
            __syncwarp();
            uint32_t m = takeA + takeB, cnt = 0, pairId = 0, last = 0;
            if (lane < m) {
                pairId = wp[lane];
                uint32_t begin = r.sideContactStart[pairId];
                last = r.sideContactStart[pairId + 1];
                cnt = last - begin;
            }
            uint32_t incl = cnt;
#pragma unroll
            for (uint32_t o = 1; o < WARP; o <<= 1) {
                uint32_t t2 = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t2;
            }
            uint32_t total = __shfl_sync(0xffffffffu, incl, WARP - 1);
            wo[lane] = incl - cnt;
            we[lane] = last;
            __syncwarp();
            for (uint32_t q0 = 0; q0 < total; q0 += WARP) {
                uint32_t count = min(total - q0, WARP);
                GatherTerms g{};
                if (lane < count) {
                    uint32_t q = q0 + lane, lo = 0, hi = m;             // last window slot with offset <= q
                    while (hi - lo > 1) { uint32_t mid = (lo + hi) >> 1; if (wo[mid] <= q) lo = mid; else hi = mid; }
                    uint32_t p = wp[lo];
                    uint32_t contact = we[lo] - 1 - (q - wo[lo]);
                    uint4 key = r.meta[contact];
                    bool source = key.x == id;
                    float4 cf = r.contactForce[contact];
                    f3 force = xyz(cf);
                    float4 pdv = r.pointDepth[contact];
                    f3 arm = xyz(pdv);
                    f3 branch = xyz(r.dpairBranch[2 * p + (key.x > key.y ? 1u : 0u)]);
                    if (c.activeTimestep != 0) {
                        f3 localArm = source ? arm : arm - branch;
                        float mobility = __fadd_rn(__fdiv_rn(1.0f, m_), __fmul_rn(dot(localArm, localArm), inverseInertia));
                        float half = __fmul_rn(r.normalArea[contact].w, 0.5f);
                        g.stiffness = __fmul_rn(__fmul_rn(__fmul_rn(2.0f, half), __fadd_rn(__fmul_rn(c.kn, __fadd_rn(1.0f, c.mu)), c.kt)), mobility);
                        g.viscous = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(2.0f, half), c.normalViscosity), __fadd_rn(1.0f, c.mu)), mobility);
                    }
                    g.force = source ? force : -force;
                    g.torque = source ? cross(arm, force) : cross(arm - branch, -force);
                    g.s0 = __fmul_rn(0.5f, force.x) * branch;
                    g.s1 = __fmul_rn(0.5f, force.y) * branch;
                    g.s2 = __fmul_rn(0.5f, force.z) * branch;
                    g.energy = __fmul_rn(0.5f, cf.w);
                    g.denom = length(force);
                    uint32_t other = source ? key.y : key.x;
                    float wmin = source ? mn(bw, r.body[other].w) : mn(r.body[other].w, bw);
                    g.depth = __fdiv_rn(pdv.w, wmin);
                    g.dissipation = __fmul_rn(0.5f, r.slip[contact].w);
                    g.normalPower = __fmul_rn(0.5f, r.normalLossPower[contact]);
                    storeTerms(terms, lane, g);
                }
                __syncwarp();
                replayChain(terms, count, chain, acc, accLow);
                __syncwarp();
            }
            __syncwarp();
            ia -= takeA;
            ib -= takeB;
        }
        // Collect the chains on lane 0.
        float sums[GATHER_CHAINS], lows[6];
#pragma unroll
        for (uint32_t j = 0; j < GATHER_CHAINS; ++j) sums[j] = __shfl_sync(0xffffffffu, acc, int(j));
#pragma unroll
        for (uint32_t j = 0; j < 6; ++j) lows[j] = __shfl_sync(0xffffffffu, accLow, int(j));
        if (laneId() == 0) {
            f3 f = mk(sums[0], sums[1], sums[2]) + mk(lows[0], lows[1], lows[2]);
            f3 t = mk(sums[3], sums[4], sums[5]) + mk(lows[3], lows[4], lows[5]);
            // energy, denominator, deepest overlap, dissipation, normal loss power, timestep rates: 15-21
            r.timestepRows[id] = make_float4(sums[20], sums[21], 0.f, 0.f);
            r.force[id] = w4(f, sums[17]);
            r.torque[id] = w4(t, sums[18]);
            r.particleStress[3 * id] = make_float4(sums[6], sums[7], sums[8], 0.f);
            r.particleStress[3 * id + 1] = make_float4(sums[9], sums[10], sums[11], 0.f);
            r.particleStress[3 * id + 2] = make_float4(sums[12], sums[13], sums[14], 0.f);
            r.particleDiagnostic[id] = make_float4(sums[19], sums[15], 0.f, sums[16]);
        }
    }
    if (!tail) return;
    // The rest of each grain's rows, a lane a grain of those the warp
    // gathered (one round of loads for all of them, not one a grain).
    __syncwarp();
    for (uint32_t id = warpGlobal() + laneId() * warpStride(); id < c.N; id += WARP * warpStride())
        gatherTail(r, c, id, finish);
}
// Two warps a CTA, twelve CTAs an SM (at most 80 registers): a CTA lasts as
// long as its slowest warp, and grains differ.  With eight warps a CTA and
// grains dealt over a fixed grid a quarter of the SMs' warps were resident on
// average (of three eighths).
constexpr uint32_t GATHER_WARPS = 2;

}  // namespace sdg

// Launches of the neighbour build, contact collection, contact law and gather
// (contacts_device.cuh).
#include "culler.cuh"
#include "contacts_device.cuh"

namespace sdg {

// ---------------------------------------------------------------- kernels
// A scan is skipped where *gate is zero, and where *failed (the solver flags) is
// not: on a failed step the phases before it return and leave stale input.
__device__ __forceinline__ bool scanSkipped(const uint32_t* gate, const uint32_t* failed) {
    return (gate && *gate == 0) || (failed && *failed != 0);
}
__global__ void k_scanReduce(const uint32_t* in, ScanCount count, const uint32_t* gate, const uint32_t* failed,
                             uint32_t* partials) {
    __shared__ uint32_t shared[32];
    if (scanSkipped(gate, failed)) return;
    uint32_t n = scanCount(count);
    uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
    uint32_t begin = blockIdx.x * chunk, end = min(n, begin + chunk);
    uint32_t sum = 0;
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) sum += in[i];
    sum = blockInclusive(sum, shared);
    if (threadIdx.x == blockDim.x - 1) partials[blockIdx.x] = sum;
}
__global__ void k_scanTop(ScanCount count, uint32_t* out, bool writeEnd, uint32_t* totalDst, const uint32_t* gate,
                          const uint32_t* failed, uint32_t* partials, uint32_t blocks) {
    __shared__ uint32_t shared[32];
    if (scanSkipped(gate, failed)) return;
    // blocks <= 1024: one element per thread.
    uint32_t v = threadIdx.x < blocks ? partials[threadIdx.x] : 0;
    uint32_t inc = blockInclusive(v, shared);
    if (threadIdx.x < blocks) partials[blocks + threadIdx.x] = inc - v;
    if (threadIdx.x == blockDim.x - 1) {
        uint32_t n = scanCount(count);
        if (writeEnd) out[n] = inc;
        if (totalDst) *totalDst = inc;
    }
}
// With `list`, the input holds flags (0 or 1): a set flag's index goes to its
// place, and a place at or past `room` is dropped whatever the input holds.
__global__ void k_scanApply(const uint32_t* in, uint32_t* out, ScanCount count, const uint32_t* gate,
                            const uint32_t* failed, const uint32_t* partials, uint32_t* list, uint32_t room) {
    __shared__ uint32_t shared[32];
    __shared__ uint32_t tileTotal;
    if (scanSkipped(gate, failed)) return;
    uint32_t n = scanCount(count);
    uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
    uint32_t begin = blockIdx.x * chunk, end = min(n, begin + chunk);
    uint32_t carry = partials[gridDim.x + blockIdx.x];
    for (uint32_t base = begin; base < end; base += blockDim.x) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < end ? in[i] : 0;
        uint32_t inc = blockInclusive(v, shared);
        if (i < end) {
            out[i] = carry + inc - v;
            if (list && v && carry + inc - v < room) list[carry + inc - v] = i;
        }
        if (threadIdx.x == blockDim.x - 1) tileTotal = inc;
        __syncthreads();
        carry += tileTotal;
        __syncthreads();
    }
}
__global__ void k_binsClear(const __grid_constant__ Params P) { binsClear(P); }
__global__ void k_binsFill(const __grid_constant__ Params P) { binsFill(P); }
// Order each bin's slots by grain id: the serial reference fills bins in id
// order, which fixes the pair order downstream.  Rank sort in shared memory.
__global__ void k_binsSort(const __grid_constant__ Params P) {
    extern __shared__ uint32_t ids[];
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[4] == 0) return;
    uint32_t cap = c.binCapacity;
    uint32_t* sorted = ids + cap;
    for (uint32_t bin = blockIdx.x; bin < c.binCount; bin += gridDim.x) {
        uint32_t occ = min(r.binCounts[bin], cap);
        for (uint32_t k = threadIdx.x; k < occ; k += blockDim.x) ids[k] = r.binParticles[bin * cap + k];
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < occ; k += blockDim.x) {
            uint32_t v = ids[k], rank = 0;
            for (uint32_t t = 0; t < occ; ++t) rank += ids[t] < v;
            sorted[rank] = v;
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < occ; k += blockDim.x) r.binParticles[bin * cap + k] = sorted[k];
        __syncthreads();
    }
}
// Keys: the same checks and bin as k_binsFill.
__global__ void k_binKeys(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t id = gtid();
    if (id >= c.N || r.control[4] == 0) return;
    RadixScratch x = radixScratch(r, c);
    uint32_t key = c.binCount;
    f3 p = xyz(r.position[id]), pl = xyz(r.positionRemainder[id]);
    uint32_t sp = specimenOf(r, id);
    float4 cell = r.cell[3 * sp];
    bool ok = finite3(p) && finite3(pl);
    if (!ok) fail(r, F_NONFINITE);
    if (ok && c.periodic == 0) {
        f3 box = xyz(cell);
        if (__fadd_rn(p.x, pl.x) < 0 || __fadd_rn(p.y, pl.y) < 0 || __fadd_rn(p.z, pl.z) < 0 ||
            __fadd_rn(__fsub_rn(p.x, box.x), pl.x) >= 0 || __fadd_rn(__fsub_rn(p.y, box.y), pl.y) >= 0 ||
            __fadd_rn(__fsub_rn(p.z, box.z), pl.z) >= 0) {
            fail(r, F_ESCAPE);
            ok = false;
        }
    }
    if (ok) {
        uint32_t b[3];
        uint4 sb = r.specimenBins[sp];
        binIndex(r, id, sb, cell, b);
        key = binFlat(sb, b);
    }
    x.keys[0][id] = key;
    x.vals[0][id] = id;
}
// Digit counts of each tile: counts[digit * tiles + tile].
__global__ void __launch_bounds__(256) k_radixCount(const __grid_constant__ Params P, uint32_t shift, uint32_t from) {
    __shared__ uint32_t hist[RADIX];
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[4] == 0) return;
    RadixScratch x = radixScratch(r, c);
    hist[threadIdx.x] = 0;
    __syncthreads();
    uint32_t base = blockIdx.x * RADIX_TILE;
    for (uint32_t k = threadIdx.x; k < RADIX_TILE && base + k < c.N; k += blockDim.x)
        atomicAdd(&hist[(x.keys[from][base + k] >> shift) & (RADIX - 1)], 1u);
    __syncthreads();
    x.counts[threadIdx.x * x.tiles + blockIdx.x] = hist[threadIdx.x];
}
// Stable scatter of a tile: its elements in index order, 256 at a time; an
// element's place is its digit's offset for the tile (the scanned counts),
// plus the tile's earlier elements with that digit (a running count), plus
// the earlier warps of the same 256 with it, plus the lower lanes of its
// warp with it (__match_any_sync).
__global__ void __launch_bounds__(256) k_radixScatter(const __grid_constant__ Params P, uint32_t shift, uint32_t from) {
    __shared__ uint32_t offset[RADIX], warpCount[8][RADIX];
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[4] == 0) return;
    RadixScratch x = radixScratch(r, c);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    offset[threadIdx.x] = x.counts[threadIdx.x * x.tiles + blockIdx.x];
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w) warpCount[w][threadIdx.x] = 0;
    __syncthreads();
    uint32_t base = blockIdx.x * RADIX_TILE;
    for (uint32_t round = 0; round < RADIX_ITEMS; ++round) {
        uint32_t i = base + round * 256 + threadIdx.x;
        bool valid = i < c.N && round * 256 + threadIdx.x < RADIX_TILE;
        uint32_t key = valid ? x.keys[from][i] : 0u, val = valid ? x.vals[from][i] : 0u;
        uint32_t digit = valid ? (key >> shift) & (RADIX - 1) : RADIX;  // RADIX: no element
        uint32_t peers = __match_any_sync(0xffffffffu, digit);
        uint32_t below = __popc(peers & lanesBelow());
        if (valid && below == 0) warpCount[warp][digit] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t place = offset[digit] + below;
            for (uint32_t w = 0; w < warp; ++w) place += warpCount[w][digit];
            x.keys[from ^ 1u][place] = key;
            x.vals[from ^ 1u][place] = val;
        }
        __syncthreads();
        // These 256 elements of each digit move its offset on.
        uint32_t total = 0;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
            total += warpCount[w][threadIdx.x];
            warpCount[w][threadIdx.x] = 0;
        }
        offset[threadIdx.x] += total;
        __syncthreads();
    }
}
// Each bin's run of the sorted grains into its reference slots.
__global__ void k_binsFromSorted(const __grid_constant__ Params P, uint32_t from) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[4] == 0) return;
    RadixScratch x = radixScratch(r, c);
    for (uint32_t k = gtid(); k < c.N; k += gstride()) {
        uint32_t bin = x.keys[from][k];
        if (bin >= c.binCount || (k > 0 && x.keys[from][k - 1] == bin)) continue;  // not the start of a run
        uint32_t occ = 0;
        while (k + occ < c.N && x.keys[from][k + occ] == bin) {
            if (occ < c.binCapacity) r.binParticles[bin * c.binCapacity + occ] = x.vals[from][k + occ];
            ++occ;
        }
        r.binCounts[bin] = occ;
        if (occ > c.binCapacity) fail(r, F_BIN);
    }
}
__global__ void __launch_bounds__(256) k_pairsCountWarp(const __grid_constant__ Params P) { pairsCountWarp(P); }
__global__ void __launch_bounds__(256) k_pairsEmitWarp(const __grid_constant__ Params P) { pairsEmitWarp(P); }
__global__ void k_byJReset(const __grid_constant__ Params P) { byJReset(P); }
__global__ void k_byJCount(const __grid_constant__ Params P) { byJCount(P); }
__global__ void k_byJFill(const __grid_constant__ Params P) { byJFill(P); }
__global__ void k_byJSort(const __grid_constant__ Params P) { byJSort(P); }
__global__ void k_pairSetup(const __grid_constant__ Params P) { pairSetup(P); }
__global__ void k_resetContacts(const __grid_constant__ Params P) {
    if (P.r.control[0] == 0) resetContacts(P.r, P.c, true);
}
// The same before a step's neighbour build: the pairs, and their set-up, are
// known only where the step keeps them ...
__global__ void k_resetContactsKept(const __grid_constant__ Params P) {
    if (P.r.control[0] == 0) resetContacts(P.r, P.c, P.r.control[4] == 0);
}
__global__ void k_pairSetupKept(const __grid_constant__ Params P) {
    if (P.r.control[4] == 0) pairSetup(P);
}
// ... else after the build.
__global__ void k_pairSetupRebuilt(const __grid_constant__ Params P) {
    const Res& r = P.r;
    if (r.control[4] == 0) return;
    if (gtid() == 0 && r.work[W_FILTER_PAIRS] != r.control[1]) atomicOr(&r.work[W_FILTER], 1u);
    pairSetup(P);
}
__global__ void k_leafCull(const __grid_constant__ Params P) { leafCull(P, P.r.control[0] == 0); }
__global__ void k_leafEmit(const __grid_constant__ Params P) { leafEmit(P); }
__global__ void __launch_bounds__(256) k_nodeFilter(const __grid_constant__ Params P) { nodeFilter(P); }
__global__ void __launch_bounds__(256) k_survivorPrefilter(const __grid_constant__ Params P) { survivorPrefilter(P); }
// Distance-bound grid of every shape (built once per library): one thread per
// cell evaluates the exact signed distance at the cell centre (meshDistance,
// the query the contacts use) and stores phi - (half diagonal) x 1.001 -
// 1e-5 (1 + |centre|_1).  The grid spans the shape's root box with cubic
// cells of edge (largest box extent) / GRID.
__global__ void k_distanceGrid(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    const uint32_t cells = GRID * GRID * GRID;
    for (uint32_t t = gtid(); t < c.shapes * cells; t += gstride()) {
        uint32_t shape = t / cells, cell = t % cells;
        uint32_t root = __ldg(&r.meshRoots[shape].x);
        f3 low = xyz(__ldg(&r.meshMin[root])), high = xyz(__ldg(&r.meshMax[root]));
        f3 extent = high - low;
        float h = __fdiv_rn(mx(mx(extent.x, extent.y), extent.z), float(GRID));
        if (cell == 0) r.distanceGridInfo[shape] = w4(low, h);
        uint32_t gx = cell % GRID, gy = (cell / GRID) % GRID, gz = cell / (GRID * GRID);
        f3 centre = low + mk(__fmul_rn(float(gx) + 0.5f, h), __fmul_rn(float(gy) + 0.5f, h),
                             __fmul_rn(float(gz) + 0.5f, h));
        uint32_t nearest;
        float phi = meshDistance(r, shape, centre, false, 0xFFFFFFFFu, &nearest).w;
        r.distanceGridTriangle[t] = nearest;
        float reach = __fmul_rn(__fmul_rn(0.8660254f, h), 1.001f);
        float slack = __fmul_rn(1e-5f, __fadd_rn(1.0f, __fadd_rn(__fadd_rn(fabsf(centre.x), fabsf(centre.y)),
                                                                 fabsf(centre.z))));
        r.distanceGrid[t] = __fsub_rn(__fsub_rn(phi, reach), slack);
    }
}
// The BVH leaf of each packed triangle (cellQuery breaks ties by it).
__global__ void k_triangleLeaf(const __grid_constant__ Params P) {
    const Res& r = P.r;
    for (uint32_t shape = blockIdx.x; shape < P.c.shapes; shape += gridDim.x) {
        uint4 nodes = __ldg(&r.meshRoots[shape]);
        for (uint32_t node = nodes.x + threadIdx.x; node < nodes.y; node += blockDim.x) {
            float4 head = __ldg(&r.meshChildren[4 * size_t(node)]);
            if (__float_as_uint(head.w) != LEAF_MARK) continue;
            uint32_t first = __float_as_uint(head.x), count = __float_as_uint(head.y);
            for (uint32_t k = 0; k < count; ++k) r.triangleLeaf[first + k] = node;
        }
    }
}
// The triangle lists of the grid cells (dem_device.cuh), once per library: a warp
// per block of 2 x 4 x 4 cells, a lane a cell, walks the BVH once for all of
// them -- a child is visited where any lane needs it -- for the triangles
// within CELL_REACH h of each cell's nearest one's distance (k_distanceGrid's),
// keeping the CELL_TRIANGLES nearest in order; a list that overflows lowers
// its limit to the nearest triangle left out.  A walk a lane ran with 6 lanes
// of 32 active: 11 ms for 64 shapes of 320 triangles and 55 ms for 64 of 320 to
// 5,120, now 4.5 and 11.7.  Cells that no exact query reaches hold an empty list: a stored
// node lies within 1.001 margins (16 at most) of its target at the build, by its
// cell's bound, and moves by less than as much again, which with the cells'
// extent is what the line below allows.  (A query there would walk: with the
// distance grid off no bound holds the stored nodes near, and every cell is listed.)
__global__ void __launch_bounds__(256) k_cellLists(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    constexpr uint32_t cells = GRID * GRID * GRID, blocks = cells / WARP;
    static_assert(GRID % 4 == 0);
    for (uint32_t w = warpGlobal(); w < c.shapes * blocks; w += warpStride()) {
        const uint32_t shape = w / blocks, block = w % blocks, lane = laneId();
        float4 info = r.distanceGridInfo[shape];
        const uint32_t gx = 2 * (block % (GRID / 2)) + (lane & 1u);
        const uint32_t gy = 4 * ((block / (GRID / 2)) % (GRID / 4)) + ((lane >> 1) & 3u);
        const uint32_t gz = 4 * (block / (GRID / 2 * (GRID / 4))) + (lane >> 3);
        const uint32_t i = shape * cells + (gz * GRID + gy) * GRID + gx;
        f3 p = xyz(info) + mk(__fmul_rn(float(gx) + 0.5f, info.w), __fmul_rn(float(gy) + 0.5f, info.w),
                              __fmul_rn(float(gz) + 0.5f, info.w));
        uint32_t* out = r.cellLists + size_t(i) * CELL_WORDS;
        const uint32_t seed = r.distanceGridTriangle[i];
        const float reached = __fadd_rn(__fmul_rn(33.0f, c.filterMargin), __fmul_rn(2.0f, info.w));
        const bool listed = seed != EMPTY && (!c.distanceGridEnabled || r.distanceGrid[i] <= reached);
        auto squared = [&](uint32_t t) {
            uint32_t feature;
            f3 q = closestTriangle(p, xyz(__ldg(&r.meshTriangles[3 * t])), xyz(__ldg(&r.meshTriangles[3 * t + 1])),
                                   xyz(__ldg(&r.meshTriangles[3 * t + 2])), feature);
            f3 dq = p - q;
            return dot(dq, dq);
        };
        float d1 = listed ? __fsqrt_rn(squared(seed)) : 0.0f;
        // Below any distance where the cell has no list.
        const float limitRoot = __fadd_rn(d1, __fmul_rn(CELL_REACH, info.w));
        float limit = listed ? __fmul_rn(limitRoot, limitRoot) : -1.0f;
        uint32_t ids[CELL_TRIANGLES], count = 0;
        float far[CELL_TRIANGLES];
        uint32_t pending[32], top = __any_sync(0xffffffffu, listed) ? 1 : 0;
        pending[0] = __ldg(&r.meshRoots[shape].x);
        while (top > 0) {
            uint32_t node = pending[--top];
            const float4* record = r.meshChildren + 4 * size_t(node);
            float4 r0 = __ldg(record), r1 = __ldg(record + 1);
            if (__float_as_uint(r0.w) != LEAF_MARK) {
                float4 r2 = __ldg(record + 2), r3 = __ldg(record + 3);
                uint32_t a = node + 1, b = __float_as_uint(r0.w);
                float da = boxDistance(xyz(r0), xyz(r1), p), db = boxDistance(xyz(r2), xyz(r3), p);
                const float reach = __fmul_rn(limit, 1.00000095367431640625f);
                bool needA = __any_sync(0xffffffffu, da <= reach), needB = __any_sync(0xffffffffu, db <= reach);
                // The child nearer to most lanes first.
                if (__popc(__ballot_sync(0xffffffffu, da < db)) > 16) {
                    uint32_t t = a; a = b; b = t;
                    bool n = needA; needA = needB; needB = n;
                }
                if (top + 2 > 32) { if (lane == 0) fail(r, F_STACK); break; }
                if (needA) pending[top++] = a;
                if (needB) pending[top++] = b;
                continue;
            }
            uint32_t first = __float_as_uint(r0.x), leaf = __float_as_uint(r0.y);
            for (uint32_t t = first; t < first + leaf; ++t) {
                float d = squared(t);
                if (d >= limit) continue;
                if (count == CELL_TRIANGLES) {
                    // Full: the farthest of them all sets the limit.
                    if (d >= far[CELL_TRIANGLES - 1]) { limit = fminf(limit, d); continue; }
                    limit = fminf(limit, far[CELL_TRIANGLES - 1]);
                    --count;
                }
                uint32_t k = count++;
                for (; k > 0 && far[k - 1] > d; --k) { far[k] = far[k - 1]; ids[k] = ids[k - 1]; }
                far[k] = d;
                ids[k] = t;
            }
        }
        if (!listed) {
            for (uint32_t k = 0; k < CELL_WORDS; ++k) out[k] = k >= 2 && k < CELL_STEPS ? EMPTY : 0u;
            continue;
        }
        float step = cellStep(info.w);
        d1 = count ? __fsqrt_rn(far[0]) : d1;
        out[0] = __float_as_uint(__fmul_rn(__fsqrt_rn(limit), 0.999999f));
        out[1] = __float_as_uint(d1);
        uint32_t packed = 0;
        for (uint32_t k = 0; k < CELL_TRIANGLES; ++k) {
            out[2 + k] = k < count ? ids[k] : EMPTY;
            float beyond = k < count ? __fmul_rn(__fdiv_rn(__fsub_rn(__fsqrt_rn(far[k]), d1), step), 0.99999f) : 0.0f;
            packed |= uint32_t(fminf(fmaxf(beyond, 0.0f), 255.0f)) << (8 * (k & 3u));
            if ((k & 3u) == 3u) {
                out[CELL_STEPS + (k >> 2)] = packed;
                packed = 0;
            }
        }
    }
}
// Per-shape counts of the kept survivors (walkBucketCount[shape]; zero on
// entry: the placement below takes each back to zero).
__global__ void k_cullCount(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t n = min(r.work[W_SURVIVORS], c.survivorCapacity);
    for (uint32_t s = gtid(); s < n; s += gstride()) {
        uint32_t shape = r.survKeep[s] ? survivorTargetShape(r, c, s) : EMPTY;
        uint32_t same = __match_any_sync(__activemask(), shape);
        if (shape != EMPTY && laneId() == uint32_t(__ffs(same) - 1)) atomicAdd(&r.walkBucketCount[shape], __popc(same));
    }
}
// Placement in shape order (walkKey); each count returns to zero.
__global__ void k_cullPlace(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t n = min(r.work[W_SURVIVORS], c.survivorCapacity);
    for (uint32_t s = gtid(); s < n; s += gstride()) {
        uint32_t shape = r.survKeep[s] ? survivorTargetShape(r, c, s) : EMPTY;
        uint32_t same = __match_any_sync(__activemask(), shape);
        uint32_t leader = __ffs(same) - 1, base = 0;
        if (shape != EMPTY && laneId() == leader) base = atomicSub(&r.walkBucketCount[shape], __popc(same));
        base = __shfl_sync(same, base, leader);
        if (shape != EMPTY) {
            uint32_t rank = __popc(same & lanesBelow());
            r.walkKey[r.walkBucketOffset[shape] + base - 1 - rank] = s;
        }
    }
}
__global__ void __launch_bounds__(CULLER_ROWS) k_cullSurvivors(const __grid_constant__ Params P) {
    __shared__ CullerShared sh;
    __shared__ uint32_t live, tested, culled;
    const Res& r = P.r;
    const Config& c = P.c;
    if (threadIdx.x == 0) {
        live = r.control[0] == 0;
        tested = culled = 0;
    }
    cullerBegin(sh);  // synchronizes
    uint32_t phase = 0;
    uint32_t n = live ? min(r.work[W_CULL_ROWS], c.survivorCapacity) : 0u;
    uint32_t tiles = (n + CULLER_ROWS - 1) / CULLER_ROWS;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint32_t i = t * CULLER_ROWS + threadIdx.x, s = EMPTY, shape = EMPTY;
        f3 local = mk(0.f, 0.f, 0.f);
        float margin = 0.0f;
        if (i < n) {
            s = r.walkKey[i];
            SurvivorNode v = survivorNode(r, s);
            local = v.local;
            shape = r.shapeId[v.dst];
            uint32_t root = __ldg(&r.meshRoots[shape].x);
            margin = r.cullerMargin[size_t(shape) * CULLER_MARGINS + 1 +
                                    cullerCell(__ldg(&r.meshMin[root]), __ldg(&r.meshMax[root]), local)];
        }
        float y;
        if (!cullerTile(sh, r.cullerParams, r.cullerW1, shape, local, phase, y)) {
            if (threadIdx.x == 0) fail(r, F_WAIT);
            break;
        }
        if (shape != EMPTY) {
            atomicAdd(&tested, 1u);
            if (y > margin) {
                r.survKeep[s] = 0u;
                atomicAdd(&culled, 1u);
            }
        }
    }
    cullerEnd(sh, phase);  // synchronizes
    if (threadIdx.x == 0 && tested) {
        atomicAdd(&r.cullerStats[0], tested);
        atomicAdd(&r.cullerStats[1], culled);
    }
}
__global__ void k_walkList(const __grid_constant__ Params P) { walkList(P); }
__global__ void k_survivorList(const __grid_constant__ Params P) { survivorList(P); }
// Exact queries of a list built every step (margin 0 or the learned culler):
// one seeded walk per node.
__global__ void __launch_bounds__(256) k_nodeWalk(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0) return;
    uint32_t n = min(r.work[W_KEPT], c.survivorCapacity);
    for (uint32_t t = gtid(); t < n; t += gstride()) {
        uint32_t s = r.walkList[t];
        SurvivorNode v = survivorNode(r, s);
        float4 pd, na;
        uint32_t shape = r.shapeId[v.dst];
        // Seed the walk with the triangle nearest to the node's grid cell.
        float4 f = meshDistance(r, shape, v.local, false, gridSeed(r, shape, v.local));
        if (nodeContactFrom(r, c, v.src, v.dst, v.node, v.arm, f, pd, na)) recordHit(r, s, v, pd, na);
    }
}
__global__ void __launch_bounds__(256, 4) k_nodeQuery(const __grid_constant__ Params P) { nodeQuery(P, P.r.control[0] == 0); }
// Four CTAs an SM (64 registers instead of 79, three): the lanes' lists differ in
// length, so the warps stall more than the spilled words cost.  With no CTA
// barrier in its loop either, a list build of 1.5 M slots takes 40 us less.
__global__ void __launch_bounds__(256, 4) k_certifyBuild(const __grid_constant__ Params P) { certifyBuild(P, P.r.control[0] == 0); }
__global__ void __launch_bounds__(256) k_nodeCertify(const __grid_constant__ Params P) { nodeCertify(P, P.r.control[0] == 0); }
__global__ void __launch_bounds__(256) k_nodeWalkSlow(const __grid_constant__ Params P) { nodeWalkSlow(P, P.r.control[0] == 0); }
// L2 prefetch, first in a step, of what the step's exact queries read
// through chains of dependent loads: the packed library (BVH node records,
// triangles, pseudonormals, node samples) and, with a stored exact-query
// list, its per-slot certificates and node records.  One bulk copy-engine
// prefetch (cp.async.bulk.prefetch.L2) per 16 KB, from two CTAs per SM: the
// lines arrive while the drift, neighbour and pair kernels run, instead of
// one latency at a time inside the walks (64 KB pieces from four CTAs took
// longer than the walks saved).  A hint only: nothing waits for it and no result
// depends on it.  Every range starts 16-byte aligned (float4/uint4/uint2
// arrays from the allocator) and is cut to a multiple of 16 bytes.
__global__ void k_prefetch(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    constexpr uint32_t CHUNK = 16u << 10;
    uint32_t kept = storedKeep(c) ? min(r.work[W_KEPT], c.survivorCapacity) : 0u;
    const void* base[8] = {r.meshTriangles, r.meshNormals, r.sample, r.walkActive, r.walkState,
                           r.walkCert, r.walkNode, r.walkContact};
    uint64_t size[8] = {16ull * c.library16[1], 16ull * c.library16[2], 16ull * c.library16[3], 4ull * kept,
                        4ull * kept, 16ull * CERT_ROWS * kept, 16ull * kept, 4ull * kept};
    uint32_t chunk = gtid();
    for (int k = 0; k < 8; ++k) {
        uint64_t bytes = size[k] & ~uint64_t(15);
        uint64_t chunks = (bytes + CHUNK - 1) / CHUNK;
        for (; chunk < chunks; chunk += gstride()) {
            uint64_t offset = uint64_t(chunk) * CHUNK;
            uint64_t left = bytes - offset;
            uint32_t n = left < CHUNK ? uint32_t(left) : CHUNK;
            const char* at = static_cast<const char*>(base[k]) + offset;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(n) : "memory");
        }
        chunk -= uint32_t(chunks);
    }
}
// Copies the hits of each item from their survivor slots to their canonical
// offsets, and clears the item's hit mask and count for the next step (also
// on a failed step, whose walks may have set bits before the failure: the
// masks are all zero whenever a step starts, so a step that reuses the
// stored survivors needs no clearing pass).
__global__ void __launch_bounds__(256) k_nodeEmit(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    bool live = r.control[0] == 0;
    uint32_t n = min(r.work[W_CANDIDATES], c.candidateCapacity);
    // Lane per item: read and clear the masks of 32 items, then the warp
    // emits the items with hits one after the other.
    for (uint32_t first = WARP * warpGlobal(); first < n; first += WARP * warpStride()) {
        uint32_t mine = first + laneId();
        uint2 own = mine < n ? r.candHitMask[mine] : make_uint2(0u, 0u);
        bool any = (own.x | own.y) != 0;
        if (any) {
            r.candHitMask[mine] = make_uint2(0u, 0u);
            r.candHitCount[mine] = 0;
        }
        uint32_t pending = __ballot_sync(0xffffffffu, any);
        if (!live) continue;
        while (pending) {
            uint32_t lane = __ffs(pending) - 1;
            pending &= pending - 1;
            uint32_t item = first + lane;
            uint2 m = make_uint2(__shfl_sync(0xffffffffu, own.x, lane), __shfl_sync(0xffffffffu, own.y, lane));
            emitItem(r, c, item, m);
        }
    }
}
// Per pair: first contact of the pair on the side being written, and counts.
__global__ void k_contactStart(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t n = activePairs(r, c);
    uint32_t total = r.control[2];
    if (total > c.contactCapacity) fail(r, F_CONTACT);
    if (r.control[0] != 0) return;
    uint32_t items = min(r.work[W_CANDIDATES], c.candidateCapacity);
    for (uint32_t p = gtid(); p <= n; p += gstride()) {
        uint32_t first = r.dpairCandOffset[2 * p];
        uint32_t start = first < items ? r.candHitOffset[first] : total;
        r.sideContactStart[p] = start;
        if (p < n) {
            uint32_t next = r.dpairCandOffset[2 * p + 2];
            uint32_t end = next < items ? r.candHitOffset[next] : total;
            r.contactCounts[p] = end - start;
        }
    }
}
__global__ void __launch_bounds__(256) k_sdfQuery(const __grid_constant__ Params P) {
    __shared__ uint32_t list[8][SDF_LIST], counts[8][2 * WARP];
    sdfQueryPairs(P, list[threadIdx.x >> 5], counts[threadIdx.x >> 5], P.r.control[0] == 0);
}
__global__ void k_wallCount(const __grid_constant__ Params P) { wallCount(P, P.r.control[0] == 0); }
__global__ void k_wallEmit(const __grid_constant__ Params P) { wallEmit(P, P.r.control[0] == 0); }
__global__ void k_gatherWallRows(const __grid_constant__ Params P) { gatherWallRows(P); }
__global__ void k_resolveWalls(const __grid_constant__ Params P) { resolveWalls(P); }
__global__ void k_resolve(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (r.control[0] != 0) return;
    uint32_t n = activeContacts(r, c);
    // With planes, the grain-grain contacts end where the plane contacts
    // begin; those are resolved by k_resolveWalls.
    if (c.wallCount != 0) n = min(n, r.work[W_WALL_BASE]);
    for (uint32_t id = gtid(); id < n; id += gstride()) {
        uint4 key = r.meta[id];
        uint32_t old = c.historyStep != 0 ? historySlot(r, c, key.x, key.y, key.z) : EMPTY;
        f3 branch = xyz(r.dpairBranch[2 * r.contactPair[id] + (key.x > key.y ? 1 : 0)]);
        if (resolveGrain(r, c, id, key.x, key.y, r.normalArea[id], r.pointDepth[id], branch, old))
            atomicAdd(&r.control[6], 1u);
    }
}
template <bool Law>
__global__ void __launch_bounds__(256) k_emitSlots(const __grid_constant__ Params P) { emitSlots<Law>(P, P.r.control[0] == 0); }
template <bool Law>
__global__ void __launch_bounds__(256) k_sdfEmit(const __grid_constant__ Params P) { sdfEmit<Law>(P); }
__global__ void __launch_bounds__(32 * GATHER_WARPS, 12) k_gather(const __grid_constant__ Params P) {
    __shared__ __align__(16) GatherScratch scratch[GATHER_WARPS];
    gather(P, scratch[threadIdx.x >> 5], P.r.control[0] == 0, false, false);
}
__global__ void __launch_bounds__(128) k_gatherTail(const __grid_constant__ Params P, bool finish) {
    const uint32_t id = gtid();
    if (id < P.c.N && P.r.control[0] == 0) gatherTail(P.r, P.c, id, finish);
}

void launch_scan(const uint32_t* in, uint32_t* out, ScanCount count, bool writeEnd, uint32_t* totalDst,
                 const uint32_t* gate, uint32_t* partials, cudaStream_t s) {
    k_scanReduce<<<SCAN_BLOCKS, 256, 0, s>>>(in, count, gate, nullptr, partials);
    k_scanTop<<<1, 1024, 0, s>>>(count, out, writeEnd, totalDst, gate, nullptr, partials, SCAN_BLOCKS);
    k_scanApply<<<SCAN_BLOCKS, 256, 0, s>>>(in, out, count, gate, nullptr, partials, nullptr, 0);
}

// The step's scans (r.scanPartials).
void launch_step_scan(const Res& r, const uint32_t* in, uint32_t* out, ScanCount count, bool writeEnd,
                      uint32_t* totalDst, const uint32_t* gate, cudaStream_t s) {
    launch_scan(in, out, count, writeEnd, totalDst, gate, r.scanPartials, s);
}
// The scan of the keep flags (survKeep, to keepOffset and *totalDst), skipped on
// a failed step; with `list`, the apply pass also lists each index whose flag is
// set at its scanned offset (stream compaction in index order).
void launch_keep_scan(const Params& P, const uint32_t* count, uint32_t* totalDst, const uint32_t* gate,
                      uint32_t* list, cudaStream_t s) {
    const Res& r = P.r;
    const ScanCount n{count, P.c.survivorCapacity, 1, 0};
    k_scanReduce<<<SCAN_BLOCKS, 256, 0, s>>>(r.survKeep, n, gate, r.control, r.scanPartials);
    k_scanTop<<<1, 1024, 0, s>>>(n, r.keepOffset, true, totalDst, gate, r.control, r.scanPartials, SCAN_BLOCKS);
    k_scanApply<<<SCAN_BLOCKS, 256, 0, s>>>(r.survKeep, r.keepOffset, n, gate, r.control, r.scanPartials, list,
                                            P.c.survivorCapacity);
}

// ---------------------------------------------------------------- launchers
static inline uint32_t blocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }
constexpr uint32_t PERSISTENT = 152 * 8;  // warps-per-item kernels: 8 CTAs of 256 per SM

// SMs of the current device (152 on GB300), read once.
static uint32_t smCount() {
    static uint32_t sms = 0;
    if (!sms) {
        int device = 0, count = 0;
        if (cudaGetDevice(&device) == cudaSuccess &&
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && count > 0)
            sms = uint32_t(count);
        else
            sms = 152;
    }
    return sms;
}
// Grid of `perSM` CTAs per SM (the tuned value, or `fallback` when 0).
static inline uint32_t grid(uint32_t perSM, uint32_t fallback) { return smCount() * (perSM ? perSM : fallback); }

// The neighbour build on rebuild steps (every kernel returns at once on the
// others): the cell list by radix sort (or, where byJPairs is too small to
// hold the sort's scratch, by atomic fill and a rank sort per bin), the pair
// search with a warp per grain, then the pairs grouped by second grain.
static void neighbours(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t T = 256;
    k_binsClear<<<blocks(c.binCount, T), T, 0, s>>>(P);
    if (uint64_t(c.pairCapacity) >= radixWords(c.N)) {
        uint32_t tiles = radixTiles(c.N), from = 0, bits = 1;
        while (bits < 32 && (uint64_t(1) << bits) <= c.binCount) ++bits;  // keys 0 .. binCount
        k_binKeys<<<blocks(c.N, T), T, 0, s>>>(P);
        RadixScratch x = radixScratch(r, c);
        for (uint32_t shift = 0; shift < bits; shift += 8, from ^= 1u) {
            k_radixCount<<<tiles, T, 0, s>>>(P, shift, from);
            launch_step_scan(r, x.counts, x.counts, ScanCount{nullptr, 0, 0, RADIX * tiles}, false, nullptr,
                             r.control + 4, s);
            k_radixScatter<<<tiles, T, 0, s>>>(P, shift, from);
        }
        k_binsFromSorted<<<blocks(c.N, T), T, 0, s>>>(P, from);
    } else {
        k_binsFill<<<blocks(c.N, T), T, 0, s>>>(P);
        k_binsSort<<<min(c.binCount, 152u * 16u), 128, 2 * c.binCapacity * sizeof(uint32_t), s>>>(P);
    }
    k_pairsCountWarp<<<PERSISTENT, T, 0, s>>>(P);
    launch_step_scan(r, r.pairCounts, r.pairOffsets, ScanCount{nullptr, 0, 0, c.N}, false, r.control + 1, r.control + 4,
                s);
    k_pairsEmitWarp<<<PERSISTENT, T, 0, s>>>(P);
    k_byJReset<<<blocks(c.N + 1, T), T, 0, s>>>(P);
    k_byJCount<<<PERSISTENT, T, 0, s>>>(P);
    launch_step_scan(r, r.byJCounts, r.byJOffsets, ScanCount{nullptr, 0, 0, c.N}, true, nullptr, r.control + 4,
                s);
    k_byJFill<<<PERSISTENT, T, 0, s>>>(P);
    k_byJSort<<<blocks(c.N, T), T, 0, s>>>(P);
}

// Pair set-up (branches, the stored-filter motion check); with the SDF
// geometry also the contact counts and their scan.
static void collectHead(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t T = 256;
    k_resetContacts<<<1, 1, 0, s>>>(P);
    k_pairSetup<<<grid(c.cullBlocksPerSM, 8), T, 0, s>>>(P);
    if (c.meshGeometry == 0) {
        k_sdfQuery<<<grid(c.queryBlocksPerSM, 8), T, 0, s>>>(P);
        launch_step_scan(r, r.contactCounts, r.contactOffsets, ScanCount{r.control + 1, c.pairCapacity, 1, 0}, false,
                    r.control + 2, nullptr, s);
    }
}
// Root masks, leaf cull and the (directed pair, leaf) item list: steps that
// build the filter results (every kernel returns at once on the others).
static void cullBuild(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (c.meshGeometry == 0) return;
    uint32_t T = 256, g = grid(c.cullBlocksPerSM, 8);
    k_leafCull<<<g, T, 0, s>>>(P);
    launch_step_scan(r, r.dpairLeafCount, r.dpairCandOffset, ScanCount{r.control + 1, c.pairCapacity, 2, 0}, true,
                r.work + W_CANDIDATES, r.work + W_FILTER, s);
    k_leafEmit<<<g, T, 0, s>>>(P);
}
// Pair set-up, leaf cull and the (directed pair, leaf) item list; with the
// SDF geometry, pair set-up, contact counts and their scan.
static void collectCull(const Params& P, cudaStream_t s) {
    collectHead(P, s);
    cullBuild(P, s);
}
// Node filter, survivor list and (with the learned culler) the kept list.
static void collectFilter(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (c.meshGeometry == 0) return;
    uint32_t warps = c.queryWarps == 4 ? 4 : 8;
    k_nodeFilter<<<grid(c.queryBlocksPerSM, 8), 32 * warps, 0, s>>>(P);
    launch_step_scan(r, r.candSurvCount, r.candSurvOffset, ScanCount{r.work + W_CANDIDATES, c.candidateCapacity, 1, 0},
                true, r.work + W_SURVIVORS, r.work + W_FILTER, s);
    k_survivorList<<<grid(c.contactBlocksPerSM, 8), 256, 0, s>>>(P);
    k_survivorPrefilter<<<grid(c.walkBlocksPerSM, 8), 256, 0, s>>>(P);
    if (c.cullerEnabled) {
        uint32_t g = grid(c.contactBlocksPerSM, 8);
        k_cullCount<<<g, 256, 0, s>>>(P);
        launch_step_scan(r, r.walkBucketCount, r.walkBucketOffset, ScanCount{nullptr, 0, 0, c.shapes}, true,
                         r.work + W_CULL_ROWS, nullptr, s);
        k_cullPlace<<<g, 256, 0, s>>>(P);
        k_cullSurvivors<<<grid(0, 4), CULLER_ROWS, 0, s>>>(P);  // 4 x 64 TMEM columns per SM
    }
    const bool stored = storedKeep(c);
    launch_keep_scan(P, r.work + W_SURVIVORS, r.work + W_KEPT, stored ? r.work + W_FILTER : nullptr, nullptr, s);
    k_walkList<<<grid(c.contactBlocksPerSM, 8), 256, 0, s>>>(P);
    if (stored) {
        k_certifyBuild<<<grid(c.walkBlocksPerSM, 8), 256, 0, s>>>(P);
        launch_keep_scan(P, r.work + W_KEPT, r.work + W_ACTIVE, r.work + W_FILTER, r.walkActive, s);
    }
}
// The exact queries.
static void collectWalk(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (c.meshGeometry == 0) {
        k_sdfEmit<false><<<grid(c.queryBlocksPerSM, 8), 256, 0, s>>>(P);
    } else if (c.filterMargin > 0.0f && c.cullerEnabled == 0) {
        uint32_t g = grid(c.walkBlocksPerSM, 8);
        k_nodeQuery<<<g, 256, 0, s>>>(P);
        k_nodeCertify<<<g, 256, 0, s>>>(P);
        k_nodeWalkSlow<<<g, 256, 0, s>>>(P);
    } else {
        k_nodeWalk<<<grid(c.walkBlocksPerSM, 8), 256, 0, s>>>(P);
    }
}
static void collectQuery(const Params& P, cudaStream_t s) {
    collectFilter(P, s);
    collectWalk(P, s);
}
// The contact records and per-pair starts (with a list built every step, also
// the canonical offsets of the hits).
static void collectEmit(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (c.meshGeometry == 0) return;
    uint32_t g = grid(c.contactBlocksPerSM, 8);
    if (storedKeep(c)) {
        k_emitSlots<false><<<g, 256, 0, s>>>(P);
        return;
    }
    launch_step_scan(r, r.candHitCount, r.candHitOffset, ScanCount{r.work + W_CANDIDATES, c.candidateCapacity, 1, 0}, true,
                r.control + 2, nullptr, s);
    k_nodeEmit<<<g, 256, 0, s>>>(P);
    k_contactStart<<<g, 256, 0, s>>>(P);
}
// Plane contacts after the grain-grain ones: counts, their scan, records.
static void collectWalls(const Params& P, cudaStream_t s) {
    const Res& r = P.r;
    const Config& c = P.c;
    if (c.wallCount == 0) return;
    uint32_t items = c.N * c.wallCount, g = min(blocks(items, 8), grid(0, 8));
    k_wallCount<<<g, 256, 0, s>>>(P);
    launch_step_scan(r, r.wallCounts, r.wallOffsets, ScanCount{nullptr, 0, 0, items}, true, nullptr, nullptr, s);
    k_wallEmit<<<g, 256, 0, s>>>(P);
}
static void contacts(const Params& P, cudaStream_t s) {
    collectCull(P, s);
    collectQuery(P, s);
    collectEmit(P, s);
    collectWalls(P, s);
}
// Contact records with their law, and plane contacts.
static void collectEmitLaw(const Params& P, cudaStream_t s) {
    if (P.c.meshGeometry == 0)
        k_sdfEmit<true><<<grid(P.c.queryBlocksPerSM, 8), 256, 0, s>>>(P);
    else
        k_emitSlots<true><<<grid(P.c.contactBlocksPerSM, 8), 256, 0, s>>>(P);
    collectWalls(P, s);
}
// The exact queries and the above: the part of the collector every step runs
// once the stored filter results are in place.
static void collectTail(const Params& P, cudaStream_t s) {
    if (P.c.meshGeometry != 0) collectWalk(P, s);
    collectEmitLaw(P, s);
}
static void resolveWalls(const Params& P, cudaStream_t s) {
    if (P.c.wallCount) k_resolveWalls<<<grid(0, 2), 256, 0, s>>>(P);
}

int launch_run(const Params& first, const Params& second, uint32_t steps, bool wide, uint32_t* active,
               cudaStream_t s) {
    const Config& c = first.c;
    RunArgs A{{first, second}, steps, c.normalViscosity > 0 ? 1u : 0u, first.r.scanPartials + 2 * SCAN_BLOCKS - 1, active};
    if (cudaError_t e = cudaMemsetAsync(A.counter, 0, sizeof(uint32_t), s); e != cudaSuccess) return int(e);
    const uint32_t ctas = min(smCount(), uint32_t(SCAN_BLOCKS));
    if (c.meshGeometry == 0) return launch_run_sdf(A, ctas, s);
    if (c.wallCount) return wide ? launch_run_walls_wide(A, ctas, s) : launch_run_walls(A, ctas, s);
    return wide ? launch_run_mesh_wide(A, ctas, s) : launch_run_mesh(A, ctas, s);
}

int launch_contacts(const std::string_view& name, const Params& P, uint32_t count, cudaStream_t s) {
    const Config& c = P.c;
    uint32_t T = 256;
    if (name == "neighbours") neighbours(P, s);
    else if (name == "collect") contacts(P, s);
    else if (name == "collectCull") collectCull(P, s);
    else if (name == "collectHead") collectHead(P, s);
    else if (name == "collectHeadKept") {
        k_resetContactsKept<<<1, 1, 0, s>>>(P);
        k_pairSetupKept<<<grid(c.cullBlocksPerSM, 8), T, 0, s>>>(P);
    }
    else if (name == "collectHeadRebuilt") k_pairSetupRebuilt<<<grid(c.cullBlocksPerSM, 8), T, 0, s>>>(P);
    else if (name == "prefetch") {
        if (c.meshGeometry != 0) k_prefetch<<<grid(0, 2), 64, 0, s>>>(P);
    }
    else if (name == "collectBuild") { cullBuild(P, s); collectFilter(P, s); }
    else if (name == "collectTail") collectTail(P, s);
    else if (name == "collectEmitLaw") collectEmitLaw(P, s);
    else if (name == "collectQuery") collectQuery(P, s);
    else if (name == "collectFilter") collectFilter(P, s);
    else if (name == "collectWalk") collectWalk(P, s);
    else if (name == "collectEmit") collectEmit(P, s);
    else if (name == "resolveContacts") {
        k_resolve<<<grid(c.contactBlocksPerSM, 8), T, 0, s>>>(P);
        resolveWalls(P, s);
    }
    else if (name == "resolveWalls") resolveWalls(P, s);
    else if (name == "distanceGrid") {
        if (c.meshGeometry != 0) {
            k_distanceGrid<<<grid(0, 8), T, 0, s>>>(P);
            if (c.triangleLeafEnabled) k_triangleLeaf<<<min(c.shapes, grid(0, 8)), T, 0, s>>>(P);
            if (c.cellListsEnabled) k_cellLists<<<grid(0, 8), T, 0, s>>>(P);
        }
    }
    else if (name == "gather" || name == "gatherFinish") {
        // A warp a grain; fewer (the tuned warps per SM) take several each.
        uint32_t ctas = blocks(c.N, GATHER_WARPS);
        if (c.gatherWarps) ctas = min(ctas, max(1u, grid(c.gatherWarps, 64) / GATHER_WARPS));
        k_gather<<<ctas, 32 * GATHER_WARPS, 0, s>>>(P);
        k_gatherTail<<<blocks(c.N, 128), 128, 0, s>>>(P, name == "gatherFinish");
    }
    else if (name == "collectWalls") collectWalls(P, s);
    else if (name == "gatherWallRows") {
        if (c.wallCount) k_gatherWallRows<<<blocks(c.N * c.wallCount, T), T, 0, s>>>(P);
    }
    else return 1;
    (void)count;
    return 0;
}

}  // namespace sdg

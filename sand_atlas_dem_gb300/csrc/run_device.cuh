// The persistent step: whole steps of an engine in one cooperative launch.
#pragma once
#include "contacts_device.cuh"

namespace sdg {

// ------------------------------------------------------- the persistent step
// Whole steps in one cooperative launch: every phase of a step as above, one
// CTA per SM going through all of them with a barrier over the grid in
// between, and the neighbour and filter builds taken when their device flags
// ask for them.  What a launched step costs besides its kernels -- 4 us per
// graph launch, 1.2 us per kernel boundary and 10 us for a conditional node
// that does not run -- becomes five barriers of 1.3 us.
//
// The barriers carry everything a kernel boundary would: writes before one
// are visible after it on every SM.  Branches around barriers depend only on
// words no CTA writes between the barrier before the branch and the next one
// (never on control[0], which any thread may set at any time).
//
// Two widths: 512 threads (up to 128 registers, no spills) where the phases
// are chains of dependent latencies, 768 (80 registers) where they fill the
// SMs (125 grains 50 / 54 us, 1,000 loose 36 / 40, 343 walled 95 / 102, 10,000
// dense 93 / 89 when both were tried).  Step, us (persistent / launched): 125
// grains 44 / 67; 1,000 loose 40 / 66; 343 walled 88 / 115; 10,000 dense (185 k
// active slots) 87 / 109; but 4,913 walled (425 k) 265 / 240 and 50,000 (1.1 M)
// 328 / 312: there the launched kernels' own register budgets win.
struct GridBarrier {
    uint32_t* counter;
    uint32_t arrived = 0;
    // Waits for every CTA; `live`: no solver flag was set before (a snapshot
    // of this CTA).  False when the wait gave up (about two seconds): the CTA
    // leaves, and so do the others in turn.
    __device__ __forceinline__ bool sync(const Res& r, bool& live) {
        __shared__ uint32_t flagged, reached;
        __syncthreads();
        if (threadIdx.x == 0) {
            arrived += gridDim.x;
            __threadfence();
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
            uint32_t seen = 0;
            for (uint32_t k = 0; k < (1u << 22); ++k) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
                if (seen >= arrived) break;
            }
            __threadfence();
            reached = seen >= arrived;
            if (!reached) fail(r, F_WAIT);
            flagged = *reinterpret_cast<volatile uint32_t*>(r.control);
        }
        __syncthreads();
        live = flagged == 0;
        return reached != 0;
    }
};
// Exclusive scan over the grid: in[0..n) to out, the total to out[n] and
// *total (where given).  With `list` the input holds flags (0 or 1), and a set
// flag's index goes to its place: not on a failed step, whose phases return and
// leave stale flags, and never at or past `room`.  One barrier inside, which
// every CTA takes (`live` may differ among them); the caller's follows.
static __device__ __noinline__ bool runScan(GridBarrier& barrier, bool& live, const Res& r, const uint32_t* in,
                                        uint32_t* out, uint32_t n, bool writeEnd, uint32_t* total,
                                        uint32_t* list = nullptr, uint32_t room = 0) {
    __shared__ uint32_t shared[32], tileTotal;
    const uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t begin = min(n, blockIdx.x * chunk), end = min(n, begin + chunk);
    uint32_t sum = 0;
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) sum += in[i];
    sum = blockInclusive(sum, shared);
    if (threadIdx.x == blockDim.x - 1) r.scanPartials[blockIdx.x] = tileTotal = sum;
    if (!barrier.sync(r, live)) return false;
    const uint32_t own = tileTotal;
    uint32_t before = 0;
    for (uint32_t k = threadIdx.x; k < blockIdx.x; k += blockDim.x) before += r.scanPartials[k];
    before = blockInclusive(before, shared);
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) tileTotal = before;
    __syncthreads();
    uint32_t carry = tileTotal;
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        if (writeEnd) out[n] = carry + own;
        if (total) *total = carry + own;
    }
    __syncthreads();
    for (uint32_t base = begin; base < end; base += blockDim.x) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < end ? in[i] : 0;
        uint32_t inc = blockInclusive(v, shared);
        if (i < end) {
            out[i] = carry + inc - v;
            if (list && v && live && carry + inc - v < room) list[carry + inc - v] = i;
        }
        if (threadIdx.x == blockDim.x - 1) tileTotal = inc;
        __syncthreads();
        carry += tileTotal;
        __syncthreads();
    }
    return true;
}
#define RUN_SYNC() do { if (!barrier.sync(r, live)) return; } while (0)
// The phases few steps take, out of line: the code every step runs stays small
// (a phase of a small run is fetched once and executed once a step).
namespace rare {
#define RARE(name) static __device__ __noinline__ void name(const Params& P) { sdg::name(P); }
#define RARE_LIVE(name) static __device__ __noinline__ void name(const Params& P, bool live) { sdg::name(P, live); }
RARE(binsClear) RARE(binsFill) RARE(binsOrder) RARE(pairsCountWarp) RARE(pairsEmitWarp) RARE(byJReset)
RARE(byJCount) RARE(byJFill) RARE(byJSort) RARE(leafEmit) RARE(nodeFilter) RARE(survivorList)
RARE(survivorPrefilter) RARE(walkList)
RARE_LIVE(leafCull) RARE_LIVE(certifyBuild) RARE_LIVE(nodeCertify) RARE_LIVE(nodeWalkSlow)
#undef RARE
#undef RARE_LIVE
}  // namespace rare
template <int Threads, bool Mesh, bool Walls>
__global__ void __launch_bounds__(Threads, 1) k_run(const __grid_constant__ RunArgs A) {
    extern __shared__ __align__(16) GatherScratch runScratch[];
    GridBarrier barrier{A.counter};
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    bool live = A.side[0].r.control[0] == 0;
    for (uint32_t k = 0; k < A.steps; ++k) {
        const Params& P = A.side[k & 1u];
        const Res& r = P.r;
        const Config& c = P.c;
        const bool guarded = c.activeTimestep != 0;
        if (guarded) {
            if (r.control[0] == 0)
                for (uint32_t id = gtid(); id < c.N; id += gstride()) checkGrainTimestep(r, c, id);
            RUN_SYNC();
        }
        // Drift; the cell rows (read by no grain here); the step's counters.
        if (r.control[0] == 0) {
            // (The last CTA's last warps, which have the fewest grains.)
            const uint32_t fromEnd = blockDim.x - 1 - threadIdx.x;
            if (blockIdx.x == gridDim.x - 1) {
                for (uint32_t sp = fromEnd; sp < c.specimens; sp += blockDim.x) advanceCellRow(r, c, sp);
                if (fromEnd == WARP) resetContacts(r, c, false);
            }
            for (uint32_t id = gtid(); id < c.N; id += gstride())
                if (beginGrain(r, c, id, A.capture != 0)) atomicOr(&r.work[W_MOVED], 1u);
        }
        RUN_SYNC();
        const bool moved = r.work[W_MOVED] != 0;
        if (first && live) r.control[4] = moved ? 1u : 0u;
        if (moved) {
            RUN_SYNC();
            rare::binsClear(P);
            RUN_SYNC();
            rare::binsFill(P);
            RUN_SYNC();
            rare::binsOrder(P);
            RUN_SYNC();
            rare::pairsCountWarp(P);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.pairCounts, r.pairOffsets, c.N, false, r.control + 1)) return;
            RUN_SYNC();
            rare::pairsEmitWarp(P);
            rare::byJReset(P);
            RUN_SYNC();
            rare::byJCount(P);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.byJCounts, r.byJOffsets, c.N, true, nullptr)) return;
            RUN_SYNC();
            rare::byJFill(P);
            RUN_SYNC();
            rare::byJSort(P);
            RUN_SYNC();
        }
        if (blockIdx.x == gridDim.x - 1 && live) {
            const uint32_t fromEnd = blockDim.x - 1 - threadIdx.x;
            for (uint32_t sp = fromEnd; sp < c.specimens; sp += blockDim.x) advanceCellLog(r, c, sp);
            if (fromEnd == WARP && Walls) advanceWallPlanes(r, c);
            if (fromEnd == 2 * WARP && r.work[W_FILTER_PAIRS] != r.control[1]) atomicOr(&r.work[W_FILTER], 1u);
        }
        pairSetup(P);
        RUN_SYNC();
        if (first) r.work[W_MOVED] = 0;
        if (Mesh && r.work[W_FILTER] != 0) {
            rare::leafCull(P, live);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.dpairLeafCount, r.dpairCandOffset, 2 * activePairs(r, c), true,
                         r.work + W_CANDIDATES))
                return;
            RUN_SYNC();
            rare::leafEmit(P);
            RUN_SYNC();
            rare::nodeFilter(P);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.candSurvCount, r.candSurvOffset,
                         min(r.work[W_CANDIDATES], c.candidateCapacity), true, r.work + W_SURVIVORS))
                return;
            RUN_SYNC();
            rare::survivorList(P);
            RUN_SYNC();
            rare::survivorPrefilter(P);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.survKeep, r.keepOffset, min(r.work[W_SURVIVORS], c.survivorCapacity), true,
                         r.work + W_KEPT))
                return;
            RUN_SYNC();
            rare::walkList(P);
            RUN_SYNC();
            rare::certifyBuild(P, live);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.survKeep, r.keepOffset, min(r.work[W_KEPT], c.survivorCapacity), true,
                         r.work + W_ACTIVE, r.walkActive, c.survivorCapacity))
                return;
            RUN_SYNC();
        }
        if (!Mesh) {
            // (the gather's scratch holds the lists: 2 x 64 words a warp)
            uint32_t* lists = reinterpret_cast<uint32_t*>(&runScratch[threadIdx.x >> 5]);
            sdfQueryPairs(P, lists, lists + SDF_LIST, live);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.contactCounts, r.contactOffsets, activePairs(r, c), false, r.control + 2)) return;
            RUN_SYNC();
            sdfEmit<true>(P);
        } else {
            nodeQuery(P, live);
            RUN_SYNC();
            bool walked = false;
            if (r.work[W_LAPSED] != 0) {
                rare::nodeCertify(P, live);
                RUN_SYNC();
                if (r.work[W_SLOW] != 0) {
                    walked = true;
                    rare::nodeWalkSlow(P, live);
                    RUN_SYNC();
                }
            }
            if (first && live && !walked) r.work[W_CERTIFIED] += min(r.work[W_KEPT], c.survivorCapacity);
            emitSlots<true>(P, live);
        }
        if (Walls) {
            RUN_SYNC();
            wallCount(P, live);
            RUN_SYNC();
            if (!runScan(barrier, live, r, r.wallCounts, r.wallOffsets, c.N * c.wallCount, true, nullptr)) return;
            RUN_SYNC();
            wallEmit(P, live);
            RUN_SYNC();
            resolveWalls(P);
        }
        RUN_SYNC();
        gather(P, runScratch[threadIdx.x >> 5], live, true, !Walls && !guarded);
        if (Walls) gatherWallRows(P);
        RUN_SYNC();
        if (Walls || guarded) {
            if (guarded) {
                if (r.control[0] == 0)
                    for (uint32_t id = gtid(); id < c.N; id += gstride()) checkGrainTimestep(r, c, id);
                RUN_SYNC();
            }
            if (r.control[0] == 0)
                for (uint32_t id = gtid(); id < c.N; id += gstride()) finishGrain(r, c, id);
            RUN_SYNC();
        }
    }
    if (first && A.active) *A.active = A.side[0].r.work[W_ACTIVE];
}
#undef RUN_SYNC

template <int Threads, bool Mesh, bool Walls>
static int launchRun(const RunArgs& A, uint32_t ctas, cudaStream_t s) {
    const void* kernel = reinterpret_cast<const void*>(k_run<Threads, Mesh, Walls>);
    const size_t shared = Threads / WARP * sizeof(GatherScratch);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shared));
    if (e != cudaSuccess) return int(e);
    void* args[] = {const_cast<RunArgs*>(&A)};
    return int(cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(Threads), args, shared, s));
}

}  // namespace sdg

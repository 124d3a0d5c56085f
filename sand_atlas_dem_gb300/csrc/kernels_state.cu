// Per-grain state kernels: kick-drift-kick integrator with affine periodic
// cell streaming, cell update, Verlet rebuild trigger, timestep guard and the
// diagnostic rows with their fixed-order tree reduction.
//
// Each kernel is one thread per grain (HBM-bound: ~0.5 KB of float4 state per
// grain and step) and restates the arithmetic of the reference kernel named
// beside it, in the same FP32 operation order.
#include "state_device.cuh"
#include "launch.h"

namespace sdg {

// solver.slang:858-888, and the rebuild trigger (:898-904) in the step's new
// cell, flagged in work[W_MOVED] for k_advanceCell.
__global__ void k_beginStep(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t id = gtid();
    if (id >= P.c.N || r.control[0] != 0) return;
    if (beginGrain(r, P.c, id, P.c.viscousCapture != 0)) atomicOr(&r.work[W_MOVED], 1u);
}

// solver.slang:170-175 (stand-alone form, used by initialize/restore paths)
__global__ void k_captureContactKinematics(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t id = gtid();
    if (id >= P.c.N || r.control[0] != 0) return;
    r.forceVelocity[id] = w4(xyz(r.velocity[id]) + xyz(r.velocityRemainder[id]), 0.f);
    r.forceOmega[id] = w4(omegaOf(r, id), 0.f);
}

// solver.slang:889-897, one thread per specimen, and the step's rebuild flag.
__global__ void k_advanceCell(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t sp = gtid();
    uint32_t moved = 0;
    if (sp == 0) {
        moved = r.work[W_MOVED];
        r.work[W_MOVED] = 0;  // also on a failed step, which is rolled back
    }
    if (sp >= P.c.specimens || r.control[0] != 0) return;
    advanceCellRow(r, P.c, sp);
    advanceCellLog(r, P.c, sp);
    if (sp == 0) r.control[4] = moved;
}

// solver.slang:898-904 by itself (the step's own check is beginStep's).
__global__ void k_checkRebuild(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t id = gtid();
    if (id >= P.c.N) return;
    uint32_t sp = specimenOf(r, id);
    if (movedBeyondSkin(P.c, xyz(r.cell[3 * sp]), xyz(r.position[id]), xyz(r.positionRemainder[id]),
                        r.referencePosition[id], r.referencePositionRemainder[id], r.referenceCell[2 * sp]))
        atomicOr(&r.control[4], 1u);
}

// solver.slang:905-920
__global__ void k_finishStep(const __grid_constant__ Params P) {
    uint32_t id = gtid();
    if (id >= P.c.N || P.r.control[0] != 0) return;
    finishGrain(P.r, P.c, id);
}

// solver.slang:815-832
__global__ void k_checkContactTimestep(const __grid_constant__ Params P) {
    uint32_t id = gtid();
    if (id >= P.c.N || P.r.control[0] != 0) return;
    checkGrainTimestep(P.r, P.c, id);
}

// solver.slang:922-936
__device__ __forceinline__ void diagnosticRow(const Res& r, uint32_t id, float4 (&row)[8]) {
    f3 v = xyz(r.velocity[id]);
    float m = r.body[id].y;
    float kinetic = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(m, dot(v, v)), dot(xyz(r.momentum[id]), omegaOf(r, id))));
    row[0] = w4(xyz(r.particleStress[3 * id]), kinetic);
    row[1] = w4(xyz(r.particleStress[3 * id + 1]), r.particleDiagnostic[id].y);
    row[2] = w4(xyz(r.particleStress[3 * id + 2]), length(xyz(r.force[id])));
    row[3] = w4(__fmul_rn(m, v.x) * v, r.particleDiagnostic[id].w);
    row[4] = w4(__fmul_rn(m, v.y) * v, r.force[id].w);
    row[5] = w4(__fmul_rn(m, v.z) * v, r.torque[id].w);
    row[6] = r.accumulated[id];
    float4 ns = r.normalDamping[id];
    row[7] = make_float4(__fadd_rn(ns.x, ns.y), ns.z, 0.f, 0.f);
}
__global__ void k_diagnosticRows(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t id = gtid();
    if (id >= P.c.N) return;
    float4 row[8];
    diagnosticRow(r, id, row);
#pragma unroll
    for (int k = 0; k < 8; ++k) r.diagnosticRows[8 * size_t(id) + k] = row[k];
}

// solver.slang:938-947
__device__ __forceinline__ void fabricRow(const Res& r, const Config& c, uint32_t id, float4& a, float4& b) {
    a = make_float4(0.f, 0.f, 0.f, 0.f);
    b = a;
    if (id < r.control[1] && r.contactCounts[id] > 0) {
        uint2 ij = r.pairs[id];
        f3 d = centerBranch64(r, c, ij.x, ij.y);
        f3 n = d * __fdiv_rn(1.0f, __fsqrt_rn(dot(d, d)));
        a = make_float4(__fmul_rn(n.x, n.x), __fmul_rn(n.y, n.y), __fmul_rn(n.z, n.z), __fmul_rn(n.x, n.y));
        b = make_float4(__fmul_rn(n.x, n.z), __fmul_rn(n.y, n.z), 1.f, 0.f);
    }
}
__global__ void k_fabricRows(const __grid_constant__ Params P) {
    const Res& r = P.r;
    uint32_t id = gtid();
    if (id >= P.c.pairCapacity) return;
    fabricRow(r, P.c, id, r.fabricRows[2 * id], r.fabricRows[2 * id + 1]);
}

// ---- all of Engine.diagnostics in two launches.  The reference reduces the
// per-grain, per-pair and per-(wall, grain) rows by 256-wide trees, level by
// level (diagnostic.slang:3-49); here the first level is taken where the rows
// are computed (no row goes through memory: 128 B a grain, 32 B a reserved
// pair) and the rest by one CTA, a warp a tree.  The pairs past the active
// ones are zeros of the same tree and are not visited.
// One 256-wide tree by a warp: value(k) for k < 256 in the order of the
// reference's strides 128, 64, ..., 1 (the first three within a lane).  With
// `maximum` the w components' largest instead of their sum, with `count`
// their sum as integers.
template <class Value>
__device__ __forceinline__ float4 treeOf256(Value&& value, bool maximum, bool count) {
    const uint32_t lane = threadIdx.x & 31u;
    float4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = value(lane + 32 * j);
    auto merge = [&](float4 a, float4 b) {
        float4 s = add4(a, b);
        if (maximum) s.w = mx(a.w, b.w);
        if (count) s.w = __uint_as_float(__float_as_uint(a.w) + __float_as_uint(b.w));
        return s;
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = merge(v[j], v[j + 4]);
    v[0] = merge(v[0], v[2]);
    v[1] = merge(v[1], v[3]);
    v[0] = merge(v[0], v[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float4 w = make_float4(__shfl_down_sync(0xffffffffu, v[0].x, o), __shfl_down_sync(0xffffffffu, v[0].y, o),
                               __shfl_down_sync(0xffffffffu, v[0].z, o), __shfl_down_sync(0xffffffffu, v[0].w, o));
        v[0] = merge(v[0], w);
    }
    return v[0];
}
// First level: CTA g < groups the grains' rows; the next pairGroups the
// pairs'; the last wallCount x groups the (wall, grain) rows.  The sums go to
// the start of the row buffers they stand for (diagnosticRows, fabricRows)
// and to wallSums, `wallStride` rows of three a wall.
__global__ void __launch_bounds__(256) k_diagnosticGroups(const __grid_constant__ Params P, uint32_t groups,
                                                          uint32_t pairGroups, float4* wallSums, uint32_t wallStride) {
    __shared__ float4 rows[8][256];
    const Res& r = P.r;
    const Config& c = P.c;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t g = blockIdx.x;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g < groups) {
        const uint32_t id = 256 * g + threadIdx.x;
        float4 row[8] = {zero, zero, zero, zero, zero, zero, zero, zero};
        if (id < c.N) diagnosticRow(r, id, row);
#pragma unroll
        for (int k = 0; k < 8; ++k) rows[k][threadIdx.x] = row[k];
        __syncthreads();
        float4 sum = treeOf256([&](uint32_t k) { return rows[warp][k]; }, warp == 4, false);
        if (lane == 0) r.diagnosticRows[8 * size_t(g) + warp] = sum;
        return;
    }
    g -= groups;
    if (g < pairGroups) {
        if (256 * g >= r.control[1]) return;  // (block-uniform) zeros: not visited above either
        const uint32_t id = 256 * g + threadIdx.x;
        float4 a = zero, b = zero;
        if (id < c.pairCapacity) fabricRow(r, c, id, a, b);
        rows[0][threadIdx.x] = a;
        rows[1][threadIdx.x] = b;
        __syncthreads();
        if (warp < 2) {
            float4 sum = treeOf256([&](uint32_t k) { return rows[warp][k]; }, false, false);
            if (lane == 0) r.fabricRows[2 * size_t(g) + warp] = sum;
        }
        return;
    }
    g -= pairGroups;
    const uint32_t wall = g / groups, group = g % groups;
    if (warp < 3) {
        float4 sum = treeOf256(
            [&](uint32_t k) {
                const uint32_t id = 256 * group + k;
                return id < c.N ? r.wallRows[3 * (size_t(wall) * c.N + id) + warp] : zero;
            },
            false, warp == 0);
        if (lane == 0) wallSums[3 * (size_t(wall) * wallStride + group) + warp] = sum;
    }
}
// The remaining levels and the words the host reads: 8 grain rows, 2 fabric
// rows, 3 cell rows, 16 control words, then per wall its 3 rows, plane,
// remainder and velocity.  One CTA.
__global__ void __launch_bounds__(1024) k_diagnosticTotals(const __grid_constant__ Params P, uint32_t groups,
                                                           uint32_t pairGroups, float4* wallSums, uint32_t wallStride,
                                                           float4* out) {
    const Res& r = P.r;
    const Config& c = P.c;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // A level's results go behind its inputs: the row buffers hold 256 times
    // the first level's sums, a wall's stride what its levels need.
    auto totals = [&](float4* rows, uint32_t n, uint32_t present, uint32_t width, int maxRow, int countRow,
                      float4* result) {
        float4* in = rows;
        while (n > 1) {
            const uint32_t next = (n + 255) / 256, left = (present + 255) / 256;
            float4* sums = in + size_t(width) * n;
            for (uint32_t u = warp; u < left * width; u += warps) {
                const uint32_t g = u / width, row = u % width;
                float4 sum = treeOf256(
                    [&](uint32_t k) {
                        const uint32_t at = 256 * g + k;
                        return at < present ? in[size_t(width) * at + row] : zero;
                    },
                    int(row) == maxRow, int(row) == countRow);
                if (lane == 0) sums[size_t(width) * g + row] = sum;
            }
            __syncthreads();
            in = sums;
            n = next;
            present = left;
        }
        if (threadIdx.x < width) result[threadIdx.x] = present ? in[threadIdx.x] : zero;
    };
    const uint32_t pairs = min(r.control[1], c.pairCapacity);
    totals(r.diagnosticRows, groups, groups, 8, 4, -1, out);
    totals(r.fabricRows, pairGroups, (pairs + 255) / 256, 2, -1, -1, out + 8);
    if (threadIdx.x < 3) out[10 + threadIdx.x] = r.cell[threadIdx.x];
    if (threadIdx.x < 16) reinterpret_cast<uint32_t*>(out + 13)[threadIdx.x] = r.control[threadIdx.x];
    float4* walls = out + 17;
    for (uint32_t w = 0; w < c.wallCount; ++w) {
        totals(wallSums + 3 * size_t(w) * wallStride, groups, groups, 3, -1, 0, walls + 6 * w);
        if (threadIdx.x == 0) {
            walls[6 * w + 3] = r.wallPlane[w];
            walls[6 * w + 4] = r.wallRemainder[w];
            walls[6 * w + 5] = r.wallVelocity[w];
        }
    }
}

// diagnostic.slang:3-28: per 256-row group, values[lane] += values[lane+step]
// for step = 128..1; (maxRow, 3) reduces with max instead of sum.
__global__ void k_reduceRows(const float4* input, float4* output, uint32_t n, uint32_t rows, int maxRow) {
    __shared__ float4 values[256];
    uint32_t lane = threadIdx.x, id = blockIdx.x * 256 + lane;
    for (uint32_t row = 0; row < rows; ++row) {
        values[lane] = id < n ? input[size_t(id) * rows + row] : make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        for (uint32_t step = 128; step > 0; step /= 2) {
            if (lane < step) {
                float4 a = values[lane], b = values[lane + step];
                float4 s = add4(a, b);
                if (int(row) == maxRow) s.w = mx(a.w, b.w);
                values[lane] = s;
            }
            __syncthreads();
        }
        if (lane == 0) output[size_t(blockIdx.x) * rows + row] = values[0];
        __syncthreads();
    }
}

// solver.slang:669-687, one thread.
__global__ void k_advanceWalls(const __grid_constant__ Params P) {
    if (gtid() == 0 && P.r.control[0] == 0) advanceWallPlanes(P.r, P.c);
}
// solver.slang:950-955: wall power of the committed rows at new wall
// velocities (no contact is re-resolved).
__global__ void k_refreshWallPower(const __grid_constant__ Params P) {
    const Res& r = P.r;
    const Config& c = P.c;
    uint32_t total = c.N * c.wallCount;
    for (uint32_t index = gtid(); index < total; index += gstride()) {
        float4 value = r.wallRows[3 * index + 1];
        value.w = -dot(xyz(r.wallRows[3 * index]), xyz(r.wallVelocity[index / c.N]));
        r.wallRows[3 * index + 1] = value;
    }
}
// diagnostic.slang:33-49: per wall, 256-row tree sums of the three
// (wall, grain) rows, the contact count (row 0, w) summed as an integer.
__global__ void k_reduceWallRows(const float4* input, float4* output, uint32_t n, uint32_t outputCount) {
    __shared__ float4 values[256];
    __shared__ uint32_t counts[256];
    uint32_t lane = threadIdx.x, id = blockIdx.x * 256 + lane, wall = blockIdx.y;
    for (uint32_t row = 0; row < 3; ++row) {
        float4 value = id < n ? input[3 * (size_t(wall) * n + id) + row] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (row == 0) {
            counts[lane] = __float_as_uint(value.w);
            value.w = 0.f;
        }
        values[lane] = value;
        __syncthreads();
        for (uint32_t step = 128; step > 0; step /= 2) {
            if (lane < step) {
                values[lane] = add4(values[lane], values[lane + step]);
                if (row == 0) counts[lane] += counts[lane + step];
            }
            __syncthreads();
        }
        if (lane == 0) {
            float4 total = values[0];
            if (row == 0) total.w = __uint_as_float(counts[0]);
            output[3 * (size_t(wall) * outputCount + blockIdx.x) + row] = total;
        }
        __syncthreads();
    }
}

static inline uint32_t blocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

int launch_state(const std::string_view& name, const Params& P, uint32_t count, cudaStream_t s) {
    const uint32_t T = 256;
    uint32_t n = count ? count : 1;
    if (name == "beginStep") k_beginStep<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "captureContactKinematics") k_captureContactKinematics<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "advanceCell") k_advanceCell<<<blocks(P.c.specimens, 64), 64, 0, s>>>(P);
    else if (name == "checkRebuild") k_checkRebuild<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "finishStep") k_finishStep<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "checkContactTimestep") k_checkContactTimestep<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "diagnosticRows") k_diagnosticRows<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "fabricRows") k_fabricRows<<<blocks(n, T), T, 0, s>>>(P);
    else if (name == "advanceWalls") k_advanceWalls<<<1, 32, 0, s>>>(P);
    else if (name == "refreshWallPower") k_refreshWallPower<<<blocks(max(1u, P.c.N * P.c.wallCount), T), T, 0, s>>>(P);
    else return 1;
    return 0;
}

uint64_t diagnostic_rows(const Config& c) { return DIAGNOSTIC_ROWS + 6ull * c.wallCount; }
uint32_t diagnostic_wall_stride(const Config& c) {
    uint32_t groups = blocks(c.N, 256), rows = groups;
    for (uint32_t n = groups; n > 1; rows += n) n = blocks(n, 256);
    return rows;
}
void launch_diagnostics(const Params& P, float4* wallSums, float4* out, cudaStream_t s) {
    const uint32_t groups = blocks(P.c.N, 256), pairGroups = blocks(P.c.pairCapacity, 256);
    const uint32_t stride = diagnostic_wall_stride(P.c);
    k_diagnosticGroups<<<groups * (1 + P.c.wallCount) + pairGroups, 256, 0, s>>>(P, groups, pairGroups, wallSums, stride);
    k_diagnosticTotals<<<1, 1024, 0, s>>>(P, groups, pairGroups, wallSums, stride, out);
}

void launch_reduce_rows(const float4* input, float4* output, uint32_t n, uint32_t rows, int maxRow, cudaStream_t s) {
    k_reduceRows<<<blocks(n, 256), 256, 0, s>>>(input, output, n, rows, maxRow);
}

void launch_reduce_wall_rows(const float4* input, float4* output, uint32_t n, uint32_t walls, cudaStream_t s) {
    uint32_t groups = blocks(n, 256);
    k_reduceWallRows<<<dim3(groups, walls), 256, 0, s>>>(input, output, n, groups);
}

}  // namespace sdg

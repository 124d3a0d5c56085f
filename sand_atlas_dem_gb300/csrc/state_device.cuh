// The integrator's per-grain steps, shared by the kernels of a launched step
// (kernels_state.cu) and the persistent step (run_device.cuh): the
// arithmetic of the reference kernel named beside each, in its FP32 order.
#pragma once
#include "dem_device.cuh"

namespace sdg {

// A grain's rows the half kicks read, loaded together before anything is
// stored: a store ends the batch of loads a thread can have in flight (the
// compiler must assume it aliases the next), and each batch costs a trip to
// L2.  The drift of 10,000 grains took seven such trips in a row.
struct KickRows {
    float4 damping, v, vl, l, ll, force, torque, q, inertia[3], stress[3], high, low;
    float mass;
};
__device__ __forceinline__ KickRows kickRows(const Res& r, uint32_t id) {
    KickRows k;
    k.damping = r.normalDamping[id];
    k.v = r.velocity[id];
    k.vl = r.velocityRemainder[id];
    k.l = r.momentum[id];
    k.ll = r.momentumRemainder[id];
    k.force = r.force[id];
    k.torque = r.torque[id];
    k.q = r.rotation[id];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        k.inertia[a] = r.invI[3 * id + a];
        k.stress[a] = r.particleStress[3 * id + a];
    }
    k.high = r.accumulated[id];
    k.low = r.accumulatedRemainder[id];
    k.mass = r.body[id].y;
    return k;
}
// solver.slang:154-158 with the inertia rows at hand
__device__ __forceinline__ f3 omegaRows(const float4 (&inertia)[3], float4 q, f3 l) {
    f3 b = qinv(q, l);
    f3 w = {dot(xyz(inertia[0]), b), dot(xyz(inertia[1]), b), dot(xyz(inertia[2]), b)};
    return qrot(q, w);
}
// solver.slang:159-163
__device__ __forceinline__ float rotationalEnergy(const float4 (&inertia)[3], float4 q, f3 l) {
    f3 b = qinv(q, l);
    f3 w = {dot(xyz(inertia[0]), b), dot(xyz(inertia[1]), b), dot(xyz(inertia[2]), b)};
    return __fmul_rn(0.5f, dot(b, w));
}
// Half kick, drag and its losses, shared by beginStep and finishStep, on the
// loaded rows in a cell of `rate`: the normal contact loss (solver.slang:
// 164-169), the kick, the drag loss and cell power (:176-180, the velocity as
// stored) and the wall work into the accumulators (:130-134), which are
// stored.  v, vl, l, ll: the kicked and dragged state.
__device__ __forceinline__ void halfKick(const Res& r, const Config& c, uint32_t id, KickRows& k, f3 rate, f3& v,
                                         f3& vl, f3& l, f3& ll) {
    float dt = c.dt, m = k.mass;
    float hdt = __fmul_rn(0.5f, dt);
    float wallWork = wallStepWork(r, c, id, hdt);
    f3 high = mk(k.damping.x, 0.f, 0.f), low = mk(k.damping.y, 0.f, 0.f);
    compensated3(high, low, mk(__fmul_rn(k.damping.z, hdt), 0.f, 0.f));
    k.damping.x = high.x;
    k.damping.y = low.x;
    v = xyz(k.v);
    vl = xyz(k.vl);
    l = xyz(k.l);
    ll = xyz(k.ll);
    compensated3(v, vl, (hdt * xyz(k.force)) / m);
    compensated3(l, ll, hdt * xyz(k.torque));
    f3 vs = v + vl;
    float loss = __fmul_rn(-expm1Stable(__fmul_rn(-c.drag, dt)),
                           __fadd_rn(__fmul_rn(__fmul_rn(0.5f, m), dot(vs, vs)),
                                     rotationalEnergy(k.inertia, k.q, l + ll)));
    f3 diagonal = mk(k.stress[0].x, k.stress[1].y, k.stress[2].z), stored = xyz(k.v);
    float cp = __fmul_rn(hdt, -dot(diagonal + (m * stored) * stored, rate));
    compensated4(k.high, k.low, make_float4(0.f, loss, cp, wallWork));
    float damping = expm1Stable(__fmul_rn(__fmul_rn(-0.5f, c.drag), dt));
    compensated3(v, vl, damping * (v + vl));
    compensated3(l, ll, damping * (l + ll));
    r.normalDamping[id] = k.damping;
    r.accumulated[id] = k.high;
    r.accumulatedRemainder[id] = k.low;
}

// Whether a grain has moved far enough from its place at the last neighbour
// build to ask for another (solver.slang:898-904), in a cell `box`.
__device__ __forceinline__ bool movedBeyondSkin(const Config& c, f3 box, f3 p, f3 pl, float4 referencePosition,
                                                float4 referenceRemainder, float4 referenceCell) {
    f3 d = (p - xyz(referencePosition)) + (pl - xyz(referenceRemainder));
    if (c.periodic != 0) {
        d = d - mk(floorf(__fadd_rn(__fdiv_rn(d.x, box.x), 0.5f)), floorf(__fadd_rn(__fdiv_rn(d.y, box.y), 0.5f)),
                   floorf(__fadd_rn(__fdiv_rn(d.z, box.z), 0.5f))) * box;
    }
    float deformation = length(box - xyz(referenceCell));
    return __fadd_rn(length(d), deformation) > __fmul_rn(0.5f, c.skin);
}
// solver.slang:858-888 (+ captureContactKinematics :170-175 with `capture`).
// The step's new cell depends on its logarithm and rate alone, so the grain
// also answers whether it asks for a neighbour build in it (checkRebuild),
// without waiting for the cell rows to be written.
__device__ __forceinline__ bool beginGrain(const Res& r, const Config& c, uint32_t id, bool capture) {
    float dt = c.dt;
    uint32_t sp = specimenOf(r, id);
    KickRows k = kickRows(r, id);
    float4 ql = r.rotationRemainder[id], position = r.position[id], remainder = r.positionRemainder[id];
    float4 referencePosition = r.referencePosition[id], referenceRemainder = r.referencePositionRemainder[id];
    f3 rate = xyz(r.cell[3 * sp + 1]), initial = xyz(r.cell[3 * sp + 2]);
    f3 logarithm = xyz(r.cellLog[2 * sp]), residual = xyz(r.cellLog[2 * sp + 1]);
    float4 referenceCell = r.referenceCell[2 * sp];
    f3 v, vl, l, ll;
    halfKick(r, c, id, k, rate, v, vl, l, ll);
    float4 q = k.q;
    f3 lt = l + ll;
    f3 w = omegaRows(k.inertia, q, lt);
    float4 mid = normalize4(add4(q, rotationIncrement(w, __fmul_rn(0.5f, dt), q)));
    w = omegaRows(k.inertia, mid, lt);
    compensated4(q, ql, rotationIncrement(w, dt, q));
    if (fabsf(__fsub_rn(dot4(q, q), 1.0f)) > 2e-6f) {
        q = normalize4(q);
        ql = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    compensated3(logarithm, residual, rate * dt);
    f3 box = initial * exp3(logarithm);
    f3 p = xyz(position), pl = xyz(remainder);
    compensated3(p, pl, expm1Stable3(rate * dt) * (p + pl) + dt * (v + vl));
    r.momentum[id] = w4(l, 0.f);
    r.momentumRemainder[id] = w4(ll, 0.f);
    r.rotation[id] = q;
    r.rotationRemainder[id] = ql;
    if (!finite3(p) || !finite3(pl)) { fail(r, F_NONFINITE); return false; }
    if (c.periodic != 0) {
        p = p - mk(floorf(__fdiv_rn(p.x, box.x)), floorf(__fdiv_rn(p.y, box.y)), floorf(__fdiv_rn(p.z, box.z))) * box;
    } else if (__fadd_rn(p.x, pl.x) < 0 || __fadd_rn(p.y, pl.y) < 0 || __fadd_rn(p.z, pl.z) < 0 ||
               __fadd_rn(__fsub_rn(p.x, box.x), pl.x) >= 0 || __fadd_rn(__fsub_rn(p.y, box.y), pl.y) >= 0 ||
               __fadd_rn(__fsub_rn(p.z, box.z), pl.z) >= 0) {
        fail(r, F_ESCAPE);
        return false;
    }
    r.position[id] = w4(p, 0.f);
    r.positionRemainder[id] = w4(pl, 0.f);
    compensated3(v, vl, expm1Stable3((-rate) * dt) * (v + vl));
    r.velocity[id] = w4(v, 0.f);
    r.velocityRemainder[id] = w4(vl, 0.f);
    if (capture) {
        r.forceVelocity[id] = w4(v + vl, 0.f);
        r.forceOmega[id] = w4(omegaRows(k.inertia, q, lt), 0.f);
    }
    return movedBeyondSkin(c, box, p, pl, referencePosition, referenceRemainder, referenceCell);
}
// solver.slang:889-897: the new cell row of specimen sp.
__device__ __forceinline__ void advanceCellRow(const Res& r, const Config& c, uint32_t sp) {
    f3 logarithm = xyz(r.cellLog[2 * sp]), residual = xyz(r.cellLog[2 * sp + 1]);
    compensated3(logarithm, residual, xyz(r.cell[3 * sp + 1]) * c.dt);
    r.cell[3 * sp] = w4(xyz(r.cell[3 * sp + 2]) * exp3(logarithm), 0.f);
}
// ... and its logarithm, with the image check.
__device__ __forceinline__ void advanceCellLog(const Res& r, const Config& c, uint32_t sp) {
    f3 logarithm = xyz(r.cellLog[2 * sp]), residual = xyz(r.cellLog[2 * sp + 1]);
    compensated3(logarithm, residual, xyz(r.cell[3 * sp + 1]) * c.dt);
    r.cellLog[2 * sp] = w4(logarithm, 0.f);
    r.cellLog[2 * sp + 1] = w4(residual, 0.f);
    float4 cell = r.cell[3 * sp];
    if (c.periodic != 0 && r.referenceCell[2 * sp + 1].w >= __fmul_rn(0.5f, mn(cell.x, mn(cell.y, cell.z))))
        fail(r, F_IMAGE);
}
// solver.slang:905-920
__device__ __forceinline__ void finishRows(const Res& r, const Config& c, uint32_t id, KickRows& k, f3 rate) {
    f3 v, vl, l, ll;
    halfKick(r, c, id, k, rate, v, vl, l, ll);
    if (!finite3(v) || !finite3(l)) { fail(r, F_NONFINITE); return; }
    r.velocity[id] = w4(v, 0.f);
    r.velocityRemainder[id] = w4(vl, 0.f);
    r.momentum[id] = w4(l, 0.f);
    r.momentumRemainder[id] = w4(ll, 0.f);
}
__device__ __forceinline__ void finishGrain(const Res& r, const Config& c, uint32_t id) {
    KickRows k = kickRows(r, id);
    finishRows(r, c, id, k, xyz(r.cell[3 * specimenOf(r, id) + 1]));
}
__device__ __forceinline__ float inverseInertiaBound(const Res& r, uint32_t id) {
    f3 one = mk(1.f, 1.f, 1.f);
    return mx(mx(dot(abs3(xyz(r.invI[3 * id])), one), dot(abs3(xyz(r.invI[3 * id + 1])), one)),
              dot(abs3(xyz(r.invI[3 * id + 2])), one));
}

// solver.slang:815-832
__device__ __forceinline__ void checkGrainTimestep(const Res& r, const Config& c, uint32_t id) {
    if (c.dt == 0) return;
    float dt = c.dt;
    float4 rates = r.timestepRows[id];
    f3 v = xyz(r.velocity[id]) + xyz(r.velocityRemainder[id]);
    float speed = __fadd_rn(length(v), __fdiv_rn(__fmul_rn(dt, length(xyz(r.force[id]))), r.body[id].y));
    float inverseInertia = inverseInertiaBound(r, id);
    float spin = __fmul_rn(inverseInertia, __fadd_rn(length(xyz(r.momentum[id]) + xyz(r.momentumRemainder[id])),
                                                     __fmul_rn(dt, length(xyz(r.torque[id])))));
    float wallSpeed = 0.f;
    for (uint32_t w = 0; w < c.wallCount; ++w) wallSpeed = mx(wallSpeed, length(xyz(r.wallVelocity[w])));
    float motion = __fmul_rn(dt, __fadd_rn(__fadd_rn(speed, __fmul_rn(r.body[id].z, spin)), wallSpeed));
    bool finite = isfinite(rates.x) && isfinite(rates.y) && isfinite(motion) && isfinite(spin);
    if (!finite) { fail(r, F_NONFINITE); return; }
    f3 rate = abs3(xyz(r.cell[3 * specimenOf(r, id) + 1]));
    if (__fmul_rn(dt, __fsqrt_rn(rates.x)) > 0.1f || __fmul_rn(dt, rates.y) > 0.1f || __fmul_rn(dt, spin) > 0.01f ||
        motion > __fmul_rn(0.25f, c.skin) || __fmul_rn(rate.x, dt) > 0.01f || __fmul_rn(rate.y, dt) > 0.01f ||
        __fmul_rn(rate.z, dt) > 0.01f)
        fail(r, F_TIMESTEP);
}

// solver.slang:669-687: the planes advance along their normals by
// velocity . normal x dt (compensated offsets); with a boundary box, its six
// planes must keep a positive gap inside the domain.  One thread.
__device__ __forceinline__ void advanceWallPlanes(const Res& r, const Config& c) {
    for (uint32_t w = 0; w < c.wallCount; ++w) {
        float4 plane = r.wallPlane[w], residual = r.wallRemainder[w];
        float inc = __fmul_rn(dot(xyz(plane), xyz(r.wallVelocity[w])), c.dt);
        float y = __fadd_rn(inc, residual.w);
        float high = __fadd_rn(plane.w, y);
        float low = __fsub_rn(y, __fsub_rn(high, plane.w));
        plane.w = high;
        residual.w = low;
        if (!isfinite(high) || !isfinite(low)) { fail(r, F_NONFINITE); return; }
        r.wallPlane[w] = plane;
        r.wallRemainder[w] = residual;
    }
    if (c.wallBoxEnabled != 0) {
        float4 box = r.cell[0];
        for (uint32_t axis = 0; axis < 3; ++axis) {
            uint32_t lo = r.wallBoxIds[2 * axis], hi = r.wallBoxIds[2 * axis + 1];
            float low = __fadd_rn(r.wallPlane[lo].w, r.wallRemainder[lo].w);
            float high = -__fadd_rn(r.wallPlane[hi].w, r.wallRemainder[hi].w);
            float extent = axis == 0 ? box.x : axis == 1 ? box.y : box.z;
            if (low < 0 || high > extent || high <= low) fail(r, F_BOX);
        }
    }
}

}  // namespace sdg

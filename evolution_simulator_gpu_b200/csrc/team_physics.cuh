// The arithmetic of a substep's passes on values, for the team kernels
// (team.cuh), with every rounding written out.
//
// The creature kernel's passes (advance.cuh) are plain expressions, and the
// compiler chooses which of their products it fuses into a multiply-add. Most
// choices follow from the expression; in a sum of two products either may be
// fused, and which one it is depends on the code around. The team kernels'
// code around is another, so here each choice is written as the creature
// kernel's compiled passes make it, which was measured: of each sum's
// variants only one turns every substep's start state of trials (taken from
// the backward run's tapes) into the next one to the bit. A kernel that reads
// its world's switches at run time fuses three of them otherwise (W::fixed).
#pragma once
#include "advance.cuh"

namespace cek {

// Ground height and slope under x (shaders/creature.cu:166-226).
// `BACK`: as the backward run's contact fuses it.
template <bool BACK = false, class W>
__device__ __forceinline__ float2 ground_of(const W& w, float x, float amp, float qphase, const ce_params& p) {
    float height = 0.0f, slope = 0.0f;
    if (w.has(CE_FLAG_TERRAIN)) {
        const float t0 = __fmaf_rn(x, 1.0f / 1.1f, qphase);
        const float u0 = fracf(t0);
        const float w0 = __fmul_rn(u0, __fsub_rn(1.0f, u0));
        const float t1 = __fadd_rn(__fmaf_rn(x, 1.0f / 0.43f, 0.3f), qphase);
        const float u1 = fracf(t1);
        const float w1 = __fmul_rn(u1, __fsub_rn(1.0f, u1));
        const float bumps = sum2(__fmul_rn(0.65f * 16.0f, w0), w0, __fmul_rn(0.35f * 16.0f, w1), w1);
        const float rise = sum2(
            __fmul_rn(__fmul_rn(0.65f * 32.0f, w0), __fsub_rn(1.0f, __fmul_rn(2.0f, u0))), 1.0f / 1.1f,
            __fmul_rn(__fmul_rn(0.35f * 32.0f, w1), __fsub_rn(1.0f, __fmul_rn(2.0f, u1))), 1.0f / 0.43f);
        if (w.has(CE_FLAG_SLOPE)) {
            height = BACK ? sum2(amp, bumps, p.slope, x) : sum2(p.slope, x, amp, bumps);
            slope = W::fixed ? __fmaf_rn(amp, rise, p.slope) : __fadd_rn(__fmul_rn(amp, rise), p.slope);
        } else {
            height = __fmul_rn(amp, bumps);
            slope = __fmul_rn(amp, rise);
        }
    } else if (w.has(CE_FLAG_SLOPE)) {
        height = __fmul_rn(p.slope, x);
        slope = p.slope;
    }
    if (w.has(CE_FLAG_GAPS)) {
        const float spacing = __fmaf_rn(4.0f, p.gaps, 2.0f);
        const float center = __fmul_rn(spacing, 0.5f);
        const float r = __fmaf_rn(-floorf(x / spacing), spacing, x);
        const float distance = fabsf(__fsub_rn(r, center));
        const float half_w = __fmul_rn(0.5f, p.gaps);
        const float run = fmaxf(fminf(kGapRun, half_w), 1e-6f);
        float factor = clampf(__fsub_rn(half_w, distance) / run, 0.0f, 1.0f);
        if (distance <= __fsub_rn(half_w, run)) {
            factor = 1.0f;
        } else if (distance >= half_w) {
            factor = 0.0f;
        }
        height = __fmaf_rn(-kGapDepth, factor, height);
        if (distance > __fsub_rn(half_w, run) && distance < half_w) {
            slope = __fmaf_rn(-kGapDepth, (r < center ? 1.0f : -1.0f) / run, slope);
        }
    }
    if (w.has(CE_FLAG_HURDLES)) {
        const float spacing = kHurdleSpacing;
        const float center = spacing * 0.5f;
        const float r = __fmaf_rn(-floorf(x / spacing), spacing, x);
        const float distance = fabsf(__fsub_rn(r, center));
        const float half_w = 0.5f * kHurdleTop;
        const float run = kHurdleRun;
        float factor = clampf((half_w + run - distance) / run, 0.0f, 1.0f);
        if (distance <= half_w) {
            factor = 1.0f;
        } else if (distance >= half_w + run) {
            factor = 0.0f;
        }
        height = __fmaf_rn(p.hurdles, factor, height);
        if (distance > half_w && distance < half_w + run) {
            slope = __fmaf_rn(p.hurdles, (r < center ? 1.0f : -1.0f) / run, slope);
        }
    }
    return make_float2(height, slope);
}

// Ice at x (shaders/creature.cu:230-235).
__device__ __forceinline__ float ice_of(float x) {
    const float w = fracf(x * kIceInv);
    const float t = fabsf(w - 0.5f) * 2.0f;
    const float s = clampf(__fmul_rn(__fsub_rn(0.7f, t), 2.5f), 0.0f, 1.0f);
    return __fmul_rn(__fmul_rn(s, s), __fmaf_rn(-2.0f, s, 3.0f));
}

__device__ __forceinline__ float wrap_of(float a) {
    return __fmaf_rn(-kTauF, floorf(__fmul_rn(__fadd_rn(a, kPiF), 1.0f / kTauF)), a);
}

template <class W, int RATE>
struct Physics {
    using C = Clock<RATE>;
    const W& w;
    const ce_params& p;
    LaneRegs& r;

    // Joint j from its two lines and the positions of its parent bone's tip
    // and pivot and of its own bone's tip and hub
    // (shaders/creature.cu:322-356).
    struct Joint {
        unsigned tip, far, hub;
        float2 g_tip, g_far, g_hub;
        float w_tip, w_far, w_hub;
    };
    __device__ __forceinline__ static Joint joint_at(unsigned j, const float4& ra, const float4& rb, const float2& pt,
                                                     const float2& pp, const float2& ct, const float2& ch) {
        Joint k;
        const unsigned topo = __float_as_uint(ra.x);
        k.tip = j + 1u;
        k.hub = topo & 31u;
        k.far = (topo >> 15u) & 31u;
        const bool at_head = ((topo >> 20u) & 1u) != 0u;
        const float2 u = make_float2(pt.x - pp.x, pt.y - pp.y);
        const float2 v = make_float2(ct.x - ch.x, ct.y - ch.y);
        const float uu = fmaxf(sum2(u.x, u.x, u.y, u.y), 1e-12f);
        const float vv = fmaxf(sum2(v.x, v.x, v.y, v.y), 1e-12f);
        k.g_tip = make_float2(-v.y / vv, v.x / vv);
        const float2 g_u = make_float2(-u.y / uu, u.x / uu);
        k.g_far = at_head ? make_float2(-g_u.x, -g_u.y) : g_u;
        complete(k, rb);
        return k;
    }
    // The rest of a joint from the gradients of its tip and far nodes.
    __device__ __forceinline__ static void complete(Joint& k, const float4& rb) {
        k.w_tip = rb.x;
        k.w_far = rb.y;
        k.w_hub = rb.z;
        k.g_hub = make_float2(-(k.g_tip.x + k.g_far.x), -(k.g_tip.y + k.g_far.y));
    }
    __device__ __forceinline__ static float joint_weight(const Joint& k) {
        const float tip = sum2(k.g_tip.x, k.g_tip.x, k.g_tip.y, k.g_tip.y);
        const float far = sum2(k.g_far.x, k.g_far.x, k.g_far.y, k.g_far.y);
        const float hub = sum2(k.g_hub.x, k.g_hub.x, k.g_hub.y, k.g_hub.y);
        return __fmaf_rn(k.w_hub, hub, sum2(k.w_far, far, k.w_tip, tip));
    }
    // The joint's angle, the turn from its range's middle.
    __device__ __forceinline__ static float angle_at(const float4& ra, const float2& pt, const float2& pp,
                                                     const float2& ct, const float2& ch) {
        const float2 u = make_float2(pt.x - pp.x, pt.y - pp.y);
        const float2 v = make_float2(ct.x - ch.x, ct.y - ch.y);
        const float turn = atan2f(sum2(u.x, v.y, -u.y, v.x), sum2(u.x, v.x, u.y, v.y));
        return __fadd_rn(ra.w, wrap_of(__fsub_rn(turn, ra.w)));
    }
    // The damping's relative turning speed at joint k.
    __device__ __forceinline__ static float joint_rate(const Joint& k, const float2& vt, const float2& vf,
                                                       const float2& vh) {
        float s = sum2(k.g_tip.x, vt.x, k.g_tip.y, vt.y);
        s = __fmaf_rn(k.g_far.x, vf.x, s);
        s = __fmaf_rn(k.g_far.y, vf.y, s);
        s = __fmaf_rn(k.g_hub.x, vh.x, s);
        return __fmaf_rn(k.g_hub.y, vh.y, s);
    }

    // A muscle's demand for the step that starts at t_now
    // (shaders/creature.cu:442-451).
    __device__ __forceinline__ float demand_at(float t_now, const float4& r0, const float4& r1, float offset) const {
        const float before = rhythm(t_now, r0.y, r0.z, offset, r0.w, r1.x, r1.y);
        const float after = rhythm(t_now + C::dt, r0.y, r0.z, offset, r0.w, r1.x, r1.y);
        const float shortening = r0.x * (after - before) * C::rate;
        return r.limp ? 0.0f : fmaxf(shortening * r1.z * 0.25f, 0.0f);
    }

    // A muscle's pull between its anchors and the direction it acts in; its
    // energy store `ms.x` moves on (shaders/creature.cu:455-508).
    struct Pull {
        float fx, fy, pull, energy;
    };
    __device__ __forceinline__ Pull muscle_at(const float4& q0, const float4& q1, const float2& ms, const float4& A0,
                                              const float4& A1, const float4& B0, const float4& B1) const {
        const float anchor_a = q0.y, anchor_b = q0.z, hill = q0.w;
        const float cap = q1.x, inv_capacity = q1.y, tendon_k = q1.z, slack = q1.w;
        const auto between = [](float x, float y, float s) { return __fmaf_rn(__fsub_rn(y, x), s, x); };
        const float dx = between(B0.x, B1.x, anchor_b) - between(A0.x, A1.x, anchor_a);
        const float dy = between(B0.y, B1.y, anchor_b) - between(A0.y, A1.y, anchor_a);
        const float rvx = between(B0.z, B1.z, anchor_b) - between(A0.z, A1.z, anchor_a);
        const float rvy = between(B0.w, B1.w, anchor_b) - between(A0.w, A1.w, anchor_a);
        const float len = fmaxf(sqrtf(sum2(dx, dx, dy, dy)), 1e-6f);
        const float ex = dx / len, ey = dy / len;
        const float lengthening = sum2(rvx, ex, rvy, ey);
        float drive = __fmul_rn(ms.y, ms.x);
        if (hill > 0.0f) {
            drive = __fmul_rn(drive, clampf(__fmaf_rn(lengthening, hill, 1.0f), 0.0f, 1.0f));
        }
        const float active = clampf(__fmaf_rn(lengthening, 0.15f, drive), -cap, cap);
        const float work = __fmul_rn(__fmul_rn(fminf(drive, cap), fmaxf(-lengthening, 0.0f)), C::h);
        const float recovery = __fmul_rn(__fmul_rn(kMuscleRecovery, p.muscle_recovery), C::h);
        const float spent = __fmaf_rn(-__fmul_rn(work, inv_capacity), p.inv_muscle_energy, ms.x);
        Pull f;
        f.energy = clampf(__fmaf_rn(recovery, __fsub_rn(1.0f, ms.x), spent), 0.0f, 1.0f);
        f.pull = __fmaf_rn(tendon_k, fmaxf(len - slack, 0.0f), active);
        f.fx = __fmul_rn(ex, f.pull);
        f.fy = __fmul_rn(ey, f.pull);
        return f;
    }

    // The world's force on node i at `q` with velocity `u`
    // (shaders/creature.cu:511-546), added to the muscles' `pulls`.
    __device__ __forceinline__ float2 force_at(unsigned i, const float4& nr, const float2& q, const float2& u,
                                               const float2& pulls) const {
        const float m = nr.x;
        const bool drags = w.has(CE_FLAG_MUD) || w.has(CE_FLAG_BRAMBLES);
        float fx = 0.0f;
        if (w.has(CE_FLAG_WIND)) {
            fx = __fmul_rn(p.wind, m);
        }
        float dry = 0.0f;
        if (w.has(CE_FLAG_MUD) || w.has(CE_FLAG_BRAMBLES)) {
            const float2 g = ground_of(w, q.x, r.amp, r.qphase, p);
            dry = (q.y - g.x) / sqrtf(__fmaf_rn(g.y, g.y, 1.0f)) - nr.z;
        }
        if (w.has(CE_FLAG_MUD)) {
            const float sink = __fmul_rn(clampf(-dry, 0.0f, p.mud), 1.0f / kMudFullDepth);
            fx = __fmaf_rn(-__fmul_rn(__fmul_rn(m, kMudDrag), sink), u.x, fx);
        }
        if (w.has(CE_FLAG_BRAMBLES)) {
            if (((r.feet >> i) & 1u) == 0u && dry < kBrambleReach) {
                fx = __fmaf_rn(-__fmul_rn(m, p.brambles), u.x, fx);
            }
        }
        fx = __fadd_rn(fx, pulls.x);
        if (w.has(CE_FLAG_WATER)) {
            const float wet = clampf((p.water - (q.y - nr.z)) / (2.0f * nr.z), 0.0f, 1.0f);
            const float lift = __fmul_rn(__fmul_rn(kWaterBuoyancy, m), p.gravity);
            const float fy = __fmaf_rn(lift, wet, __fmul_rn(-p.gravity, m));
            return make_float2(fx, __fadd_rn(fy, pulls.y));
        }
        return make_float2(fx, W::fixed || !drags ? __fmaf_rn(-p.gravity, m, pulls.y) : __fadd_rn(__fmul_rn(-p.gravity, m), pulls.y));
    }

    // Velocity and predicted position of node i, `s` = (x, y, vx, vy), from
    // the world's force and the muscles' `pulls`.
    __device__ __forceinline__ void integrate_at(unsigned i, const float4& nr, const float2& pulls, float4& s) const {
        const float2 f = force_at(i, nr, make_float2(s.x, s.y), make_float2(s.z, s.w), pulls);
        s.z = __fmaf_rn(__fmul_rn(C::h, f.x), nr.y, s.z);
        s.w = __fmaf_rn(__fmul_rn(C::h, f.y), nr.y, s.w);
        if (w.has(CE_FLAG_AIR)) {
            s.z = __fmul_rn(s.z, p.air_sub);
            s.w = __fmul_rn(s.w, p.air_sub);
        }
        s.x = __fmaf_rn(C::h, s.z, s.x);
        s.y = __fmaf_rn(C::h, s.w, s.y);
    }

    // The part of a bone's water drag that its ends' positions and radii
    // give: its direction and the drag factor before the speed.
    struct Wet {
        float ax, ay, factor;
    };
    __device__ __forceinline__ Wet wet_at(const float4& ba, float r0, float r1, const float2& p0,
                                          const float2& p1) const {
        const float width = r0 + r1;
        const float wet0 = clampf((p.water - (p0.y - r0)) / (2.0f * r0), 0.0f, 1.0f);
        const float wet1 = clampf((p.water - (p1.y - r1)) / (2.0f * r1), 0.0f, 1.0f);
        const float wet = 0.5f * (wet0 + wet1);
        return Wet{(p1.x - p0.x) / ba.y, (p1.y - p0.y) / ba.y, kWaterDrag * wet * ba.y * width};
    }
    // Air and water drag on a bone (shaders/creature.cu:553-593), from its
    // line `bb` (air drag factor, drag limit, the two velocity scales), its
    // water drag `k` and its ends' velocities `v0`, `v1` (updated).
    __device__ __forceinline__ void drag_at(const float4& bb, const Wet& k, float2& v0, float2& v1) const {
        const float wx = 0.5f * (v0.x + v1.x), wy = 0.5f * (v0.y + v1.y);
        const float speed = sqrtf(sum2(wx, wx, wy, wy));
        const float limit = bb.y;
        const float k_air = fminf(__fmul_rn(bb.x, speed), limit);
        float dfx, dfy;
        if (w.has(CE_FLAG_WATER)) {
            const float along = sum2(wx, k.ax, wy, k.ay);
            const float lx = __fmul_rn(k.ax, along), ly = __fmul_rn(k.ay, along);
            const float sx = __fsub_rn(wx, lx), sy = __fsub_rn(wy, ly);
            const float k_water = fminf(__fmul_rn(k.factor, speed), limit);
            const float zx = sum2(sx, k_water, __fmul_rn(lx, k_water), kWaterAlong);
            const float zy = sum2(sy, k_water, __fmul_rn(ly, k_water), kWaterAlong);
            dfx = __fmaf_rn(-wx, k_air, -zx);
            dfy = __fmaf_rn(-wy, k_air, -zy);
        } else {
            dfx = __fmul_rn(-wx, k_air);
            dfy = __fmul_rn(-wy, k_air);
        }
        const float s0 = bb.z, s1 = bb.w;
        v0 = make_float2(__fmaf_rn(s0, dfx, v0.x), __fmaf_rn(s0, dfy, v0.y));
        v1 = make_float2(__fmaf_rn(s1, dfx, v1.x), __fmaf_rn(s1, dfy, v1.y));
    }

    // Length of a bone (shaders/creature.cu:597-613).
    __device__ __forceinline__ static void bone_at(const float4& ba, float2& p0, float2& p1) {
        const float dx = p1.x - p0.x, dy = p1.y - p0.y;
        const float len = fmaxf(sqrtf(sum2(dx, dx, dy, dy)), 1e-9f);
        const float w0 = ba.z, w1 = ba.w;
        const float s = __fsub_rn(len, ba.y) / __fmul_rn(__fadd_rn(w0, w1), len);
        const float s0 = __fmul_rn(w0, s), s1 = -__fmul_rn(w1, s);
        p0 = make_float2(__fmaf_rn(s0, dx, p0.x), __fmaf_rn(s0, dy, p0.y));
        p1 = make_float2(__fmaf_rn(s1, dx, p1.x), __fmaf_rn(s1, dy, p1.y));
    }

    // Ground contact and friction of a node (shaders/creature.cu:640-679).
    // `q` is the node's position (moved when it touches) and `f0` its
    // position at the start of the substep. Returns whether it touches, the
    // push out of the ground and back along it (a recording's forces), and
    // whether it slid.
    __device__ __forceinline__ bool ground_at(const float4& nr, float2& q, const float2& f0, float& depth, float& back,
                                              bool& slid) const {
        if (!w.has(CE_FLAG_GROUND)) {
            return false;
        }
        const float2 g = ground_of(w, q.x, r.amp, r.qphase, p);
        const float secant = sqrtf(__fmaf_rn(g.y, g.y, 1.0f));
        const float nx = -g.y / secant, ny = 1.0f / secant;
        const float dry = (q.y - g.x) / secant - nr.z;
        float mu = __fmul_rn(nr.w, p.friction);
        if (w.has(CE_FLAG_MUD)) {
            depth = -__fadd_rn(dry, p.mud);
            const float sink = __fmul_rn(clampf(-dry, 0.0f, p.mud), 1.0f / kMudFullDepth);
            mu = __fmul_rn(__fmul_rn(mu, __fmaf_rn(kMudGrip, sink, 1.0f)), __fmaf_rn(kMudNormal, sink, 1.0f));
        } else {
            depth = -dry;
        }
        if (depth <= 0.0f) {
            return false;
        }
        if (w.has(CE_FLAG_ICE)) {
            mu = __fmul_rn(mu, __fmaf_rn(-p.patches, ice_of(q.x), 1.0f));
        }
        q.x = __fmaf_rn(nx, depth, q.x);
        q.y = __fmaf_rn(ny, depth, q.y);
        const float tx = ny, ty = -nx;
        const float slide = sum2(q.x - f0.x, tx, q.y - f0.y, ty);
        const float budget = __fmul_rn(mu, depth);
        slid = !(fabsf(slide) <= budget);
        back = slid ? copysignf(budget, slide) : slide;
        q.x = __fmaf_rn(-tx, back, q.x);
        q.y = __fmaf_rn(-ty, back, q.y);
        return true;
    }
};

}  // namespace cek

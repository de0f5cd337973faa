// The terms of a substep's reverse (adjoint.cu) on values, for the team
// kernel's backward run (team_adjoint.cu): the adjoint of each pass's item
// from the values that the item saw and the adjoints of what it gave.
//
// As in team_physics.cuh every rounding is written out, as the compiled
// backward run of one creature a lane makes it, so that both runs' gradients
// are the same to the bit. Of each sum's variants the one here is the only
// one with which no gradient of 13,500 trials differs (short trials in the
// air, on the ground and in water, with weak muscles and with ones strong
// enough for the smallest terms to show).
#pragma once
#include "team_physics.cuh"

namespace cek {

// d slope / d x of the ground under x: the terrain's second derivative (the
// slope, gap and hurdle terms are linear in x between their kinks).
template <class W>
__device__ __forceinline__ float ground_curvature(const W& w, float x, float amp, float qphase) {
    if (!w.has(CE_FLAG_TERRAIN)) {
        return 0.0f;
    }
    const float u0 = fracf(x * (1.0f / 1.1f) + qphase);
    const float u1 = fracf(x * (1.0f / 0.43f) + 0.3f + qphase);
    const float c0 = sum2(1.0f - 2.0f * u0, 1.0f - 2.0f * u0, -2.0f * u0, 1.0f - u0);
    const float c1 = sum2(1.0f - 2.0f * u1, 1.0f - 2.0f * u1, -2.0f * u1, 1.0f - u1);
    return __fmul_rn(amp, sum2(__fmul_rn(0.65f * 32.0f, c0), 1.0f / (1.1f * 1.1f), __fmul_rn(0.35f * 32.0f, c1), 1.0f / (0.43f * 0.43f)));
}

// d ice_at / d x (the smoothstep of ice_at; 0 outside its ramps).
__device__ __forceinline__ float ice_slope(float x) {
    const float w = fracf(x * kIceInv);
    const float t = fabsf(w - 0.5f) * 2.0f;
    const float z = (0.7f - t) * 2.5f;
    if (z < 0.0f || z > 1.0f) {
        return 0.0f;
    }
    const float dt = (w - 0.5f < 0.0f ? -2.0f : 2.0f) * kIceInv;
    return 6.0f * z * (1.0f - z) * -2.5f * dt;
}

// w -> perp(w) / |w|^2: its adjoint `lg` into w's (Backward::perp_back). The
// damping's and the range test's copies fuse one sum each its own way.
template <bool DAMPING>
__device__ __forceinline__ void perp_term(float2 w, float ww, float2 gw, float2 lg, float2& lw) {
    lw.x += lg.y / ww;
    lw.y += -lg.x / ww;
    if (ww >= 1e-12f && sum2(w.x, w.x, w.y, w.y) >= 1e-12f) {
        const float c =
            2.0f * (DAMPING ? sum2(lg.y, gw.y, lg.x, gw.x) : sum2(lg.x, gw.x, lg.y, gw.y)) / ww;
        lw.x = __fmaf_rn(-c, w.x, lw.x);
        lw.y = __fmaf_rn(-c, w.y, lw.y);
    }
}

// The adjoints of a joint's gradient vectors (lgt, lgf) and angle (lturn, 0
// for damping) into those of the parent bone (lu) and its own (lv).
template <bool DAMPING>
__device__ __forceinline__ void joint_geometry_back(float2 pt, float2 pp, float2 ct, float2 ch, bool at_head, float2 lgt,
                                                    float2 lgf, float lturn, float2& lu, float2& lv) {
    const float2 u = make_float2(pt.x - pp.x, pt.y - pp.y);
    const float2 v = make_float2(ct.x - ch.x, ct.y - ch.y);
    const float uu = fmaxf(sum2(u.x, u.x, u.y, u.y), 1e-12f), vv = fmaxf(sum2(v.x, v.x, v.y, v.y), 1e-12f);
    const float2 g_tip = make_float2(-v.y / vv, v.x / vv);
    const float2 g_u = make_float2(-u.y / uu, u.x / uu);
    const float2 lgu = at_head ? make_float2(-lgf.x, -lgf.y) : lgf;
    lu = make_float2(0.0f, 0.0f);
    lv = make_float2(0.0f, 0.0f);
    perp_term<DAMPING>(v, vv, g_tip, lgt, lv);
    perp_term<DAMPING>(u, uu, g_u, lgu, lu);
    if (!DAMPING && lturn != 0.0f) {
        const float cr = sum2(u.x, v.y, -u.y, v.x), dt = sum2(u.x, v.x, u.y, v.y);
        const float den = sum2(cr, cr, dt, dt);
        if (den > 0.0f) {
            const float lc = lturn * dt / den, ld = -lturn * cr / den;
            lu.x += sum2(lc, v.y, ld, v.x);
            lu.y += sum2(ld, v.y, -lc, v.x);
            lv.x += sum2(ld, u.x, -lc, u.y);
            lv.y += sum2(lc, u.x, ld, u.y);
        }
    }
}

// The shares of a push's three gradient vectors: lgt and lgf with lgh folded
// in (g_hub = -(g_tip + g_far)).
template <class K>
__device__ __forceinline__ void damping_back(const K& k, float wgt, float share, float2 vt, float2 vf, float2 vh,
                                             float2 at, float2 af, float2 ah, float& lam, float& lrate, float& lwgt,
                                             float2& lgt, float2& lgf) {
    float rate = sum2(k.g_tip.x, vt.x, k.g_tip.y, vt.y);
    rate = __fmaf_rn(k.g_far.x, vf.x, rate);
    rate = __fmaf_rn(k.g_far.y, vf.y, rate);
    rate = __fmaf_rn(k.g_hub.x, vh.x, rate);
    rate = __fmaf_rn(k.g_hub.y, vh.y, rate);
    lam = __fmul_rn(-share, rate) / wgt;
    const float lt = sum2(k.g_tip.x, at.x, k.g_tip.y, at.y), lf = sum2(k.g_far.x, af.x, k.g_far.y, af.y),
                lh = sum2(k.g_hub.y, ah.y, k.g_hub.x, ah.x);
    const float llam = __fmaf_rn(k.w_hub, lh, sum2(k.w_tip, lt, k.w_far, lf));
    lrate = __fmul_rn(-share, llam) / wgt;
    lwgt = __fmul_rn(__fmul_rn(llam, share), rate) / __fmul_rn(wgt, wgt);
    const auto share_of = [&](float w, float g, float a, float v) {
        return __fmaf_rn(__fmul_rn(__fmul_rn(2.0f, w), g), lwgt, sum2(__fmul_rn(w, lam), a, lrate, v));
    };
    lgt = make_float2(share_of(k.w_tip, k.g_tip.x, at.x, vt.x), share_of(k.w_tip, k.g_tip.y, at.y, vt.y));
    lgf = make_float2(share_of(k.w_far, k.g_far.x, af.x, vf.x), share_of(k.w_far, k.g_far.y, af.y, vf.y));
    const float2 lgh = make_float2(share_of(k.w_hub, k.g_hub.x, ah.x, vh.x), share_of(k.w_hub, k.g_hub.y, ah.y, vh.y));
    lgt.x -= lgh.x;
    lgt.y -= lgh.y;
    lgf.x -= lgh.x;
    lgf.y -= lgh.y;
}

// A joint-limit push from the positions its test saw (Backward::
// joint_limit_back).
__device__ __forceinline__ void limit_back(const float4& ra, const float4& rb, float2 pt, float2 pp, float2 ct,
                                           float2 ch, float2 at, float2 af, float2 ah, float& lam, float& lerr,
                                           float& lwgt, float2& lgt, float2& lgf, float2& g_tip, float2& g_far,
                                           float2& g_hub) {
    const bool at_head = ((__float_as_uint(ra.x) >> 20u) & 1u) != 0u;
    const float2 u = make_float2(pt.x - pp.x, pt.y - pp.y);
    const float2 v = make_float2(ct.x - ch.x, ct.y - ch.y);
    const float uu = fmaxf(sum2(u.x, u.x, u.y, u.y), 1e-12f), vv = fmaxf(sum2(v.x, v.x, v.y, v.y), 1e-12f);
    const float turn = atan2f(sum2(u.x, v.y, -u.y, v.x), sum2(u.x, v.x, u.y, v.y));
    const float mid = ra.w;
    const float angle = __fadd_rn(mid, wrap_of(__fsub_rn(turn, mid)));
    const float lo = ra.y, hi = ra.z;
    float error = 0.0f;
    if (angle < lo) {
        error = angle - lo;
    }
    if (angle > hi) {
        error = angle - hi;
    }
    g_tip = make_float2(-v.y / vv, v.x / vv);
    const float2 g_u = make_float2(-u.y / uu, u.x / uu);
    g_far = at_head ? make_float2(-g_u.x, -g_u.y) : g_u;
    g_hub = make_float2(-(g_tip.x + g_far.x), -(g_tip.y + g_far.y));
    const float w_tip = rb.x, w_far = rb.y, w_hub = rb.z;
    const float wt = sum2(g_tip.x, g_tip.x, g_tip.y, g_tip.y), wf = sum2(g_far.x, g_far.x, g_far.y, g_far.y),
                wh = sum2(g_hub.x, g_hub.x, g_hub.y, g_hub.y);
    const float wgt = __fmaf_rn(w_hub, wh, sum2(w_far, wf, w_tip, wt));
    lam = -error / wgt;
    const float lt = sum2(g_tip.x, at.x, g_tip.y, at.y), lf = sum2(g_far.x, af.x, g_far.y, af.y),
                lh = sum2(g_hub.y, ah.y, g_hub.x, ah.x);
    const float llam = __fmaf_rn(w_hub, lh, sum2(w_tip, lt, w_far, lf));
    lerr = -llam / wgt;
    lwgt = __fmul_rn(llam, error) / __fmul_rn(wgt, wgt);
    const auto share_of = [&](float w, float g, float a) {
        return sum2(__fmul_rn(w, lam), a, __fmul_rn(__fmul_rn(2.0f, w), g), lwgt);
    };
    lgt = make_float2(share_of(w_tip, g_tip.x, at.x), share_of(w_tip, g_tip.y, at.y));
    lgf = make_float2(share_of(w_far, g_far.x, af.x), share_of(w_far, g_far.y, af.y));
    const float2 lgh = make_float2(share_of(w_hub, g_hub.x, ah.x), share_of(w_hub, g_hub.y, ah.y));
    lgt.x -= lgh.x;
    lgt.y -= lgh.y;
    lgf.x -= lgh.x;
    lgf.y -= lgh.y;
}

// A bone's length: the adjoints of its ends (updated) and of their inverse
// masses (d0, d1), from the positions `pre` that its projection saw.
__device__ __forceinline__ void bone_length_back(const float4& ba, const float4& pre, float2& l0, float2& l1,
                                                 float& d0, float& d1) {
    const float dx = pre.z - pre.x, dy = pre.w - pre.y;
    const float len0 = sqrtf(sum2(dx, dx, dy, dy));
    const float len = fmaxf(len0, 1e-9f);
    const float w0 = ba.z, w1 = ba.w;
    const float sc = __fsub_rn(len, ba.y) / __fmul_rn(__fadd_rn(w0, w1), len);
    const float along0 = sum2(dx, l0.x, dy, l0.y), along1 = sum2(dx, l1.x, dy, l1.y);
    const float ls = sum2(w0, along0, -w1, along1);
    const float s0 = __fmul_rn(w0, sc), s1 = __fmul_rn(w1, sc);
    float ldx = sum2(s0, l0.x, -s1, l1.x), ldy = sum2(s0, l0.y, -s1, l1.y);
    if (len0 >= 1e-9f) {
        const float llen = __fmul_rn(ls, ba.y) / __fmul_rn(__fmul_rn(__fadd_rn(w0, w1), len), len);
        ldx = add_over(ldx, __fmul_rn(llen, dx), len);
        ldy = add_over(ldy, __fmul_rn(llen, dy), len);
    }
    const float lsw = __fmul_rn(-ls, sc) / __fadd_rn(w0, w1);
    d0 = __fmaf_rn(sc, sum2(dx, l0.x, dy, l0.y), lsw);
    d1 = __fmaf_rn(-sc, sum2(dx, l1.x, dy, l1.y), lsw);
    l0 = make_float2(l0.x - ldx, l0.y - ldy);
    l1 = make_float2(l1.x + ldx, l1.y + ldy);
}

// A node's integration (y0 its start height, F the muscles' force): the
// adjoints of its start position, velocity and force, and its mass's share.
template <class C, class W>
__device__ __forceinline__ void integrate_back(const W& w, const ce_params& p, const float4& nr, float2 F, float y0,
                                               float2 lq1, float2 lq0, float2& lp, float2& lv1, float2& lf,
                                               float& dm) {
    const float im = nr.y;
    lp = make_float2(lq1.x + lq0.x, lq1.y + lq0.y);
    lv1 = make_float2(C::h * lq1.x, C::h * lq1.y);
    if (w.has(CE_FLAG_AIR)) {
        lv1.x *= p.air_sub;
        lv1.y *= p.air_sub;
    }
    if (w.has(CE_FLAG_WATER)) {
        const float z = (p.water - (y0 - nr.z)) / (2.0f * nr.z);
        if (z >= 0.0f && z <= 1.0f) {
            const float lift = __fmul_rn(
                __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(lv1.y, C::h), im), kWaterBuoyancy), nr.x), p.gravity);
            lp.y = add_over(lp.y, -lift, 2.0f * nr.z);
        }
    }
    lf = make_float2(__fmul_rn(__fmul_rn(lv1.x, C::h), im), __fmul_rn(__fmul_rn(lv1.y, C::h), im));
    dm = sum2(lv1.x, F.x, lv1.y, F.y);
}

// A bone's drag from the velocities `pre` that it saw: the adjoints of its
// ends' velocities (l0, l1) and, in water, positions (e0, e1; p0, p1 the start
// positions, r0, r1 the radii), of its drag limit, and of the inverse masses.
template <class C, class W>
__device__ __forceinline__ void bone_drag_back(const W& w, const ce_params& p, const float4& ba, const float4& bb,
                                               const float4& pre, float r0, float r1, float2 p0, float2 p1,
                                               float2& l0, float2& l1, float2& e0, float2& e1, float& llimit,
                                               float& d0, float& d1) {
    const float wx = 0.5f * (pre.x + pre.z), wy = 0.5f * (pre.y + pre.w);
    const float speed = sqrtf(sum2(wx, wx, wy, wy));
    const float limit = bb.y;
    const float k_air = fminf(__fmul_rn(bb.x, speed), limit);
    const float ldx = sum2(bb.z, l0.x, bb.w, l1.x), ldy = sum2(bb.z, l0.y, bb.w, l1.y);
    float lwx, lwy, dfx, dfy;
    const float lk = -sum2(wx, ldx, wy, ldy);
    float lspeed = 0.0f;
    llimit = 0.0f;
    if (__fmul_rn(bb.x, speed) <= limit) {
        lspeed = __fmul_rn(lk, bb.x);
    } else {
        llimit = lk;
    }
    if (w.has(CE_FLAG_WATER)) {
        const float width = r0 + r1;
        const float z0 = (p.water - (p0.y - r0)) / (2.0f * r0);
        const float z1 = (p.water - (p1.y - r1)) / (2.0f * r1);
        const float wet = 0.5f * (clampf(z0, 0.0f, 1.0f) + clampf(z1, 0.0f, 1.0f));
        const float ax = (p1.x - p0.x) / ba.y, ay = (p1.y - p0.y) / ba.y;
        const float along = sum2(wx, ax, wy, ay);
        const float lx = __fmul_rn(ax, along), ly = __fmul_rn(ay, along);
        const float sx = __fsub_rn(wx, lx), sy = __fsub_rn(wy, ly);
        const float kw = __fmul_rn(__fmul_rn(__fmul_rn(kWaterDrag, wet), ba.y), width);
        const float xw = __fmul_rn(kw, speed);
        const float k_water = fminf(xw, limit);
        const float zx = sum2(sx, k_water, __fmul_rn(lx, k_water), kWaterAlong);
        const float zy = sum2(sy, k_water, __fmul_rn(ly, k_water), kWaterAlong);
        dfx = __fmaf_rn(-wx, k_air, -zx);
        dfy = __fmaf_rn(-wy, k_air, -zy);
        const float lkw = __fmaf_rn(-kWaterAlong, sum2(lx, ldx, ly, ldy), -sum2(sx, ldx, sy, ldy));
        const float llx = sum2(__fmul_rn(-k_water, kWaterAlong), ldx, k_water, ldx);
        const float lly = sum2(__fmul_rn(-k_water, kWaterAlong), ldy, k_water, ldy);
        lwx = sum2(-k_air, ldx, -k_water, ldx);
        lwy = sum2(-k_air, ldy, -k_water, ldy);
        const float lalong = sum2(llx, ax, lly, ay);
        lwx = __fmaf_rn(lalong, ax, lwx);
        lwy = __fmaf_rn(lalong, ay, lwy);
        const float lax = sum2(llx, along, lalong, wx), lay = sum2(lly, along, lalong, wy);
        float lwet = 0.0f;
        if (xw <= limit) {
            lwet = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(lkw, kWaterDrag), ba.y), width), speed);
            lspeed = __fmaf_rn(__fmul_rn(__fmul_rn(__fmul_rn(lkw, kWaterDrag), wet), ba.y), width, lspeed);
        } else {
            llimit += lkw;
        }
        e0.x = __fadd_rn(e0.x, -lax / ba.y);
        e0.y = __fadd_rn(e0.y, -lay / ba.y);
        if (z0 >= 0.0f && z0 <= 1.0f) {
            e0.y = add_over(e0.y, -0.5f * lwet, 2.0f * r0);
        }
        e1.x = __fadd_rn(e1.x, lax / ba.y);
        e1.y = __fadd_rn(e1.y, lay / ba.y);
        if (z1 >= 0.0f && z1 <= 1.0f) {
            e1.y = add_over(e1.y, -0.5f * lwet, 2.0f * r1);
        }
    } else {
        lwx = __fmul_rn(-k_air, ldx);
        lwy = __fmul_rn(-k_air, ldy);
        dfx = __fmul_rn(-wx, k_air);
        dfy = __fmul_rn(-wy, k_air);
    }
    if (speed > 0.0f) {
        lwx = add_over(lwx, __fmul_rn(lspeed, wx), speed);
        lwy = add_over(lwy, __fmul_rn(lspeed, wy), speed);
    }
    d0 = __fmul_rn(0.5f * C::h, sum2(l0.x, dfx, l0.y, dfy));
    d1 = __fmul_rn(0.5f * C::h, sum2(l1.x, dfx, l1.y, dfy));
    l0 = make_float2(l0.x + 0.5f * lwx, l0.y + 0.5f * lwy);
    l1 = make_float2(l1.x + 0.5f * lwx, l1.y + 0.5f * lwy);
}

// A node's contact from its position `q` before it and the substep's start
// position `f0`: the adjoint of its position (lq, of the result on entry), the
// start position's share (lf) and the friction's.
template <class W>
__device__ __forceinline__ void contact_back(const W& w, const ce_params& p, float amp, float qphase, const float4& nr,
                                             float2 q, float2 f0, bool slipped, float2& lq_io, float2& lf,
                                             float& fric) {
    const float2 gr = ground_of<true>(w, q.x, amp, qphase, p);
    const float sec = sqrtf(__fmaf_rn(gr.y, gr.y, 1.0f));
    const float nx = -gr.y / sec, ny = 1.0f / sec;
    const float dry = (q.y - gr.x) / sec - nr.z;
    const float depth = -dry;
    float mu = __fmul_rn(nr.w, p.friction), ice = 1.0f;
    if (w.has(CE_FLAG_ICE)) {
        ice = __fmaf_rn(-p.patches, ice_of(q.x), 1.0f);
        mu = __fmul_rn(mu, ice);
    }
    const float2 q1 = make_float2(__fmaf_rn(nx, depth, q.x), __fmaf_rn(ny, depth, q.y));
    const float tx = ny, ty = -nx;
    const float slide = sum2(q1.x - f0.x, tx, q1.y - f0.y, ty);
    const float S = gr.y;
    const float budget = __fmul_rn(mu, depth);
    const float back = slipped ? copysignf(budget, slide) : slide;
    const float2 l2 = lq_io;
    const float lback = -sum2(l2.x, tx, l2.y, ty);
    float lpush = 0.0f, lmu = 0.0f, lslide = 0.0f;
    if (slipped) {
        const float lbudget = slide < 0.0f ? -lback : lback;
        lmu = __fmul_rn(lbudget, depth);
        lpush = lbudget;
    } else {
        lslide = lback;
    }
    const float2 lq1 = make_float2(__fmaf_rn(lslide, tx, l2.x), __fmaf_rn(lslide, ty, l2.y));
    lf.x = __fmaf_rn(-lslide, tx, lf.x);
    lf.y = __fmaf_rn(-lslide, ty, lf.y);
    const float ltx = sum2(lslide, q1.x - f0.x, -back, l2.x), lty = sum2(lslide, q1.y - f0.y, -back, l2.y);
    const float lnx = __fmaf_rn(lq1.x, depth, -lty), lny = __fmaf_rn(lq1.y, depth, ltx);
    const float lout = sum2(lq1.x, nx, lq1.y, ny);
    const float ldepth = slipped ? __fadd_rn(__fmul_rn(lpush, mu), lout) : lout;
    float2 lq = lq1;
    float lx = 0.0f;
    if (lmu != 0.0f) {
        fric = w.has(CE_FLAG_ICE) ? __fmaf_rn(__fmul_rn(lmu, p.friction), ice, fric) : __fmaf_rn(lmu, p.friction, fric);
        if (w.has(CE_FLAG_ICE)) {
            lx = -__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(lmu, nr.w), p.friction), p.patches), ice_slope(q.x));
        }
    }
    lq.y = __fadd_rn(lq.y, -ldepth / sec);
    const float lheight = ldepth / sec;
    const float sec2 = __fmul_rn(sec, sec);
    const float lsec = add_over(__fmaf_rn(lnx, S, -lny) / sec2, __fmul_rn(ldepth, q.y - gr.x), sec2);
    const float lslope = add_over(-lnx / sec, __fmul_rn(lsec, S), sec);
    lx += sum2(lheight, S, lslope, ground_curvature(w, q.x, amp, qphase));
    lq.x += lx;
    lq_io = lq;
}

// A muscle's pass: the adjoints of its anchors' distance (ld) and relative
// speed (lrv), energy store and demand, and of its record fields.
struct MuscleBack {
    float ldx, ldy, lrvx, lrvy, le, ld, hill, cap, icap;
};
template <class C>
__device__ __forceinline__ void muscle_back(const ce_params& p, const float4& q0, const float4& q1, const float2& ms,
                                            const float4& A0, const float4& A1, const float4& B0, const float4& B1,
                                            const float2& fa0, const float2& fa1, const float2& fb0,
                                            const float2& fb1, const float2& lm, MuscleBack& out) {
    const float c = kMuscleRecovery * p.muscle_recovery * C::h;
    const float anchor_a = q0.y, anchor_b = q0.z, hill = q0.w;
    const float cap = q1.x, inv_capacity = q1.y, tendon_k = q1.z, slack = q1.w;
    const auto between = [](float u, float v, float s) { return __fmaf_rn(__fsub_rn(v, u), s, u); };
    const float dx = between(B0.x, B1.x, anchor_b) - between(A0.x, A1.x, anchor_a);
    const float dy = between(B0.y, B1.y, anchor_b) - between(A0.y, A1.y, anchor_a);
    const float rvx = between(B0.z, B1.z, anchor_b) - between(A0.z, A1.z, anchor_a);
    const float rvy = between(B0.w, B1.w, anchor_b) - between(A0.w, A1.w, anchor_a);
    const float len0 = sqrtf(sum2(dx, dx, dy, dy));
    const float len = fmaxf(len0, 1e-6f);
    const float ex = dx / len, ey = dy / len;
    const float lengthening = sum2(rvx, ex, rvy, ey);
    const float drive0 = __fmul_rn(ms.y, ms.x);
    float drive = drive0, hc = 1.0f, hz = 0.0f;
    if (hill > 0.0f) {
        hz = __fmaf_rn(lengthening, hill, 1.0f);
        hc = clampf(hz, 0.0f, 1.0f);
        drive = __fmul_rn(drive0, hc);
    }
    const float ya = __fmaf_rn(lengthening, 0.15f, drive);
    const float active = clampf(ya, -cap, cap);
    const float m1 = fminf(drive, cap), m2 = fmaxf(-lengthening, 0.0f);
    const float work = __fmul_rn(__fmul_rn(m1, m2), C::h);
    const float z = __fmaf_rn(c, __fsub_rn(1.0f, ms.x), __fmaf_rn(-__fmul_rn(work, inv_capacity), p.inv_muscle_energy, ms.x));
    const float pull = __fmaf_rn(tendon_k, fmaxf(len - slack, 0.0f), active);
    const auto pulled = [&](float f0, float f1, float f2, float f3) {
        return __fmaf_rn(-anchor_b, f3, __fmaf_rn(-(1.0f - anchor_b), f2, sum2(1.0f - anchor_a, f0, anchor_a, f1)));
    };
    const float lfx = pulled(fa0.x, fa1.x, fb0.x, fb1.x), lfy = pulled(fa0.y, fa1.y, fb0.y, fb1.y);
    const float lpull = sum2(lfx, ex, lfy, ey);
    const float lz = (z >= 0.0f && z <= 1.0f) ? lm.x : 0.0f;
    const float lwork = __fmul_rn(__fmul_rn(-lz, inv_capacity), p.inv_muscle_energy);
    out.icap = __fmul_rn(-lz, work);
    float g_cap = 0.0f, g_hill = 0.0f;
    float ldrive = 0.0f, llg = 0.0f, llen = 0.0f;
    const float lm1 = __fmul_rn(__fmul_rn(lwork, m2), C::h), lm2 = __fmul_rn(__fmul_rn(lwork, m1), C::h);
    if (drive <= cap) {
        ldrive = lm1;
    } else {
        g_cap = lm1;
    }
    if (-lengthening >= 0.0f) {
        llg = -lm2;
    }
    if (len - slack >= 0.0f) {
        llen = __fmul_rn(lpull, tendon_k);
    }
    if (ya >= -cap && ya <= cap) {
        ldrive = __fadd_rn(ldrive, lpull);
        llg = __fmaf_rn(0.15f, lpull, llg);
    } else if (ya > cap) {
        g_cap = __fadd_rn(g_cap, lpull);
    } else {
        g_cap = __fsub_rn(g_cap, lpull);
    }
    float ldrive0 = ldrive;
    if (hill > 0.0f) {
        ldrive0 = __fmul_rn(ldrive, hc);
        if (hz >= 0.0f && hz <= 1.0f) {
            const float lhc = __fmul_rn(ldrive, drive0);
            llg = __fmaf_rn(lhc, hill, llg);
            g_hill = __fmul_rn(lhc, lengthening);
        }
    }
    out.ld = __fadd_rn(__fmul_rn(ldrive0, ms.x), lm.y);
    out.lrvx = __fmul_rn(llg, ex);
    out.lrvy = __fmul_rn(llg, ey);
    const float lex = sum2(llg, rvx, lfx, pull), ley = sum2(llg, rvy, lfy, pull);
    float ldx = lex / len, ldy = ley / len;
    llen = add_over(llen, -sum2(lex, ex, ley, ey), len);
    if (len0 >= 1e-6f) {
        ldx = add_over(ldx, __fmul_rn(llen, dx), len);
        ldy = add_over(ldy, __fmul_rn(llen, dy), len);
    }
    out.ldx = ldx;
    out.ldy = ldy;
    out.le = sum2(ldrive0, ms.y, lz, 1.0f - c);
    out.hill = g_hill;
    out.cap = g_cap;
}

// d rhythm(t) into (phase, duty, 1/duty, 1/(1-duty)) times `lr`.
__device__ __forceinline__ void rhythm_term(float t, const float4& r0, const float4& r1, float offset, float lr,
                                            float4& g1) {
    const float ph = fracf(t * r0.y + r0.z + offset);
    const float duty = r0.w, inv_duty = r1.x, inv_comp = r1.y;
    if (ph < duty) {
        const float sn = __sinf(kPiF * ph * inv_duty);
        g1.x = __fadd_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(lr, 0.5f), kPiF), inv_duty), sn), g1.x);
        g1.z = __fmaf_rn(__fmul_rn(__fmul_rn(__fmul_rn(lr, 0.5f), kPiF), ph), sn, g1.z);
    } else {
        const float sn = __sinf(kPiF * (ph - duty) * inv_comp);
        const float x = __fmul_rn(__fmul_rn(lr, 0.5f), kPiF);
        const float y = __fmul_rn(__fmul_rn(x, inv_comp), sn);
        g1.x = __fsub_rn(g1.x, y);
        g1.y = __fadd_rn(g1.y, y);
        g1.w = __fmaf_rn(-__fmul_rn(x, ph - duty), sn, g1.w);
    }
}

// A muscle's demand: its adjoint `ld` into the muscle's gradient (kGradMuscle
// floats).
template <class C>
__device__ __forceinline__ void demand_back(float t_now, const float4& r0, const float4& r1, float offset, bool limp,
                                            float ld, float* g) {
    const float before = rhythm(t_now, r0.y, r0.z, offset, r0.w, r1.x, r1.y);
    const float after = rhythm(t_now + C::dt, r0.y, r0.z, offset, r0.w, r1.x, r1.y);
    const float shortening = r0.x * (after - before) * C::rate;
    const float xd = shortening * r1.z * 0.25f;
    if (limp || xd < 0.0f || ld == 0.0f) {
        return;
    }
    const float lsh = __fmul_rn(__fmul_rn(ld, r1.z), 0.25f);
    const float lr = __fmul_rn(__fmul_rn(lsh, r0.x), C::rate);
    float4 g1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    rhythm_term(t_now + C::dt, r0, r1, offset, lr, g1);
    rhythm_term(t_now, r0, r1, offset, -lr, g1);
    g[0] = __fmaf_rn(__fmul_rn(lsh, after - before), C::rate, g[0]);
    g[4] += g1.x;
    g[5] += g1.y;
    g[6] += g1.z;
    g[7] += g1.w;
    g[8] = __fmaf_rn(__fmul_rn(ld, shortening), 0.25f, g[8]);
}

}  // namespace cek

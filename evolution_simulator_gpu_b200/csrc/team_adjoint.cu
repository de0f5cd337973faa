// The backward run on teams of lanes: the adjoint of adjoint.cu, whose
// account of the method stands for this one too, with the team kernels'
// mapping (team.cuh).
//
// The reverse of a substep takes the passes backwards and in each pass the
// items from last to first. Lane i reverses node i, the bone that ends there
// and that bone's joint; the items of a pass run in levels from the end (an
// item goes when every later item at its nodes has), the muscles go round the
// lanes and each node's lane adds up its own in the muscles' order. What the
// reverse reads of a substep (the values that each pass saw, the contact)
// goes to the segment's tape as the rerun meets it, 9 float4 a lane, and is
// fetched a substep ahead; every sum has the order of the serial reverse.
//
// Bound by the chain of a creature's dependent operations where the launch
// leaves schedulers idle, and by instruction issue above; the tape's 300 B a
// lane and substep are under a tenth of the memory's rate. Running each
// substep again before its reverse, with those values in registers, moves 32 B
// instead and took 92 ms against 68 at 1,021 creatures of the refined search's
// world x 4 s, 152 / 110 ms at 8,192 and 144 / 107 ms at 16,384 calm ones x 2 s
// (on lanes: 269, 366 and 188 ms). 4 blocks of 64 threads an SM have 255
// registers; 5 and 6 (168, with spills) took 79 ms.
#include <cuda_runtime.h>

#include <type_traits>

#include "adjoint_terms.cuh"
#include "team.cuh"

namespace cek {

namespace {

// Shared memory of a creature's backward run, behind its TeamLayout.
struct TeamAdjointLayout {
    unsigned vel, force, mass, muscle, grad, back, bytes;
    __host__ __device__ static TeamAdjointLayout make(unsigned lanes, unsigned mm) {
        TeamAdjointLayout s;
        s.vel = 8u * lanes;                   // after the positions' adjoints
        s.force = s.vel + 8u * lanes;         // muscle forces' and start positions'
        s.back = s.force + 8u * lanes;        // of the anchors' distance and speed, a muscle
        s.muscle = s.back + 16u * mm;         // (energy store, demand)
        s.mass = s.muscle + 8u * mm;          // gradient of the masses
        s.grad = s.mass + 4u * lanes;         // kGradMuscle a muscle
        const unsigned end = s.grad + 4u * kGradMuscle * mm;
        s.bytes = ((end + 127u) / 128u) * 128u;
        return s;
    }
};

// A substep's entry in a team's segment tape: float4s of every lane, its start
// state (x, y, vx, vy) and what the reverse reads of the substep, then the
// energy stores.
enum TapePart : unsigned {
    kTapeState, kTapePulls, kTapeDrag, kTapeBone, kTapeEnds, kTapeHub, kTapeTurn, kTapeParent, kTapeOwn, kTapeParts
};
__host__ __device__ inline unsigned team_tape_floats(unsigned lanes, unsigned mm) {
    return 4u * kTapeParts * lanes + ((mm + 3u) & ~3u);
}
__host__ __device__ inline unsigned team_tape_warp_floats(unsigned rows, unsigned mm) {
    unsigned most = 0u;
    for (unsigned lanes = 8u; lanes <= team_lanes(rows); lanes *= 2u) {
        const unsigned n = 32u / lanes * team_tape_floats(lanes, mm);
        if (n > most) most = n;
    }
    return 256u * most;
}

struct TeamAdjointArgs {
    float* tape;
    float* grads;
    const float* weights;
    uint32_t* mismatch;
};

template <class W, int RATE>
struct TeamBackward : Team<W, false, RATE, false> {
    using Base = Team<W, false, RATE, false>;
    using C = Clock<RATE>;
    using P = Physics<W, RATE>;
    using Joint = typename P::Joint;
    using Kept = typename Base::Kept;
    using Base::a;
    using Base::ba;
    using Base::bb;
    using Base::damp_level;
    using Base::entry;
    using Base::f;
    using Base::from;
    using Base::has_bone;
    using Base::has_joint;
    using Base::has_node;
    using Base::i;
    using Base::level;
    using Base::mem;
    using Base::nr;
    using Base::offset;
    using Base::pos;
    using Base::pull0;
    using Base::pull1;
    using Base::r;
    using Base::ra;
    using Base::rb;
    using Base::store;
    using Base::T;
    using Base::vel;

    TeamAdjointArgs x;
    TeamAdjointLayout A;
    char* adj = nullptr;  // its creature's adjoints
    float* tape = nullptr;
    unsigned end = 0u, seg = 0u, back_level = 0u, back_levels = 0u, bone_back = 0u, bone_backs = 0u;
    float weight = 1.0f, fric = 0.0f;

    __device__ __forceinline__ TeamBackward(const P& f_, const KernelArgs& a_, LaneRegs& r_, const TeamAdjointArgs& x_)
        : Base{f_, a_, r_}, x(x_) {}

    __device__ __forceinline__ float2& gpos(unsigned n) const { return reinterpret_cast<float2*>(adj)[n]; }
    __device__ __forceinline__ float2& gvel(unsigned n) const { return reinterpret_cast<float2*>(adj + A.vel)[n]; }
    __device__ __forceinline__ float2& gforce(unsigned n) const { return reinterpret_cast<float2*>(adj + A.force)[n]; }
    __device__ __forceinline__ float4& gback(unsigned k) const { return reinterpret_cast<float4*>(adj + A.back)[k]; }
    __device__ __forceinline__ float2& gmuscle(unsigned k) const { return reinterpret_cast<float2*>(adj + A.muscle)[k]; }
    __device__ __forceinline__ float& gmass(unsigned n) const { return reinterpret_cast<float*>(adj + A.mass)[n]; }
    __device__ __forceinline__ float* ggrad(unsigned k) const {
        return reinterpret_cast<float*>(adj + A.grad) + kGradMuscle * k;
    }

    // d J / d w of an inverse mass w = 1 / m, as d J / d m.
    __device__ __forceinline__ void add_inverse_mass(unsigned n, float w, float dw) const {
        gmass(n) = __fmaf_rn(__fmul_rn(-dw, w), w, gmass(n));
    }

    __device__ __forceinline__ void settle(unsigned lane, unsigned lanes, char* warp_mem, float* warp_tape) {
        A = TeamAdjointLayout::make(lanes, a.mm);
        this->place(lane, lanes, warp_mem, A.bytes);
        back_level = bone_back = 0u;
        adj = mem + this->S.bytes;
        // A region is an odd multiple of 64 bytes: the adjoints start there.
        tape = warp_tape + (size_t)(this->base / T) * 256u * team_tape_floats(T, a.mm);
    }

    __device__ __forceinline__ void leave() {
        Base::leave();
        back_level = bone_back = 0u;
    }

    // Takes creature `cidx` on the `fresh` teams (Backward::start); returns
    // whether this lane's team has a trial to run back.
    __device__ __forceinline__ bool start(bool fresh, unsigned cidx) {
        this->begin(fresh, cidx, 0u);
        // Levels from the last item.
        const unsigned topo = __float_as_uint(ra.x);
        const unsigned mine = has_joint() ? (1u << i) | (1u << (topo & 31u)) | (1u << ((topo >> 5u) & 31u)) |
                                                (1u << ((topo >> 10u) & 31u))
                                          : 0u;
        const unsigned ends = has_bone() ? (1u << i) | (1u << (__float_as_uint(ba.x) & 31u)) : 0u;
        unsigned jl = mine != 0u ? 1u : 0u, bl = ends != 0u ? 1u : 0u;
        for (unsigned s = T; s-- > 1u;) {
            const unsigned js = from(jl, s), bs = from(bl, s), ms = from(mine, s), es = from(ends, s);
            if (s > i && (ms & mine) != 0u) jl = max(jl, js + 1u);
            if (s > i && (es & ends) != 0u) bl = max(bl, bs + 1u);
        }
        back_level = jl;
        bone_back = bl;
        back_levels = __reduce_max_sync(kFull, jl);
        bone_backs = __reduce_max_sync(kFull, bl);
        bool usable = false;
        if (fresh) {
            end = a.ends[cidx];
            weight = x.weights ? x.weights[cidx] : 1.0f;
            usable = end > 0u && a.results[cidx].fitness > -1e19f;
            for (unsigned k = i; k < r.muscles; k += T) {
                for (unsigned q = 0u; q < kGradMuscle; q++) {
                    ggrad(k)[q] = 0.0f;
                }
                gmuscle(k) = make_float2(0.0f, 0.0f);
            }
            gpos(i) = make_float2(usable ? weight * nr.x * r.inv_mass : 0.0f, 0.0f);
            gvel(i) = make_float2(0.0f, 0.0f);
            gforce(i) = make_float2(0.0f, 0.0f);
            gmass(i) = 0.0f;
            fric = 0.0f;
            seg = usable ? (end - 1u) / 16u : 0u;
        }
        __syncwarp();
        if (fresh && !usable) {
            finish();
        }
        return usable;
    }

    // The gradients of this lane's part of its creature (Backward::finish).
    __device__ __forceinline__ void finish() const {
        float* out = x.grads + (size_t)r.cidx * grad_floats(a.rows, a.mm);
        for (unsigned k = i; k < r.muscles; k += T) {
            for (unsigned q = 0u; q < kGradMuscle; q++) {
                out[kGradMuscle * k + q] = ggrad(k)[q];
            }
        }
        if (has_node()) {
            out[kGradMuscle * a.mm + i] = fric;
            out[kGradMuscle * a.mm + a.rows + i] = gmass(i);
            const float2 l0 = gpos(i);
            out[kGradMuscle * a.mm + 2u * a.rows + 2u * i] = l0.x;
            out[kGradMuscle * a.mm + 2u * a.rows + 2u * i + 1u] = l0.y;
        }
    }

    __device__ __forceinline__ float* tape_at(unsigned k) const { return tape + (size_t)k * team_tape_floats(T, a.mm); }
    __device__ __forceinline__ float4& part(unsigned k, TapePart n) const {
        return reinterpret_cast<float4*>(tape_at(k))[n * T + i];
    }
    __device__ __forceinline__ static float4 pair(float2 u, float2 v) { return make_float4(u.x, u.y, v.x, v.y); }
    __device__ __forceinline__ void save_state(unsigned k) const {
        if (has_node()) {
            part(k, kTapeState) = pair(pos(i), vel(i));
        }
        float* s = tape_at(k) + 4u * kTapeParts * T;
        for (unsigned m = i; m < r.muscles; m += T) {
            s[m] = store(m).x;
        }
    }
    __device__ __forceinline__ void put_state(unsigned k, const float4& s) const {
        if (has_node()) {
            pos(i) = make_float2(s.x, s.y);
            vel(i) = make_float2(s.z, s.w);
        }
        const float* e = tape_at(k) + 4u * kTapeParts * T;
        for (unsigned m = i; m < r.muscles; m += T) {
            store(m).x = e[m];
        }
    }
    // What the rerun of substep k kept. Of the joint's gradients the hub's and
    // the weight follow from the other two; the positions of a push are saved
    // when there was one.
    __device__ __forceinline__ void save_kept(unsigned k, const Kept& kept) const {
        if (!has_node()) {
            return;
        }
        const unsigned flags = (kept.pushed ? 1u : 0u) | (kept.touched ? 2u : 0u) | (kept.slid ? 4u : 0u);
        part(k, kTapePulls) = pair(kept.pulls, kept.landing);
        part(k, kTapeDrag) = pair(kept.drag0, kept.drag1);
        part(k, kTapeBone) = pair(kept.bone0, kept.bone1);
        part(k, kTapeHub) = make_float4(kept.vh.x, kept.vh.y, __uint_as_float(flags), 0.0f);
        if (has_joint()) {
            part(k, kTapeEnds) = pair(kept.vt, kept.vf);
            part(k, kTapeTurn) = pair(kept.k.g_tip, kept.k.g_far);
        }
        if (kept.pushed) {
            part(k, kTapeParent) = pair(kept.pt, kept.pp);
            part(k, kTapeOwn) = pair(kept.ct, kept.ch);
        }
    }
    struct Entry {
        float4 state, pulls, drag, bone, ends, hub, turn;
    };
    __device__ __forceinline__ Entry entry_of(unsigned k) const {
        const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        Entry e{none, none, none, none, none, none, none};
        if (has_node()) {
            e.state = part(k, kTapeState);
            e.pulls = part(k, kTapePulls);
            e.drag = part(k, kTapeDrag);
            e.bone = part(k, kTapeBone);
            e.hub = part(k, kTapeHub);
            if (has_joint()) {
                e.ends = part(k, kTapeEnds);
                e.turn = part(k, kTapeTurn);
            }
        }
        return e;
    }
    __device__ __forceinline__ Kept kept_of(unsigned k, const Entry& e) const {
        const auto head = [](const float4& v) { return make_float2(v.x, v.y); };
        const auto tail = [](const float4& v) { return make_float2(v.z, v.w); };
        const unsigned flags = __float_as_uint(e.hub.z);
        Kept kept;
        kept.pulls = head(e.pulls);
        kept.landing = tail(e.pulls);
        kept.drag0 = head(e.drag);
        kept.drag1 = tail(e.drag);
        kept.bone0 = head(e.bone);
        kept.bone1 = tail(e.bone);
        kept.vt = head(e.ends);
        kept.vf = tail(e.ends);
        kept.vh = head(e.hub);
        kept.pushed = (flags & 1u) != 0u;
        kept.touched = (flags & 2u) != 0u;
        kept.slid = (flags & 4u) != 0u;
        kept.wgt = 0.0f;
        if (has_joint()) {
            kept.k.g_tip = head(e.turn);
            kept.k.g_far = tail(e.turn);
            P::complete(kept.k, rb);
            kept.wgt = P::joint_weight(kept.k);
        }
        if (kept.pushed) {
            const float4 parent = part(k, kTapeParent), own = part(k, kTapeOwn);
            kept.pt = head(parent);
            kept.pp = tail(parent);
            kept.ct = head(own);
            kept.ch = tail(own);
        }
        return kept;
    }
    __device__ __forceinline__ bool same(float x0, float x1) const { return __float_as_uint(x0) == __float_as_uint(x1); }
    __device__ __forceinline__ const float* checkpoint(unsigned s) const {
        return a.ckpt + (size_t)s * checkpoint_floats(a.rows, a.mm) * a.count + r.cidx;
    }
    __device__ __forceinline__ bool same_as_checkpoint(unsigned s) const {
        const size_t n = a.count;
        const float* c = checkpoint(s);
        bool ok = true;
        if (has_node()) {
            const float2 q = pos(i), u = vel(i);
            ok = same(c[(2u * i) * n], q.x) && same(c[(2u * i + 1u) * n], q.y) &&
                 same(c[(2u * a.rows + 2u * i) * n], u.x) && same(c[(2u * a.rows + 2u * i + 1u) * n], u.y);
        }
        for (unsigned m = i; m < r.muscles; m += T) {
            ok = ok && same(c[(4u * a.rows + m) * n], store(m).x);
        }
        return ok;
    }
    __device__ __forceinline__ void load_checkpoint(unsigned s) const {
        const size_t n = a.count;
        const float* c = checkpoint(s);
        if (has_node()) {
            pos(i) = make_float2(c[(2u * i) * n], c[(2u * i + 1u) * n]);
            vel(i) = make_float2(c[(2u * a.rows + 2u * i) * n], c[(2u * a.rows + 2u * i + 1u) * n]);
        }
        for (unsigned m = i; m < r.muscles; m += T) {
            store(m).x = c[(4u * a.rows + m) * n];
        }
    }

    // A joint's push node += w lam g with lam = -e / wgt: the inverse mass's
    // share (Backward::weights_back).
    template <bool HUB = false>
    __device__ __forceinline__ void weights_back(unsigned node, float w, float2 gv, float2 ap, float lam,
                                                 float lwgt) const {
        const float pushed = HUB ? sum2(gv.y, ap.y, gv.x, ap.x) : sum2(gv.x, ap.x, gv.y, ap.y);
        add_inverse_mass(node, w, sum2(lam, pushed, lwgt, sum2(gv.x, gv.x, gv.y, gv.y)));
    }
    // The adjoint of a joint's geometry into its nodes' positions: `lu` of the
    // parent bone, `lv` of its own.
    __device__ __forceinline__ void geometry_back(float2 lu, float2 lv) const {
        const unsigned topo = __float_as_uint(ra.x);
        const unsigned hub = topo & 31u, ptip = (topo >> 5u) & 31u, ppivot = (topo >> 10u) & 31u;
        float2 e = gpos(ptip);
        gpos(ptip) = make_float2(e.x + lu.x, e.y + lu.y);
        e = gpos(ppivot);
        gpos(ppivot) = make_float2(e.x - lu.x, e.y - lu.y);
        e = gpos(i);
        gpos(i) = make_float2(e.x + lv.x, e.y + lv.y);
        e = gpos(hub);
        gpos(hub) = make_float2(e.x - lv.x, e.y - lv.y);
    }

    // The reverse of a substep (Backward::reverse_substep) from what its rerun
    // kept and the state `s0` at its start (tape entry k_tape). Shared memory
    // holds the positions at its end, the start of the one after, and then
    // those at its start.
    __device__ __forceinline__ void reverse_substep(unsigned k_tape, const float4& s0, const Kept& kept) {
        const ce_params& p = f.p;
        const unsigned topo = __float_as_uint(ra.x);
        const unsigned hub = topo & 31u, ptip = (topo >> 5u) & 31u, ppivot = (topo >> 10u) & 31u,
                       far = (topo >> 15u) & 31u;
        const unsigned i0 = __float_as_uint(ba.x) & 31u;
        const bool node = has_node(), joint = has_joint();
        // Damping.
        for (unsigned l = 1u; l <= back_levels; l++) {
            if (joint && back_level == l && kept.wgt > 0.0f) {
                float2 lgt, lgf;
                float lam, lrate, lwgt;
                const Joint& k = kept.k;
                const float2 at = gvel(i), af = gvel(far), ah = gvel(hub);
                damping_back(k, kept.wgt, fminf(C::h * kInvJointDamping, 1.0f), kept.vt, kept.vf, kept.vh, at, af, ah,
                             lam, lrate, lwgt, lgt, lgf);
                gvel(i) = make_float2(__fmaf_rn(lrate, k.g_tip.x, at.x), __fmaf_rn(lrate, k.g_tip.y, at.y));
                gvel(far) = make_float2(__fmaf_rn(lrate, k.g_far.x, af.x), __fmaf_rn(lrate, k.g_far.y, af.y));
                gvel(hub) = make_float2(__fmaf_rn(lrate, k.g_hub.x, ah.x), __fmaf_rn(lrate, k.g_hub.y, ah.y));
                weights_back(i, k.w_tip, k.g_tip, at, lam, lwgt);
                weights_back(far, k.w_far, k.g_far, af, lam, lwgt);
                this->template weights_back<true>(hub, k.w_hub, k.g_hub, ah, lam, lwgt);
                float2 lu, lv;
                joint_geometry_back<true>(pos(ptip), pos(ppivot), pos(i), pos(hub), ((topo >> 20u) & 1u) != 0u, lgt, lgf, 0.0f, lu, lv);
                geometry_back(lu, lv);
            }
            __syncwarp();
        }
        // Velocity from the positions, then the ground contact.
        if (node) {
            const float2 lv = gvel(i);
            float2 lq = gpos(i);
            lq.x = __fmaf_rn(lv.x, C::inv_h, lq.x);
            lq.y = __fmaf_rn(lv.y, C::inv_h, lq.y);
            float2 lf = make_float2(-lv.x * C::inv_h, -lv.y * C::inv_h);
            if (kept.touched) {
                contact_back(f.w, p, r.amp, r.qphase, nr, kept.landing, make_float2(s0.x, s0.y), kept.slid, lq, lf, fric);
            }
            gpos(i) = lq;
            gforce(i) = lf;
            gvel(i) = make_float2(0.0f, 0.0f);
        }
        __syncwarp();
        // Joint limits, where a joint was pushed.
        if (__any_sync(kFull, kept.pushed)) {
            for (unsigned l = 1u; l <= back_levels; l++) {
                if (kept.pushed && back_level == l) {
                    float2 lgt, lgf;
                    float lam, lerr, lwgt;
                    float2 g_tip, g_far, g_hub;
                    const float2 at = gpos(i), af = gpos(far), ah = gpos(hub);
                    limit_back(ra, rb, kept.pt, kept.pp, kept.ct, kept.ch, at, af, ah, lam, lerr, lwgt, lgt, lgf, g_tip,
                               g_far, g_hub);
                    weights_back(i, rb.x, g_tip, at, lam, lwgt);
                    weights_back(far, rb.y, g_far, af, lam, lwgt);
                    this->template weights_back<true>(hub, rb.z, g_hub, ah, lam, lwgt);
                    float2 lu, lv;
                    joint_geometry_back<false>(kept.pt, kept.pp, kept.ct, kept.ch, ((topo >> 20u) & 1u) != 0u, lgt, lgf, lerr, lu, lv);
                    geometry_back(lu, lv);
                }
                __syncwarp();
            }
        }
        // Bone lengths.
        for (unsigned l = 1u; l <= bone_backs; l++) {
            if (bone_back == l) {
                const float4 pre = make_float4(kept.bone0.x, kept.bone0.y, kept.bone1.x, kept.bone1.y);
                float2 l0 = gpos(i0), l1 = gpos(i);
                float d0, d1;
                bone_length_back(ba, pre, l0, l1, d0, d1);
                gpos(i0) = l0;
                gpos(i) = l1;
                add_inverse_mass(i0, ba.z, d0);
                add_inverse_mass(i, ba.w, d1);
            }
            __syncwarp();
        }
        // Integration.
        if (node) {
            const float2 lq1 = gpos(i), lq0 = gforce(i);
            float2 lp, lv1, lf;
            float dm;
            integrate_back<C>(f.w, p, nr, kept.pulls, s0.y, lq1, lq0, lp, lv1, lf, dm);
            gpos(i) = lp;
            gvel(i) = lv1;
            gforce(i) = lf;
            gmass(i) = __fmaf_rn(__fmul_rn(__fmul_rn(-C::h, nr.y), nr.y), dm, gmass(i));
        }
        // The substep's start state, for the water's share and the muscles.
        put_state(k_tape, s0);
        __syncwarp();
        // Bone drag.
        float r0 = 0.0f, im0 = from(nr.y, i0);
        if (f.w.has(CE_FLAG_WATER)) {
            r0 = from(nr.z, i0);
        }
        for (unsigned l = 1u; l <= bone_backs; l++) {
            if (bone_back == l) {
                const float4 pre = make_float4(kept.drag0.x, kept.drag0.y, kept.drag1.x, kept.drag1.y);
                float2 l0 = gvel(i0), l1 = gvel(i), e0, e1;
                float llimit, d0, d1;
                const bool water = f.w.has(CE_FLAG_WATER);
                if (water) {
                    e0 = gpos(i0);
                    e1 = gpos(i);
                }
                bone_drag_back<C>(f.w, p, ba, bb, pre, r0, nr.z, pos(i0), pos(i), l0, l1, e0, e1, llimit, d0, d1);
                if (water) {
                    gpos(i0) = e0;
                    gpos(i) = e1;
                }
                if (llimit != 0.0f) {
                    gmass(i0) = __fmaf_rn(0.5f * C::inv_h, llimit, gmass(i0));
                    gmass(i) = __fmaf_rn(0.5f * C::inv_h, llimit, gmass(i));
                }
                add_inverse_mass(i0, im0, d0);
                add_inverse_mass(i, nr.y, d1);
                gvel(i0) = l0;
                gvel(i) = l1;
            }
            __syncwarp();
        }
        muscles_back();
    }

    // The reverse of the muscle pass (Backward::muscles_back).
    __device__ __forceinline__ void muscles_back() const {
        bool finite = true;
        for (unsigned k = i; k < r.muscles; k += T) {
            const float4 q0 = pull0(k);
            const unsigned nodes = __float_as_uint(q0.x);
            const unsigned a0 = nodes & 255u, a1 = (nodes >> 8u) & 255u, b0 = (nodes >> 16u) & 255u, b1 = nodes >> 24u;
            const auto at = [&](unsigned n) {
                const float2 q = pos(n), u = vel(n);
                return make_float4(q.x, q.y, u.x, u.y);
            };
            const float2 lm = gmuscle(k);
            MuscleBack m;
            muscle_back<C>(f.p, q0, pull1(k), store(k), at(a0), at(a1), at(b0), at(b1), gforce(a0), gforce(a1), gforce(b0),
                           gforce(b1), lm, m);
            gback(k) = make_float4(m.ldx, m.ldy, m.lrvx, m.lrvy);
            gmuscle(k) = make_float2(m.le, m.ld);
            float* g = ggrad(k);
            g[1] += m.hill;
            g[2] += m.cap;
            g[3] = __fmaf_rn(m.icap, f.p.inv_muscle_energy, g[3]);
            finite = finite && fabsf(m.ldx) < 1e38f && fabsf(m.ldy) < 1e38f && fabsf(m.lrvx) < 1e38f &&
                     fabsf(m.lrvy) < 1e38f;
        }
        const bool all_finite = __all_sync(kFull, finite);
        __syncwarp();
        if (has_node()) {
            float2 e = gpos(i), u = gvel(i);
            if (all_finite) {
                for (unsigned n = this->e0; n < this->e1; n++) {
                    const float2 w = entry(n);
                    const float4 d = gback(__float_as_uint(w.y));
                    e.x = __fmaf_rn(-w.x, d.x, e.x);
                    e.y = __fmaf_rn(-w.x, d.y, e.y);
                    u.x = __fmaf_rn(-w.x, d.z, u.x);
                    u.y = __fmaf_rn(-w.x, d.w, u.y);
                }
            } else {
                for (unsigned k = 0u; k < r.muscles; k++) {
                    const float4 q0 = pull0(k), d = gback(k);
                    const unsigned nodes = __float_as_uint(q0.x);
                    const float weights[4] = {1.0f - q0.y, q0.y, -(1.0f - q0.z), -q0.z};
                    for (unsigned n = 0u; n < 4u; n++) {
                        if (((nodes >> (8u * n)) & 255u) == i) {
                            e.x = __fmaf_rn(-weights[n], d.x, e.x);
                            e.y = __fmaf_rn(-weights[n], d.y, e.y);
                            u.x = __fmaf_rn(-weights[n], d.z, u.x);
                            u.y = __fmaf_rn(-weights[n], d.w, u.y);
                        }
                    }
                }
            }
            gpos(i) = e;
            gvel(i) = u;
        }
        __syncwarp();
    }

    // The reverse of the step's demands (Backward::demands_back).
    __device__ __forceinline__ void demands_back(float t_now) const {
        if (r.nodes == 0u) {
            return;
        }
        const float4* mus = reinterpret_cast<const float4*>(a.muscles + this->rhythm_at);
        for (unsigned k = i; k < r.muscles; k += T) {
            const float ld = gmuscle(k).y;
            gmuscle(k).y = 0.0f;
            demand_back<C>(t_now, __ldg(mus + 5u * k + 2u), __ldg(mus + 5u * k + 3u), offset(k), r.limp, ld, ggrad(k));
        }
    }

    // A team without a step to run in the warp's turn sits it out.
    struct Hidden {
        unsigned nodes, muscles, level, damp_level, back_level, bone_back, e0, e1;
        float topo;
    };
    __device__ __forceinline__ Hidden hide(bool out) {
        const Hidden h{r.nodes, r.muscles, level, damp_level, back_level, bone_back, this->e0, this->e1, ra.x};
        if (out) {
            r.nodes = r.muscles = 0u;
            level = damp_level = back_level = bone_back = 0u;
            this->e0 = this->e1 = 0u;
            ra.x = __uint_as_float(kNone);
        }
        return h;
    }
    __device__ __forceinline__ void show(const Hidden& h) {
        r.nodes = h.nodes;
        r.muscles = h.muscles;
        level = h.level;
        damp_level = h.damp_level;
        back_level = h.back_level;
        bone_back = h.bone_back;
        this->e0 = h.e0;
        this->e1 = h.e1;
        ra.x = h.topo;
    }

    // One segment of every `live` team, backwards (Backward::segment).
    // Returns whether segments remain.
    __device__ __forceinline__ bool segment(bool live) {
        const unsigned s0 = seg * 16u, steps = live ? min(16u, end - s0) : 0u;
        const unsigned most = __reduce_max_sync(kFull, steps);
        if (live) {
            load_checkpoint(seg);
        }
        __syncwarp();
        for (unsigned s = 0u; s < most; s++) {
            const bool on = s < steps;
            const Hidden h = hide(!on);
            this->demands(__fmul_rn((float)(s0 + s), C::dt));
            __syncwarp();
            for (unsigned q = 0u; q < 16u; q++) {
                Kept kept;
                save_state(s * 16u + q);
                this->template substep<true>(&kept);
                save_kept(s * 16u + q, kept);
            }
            show(h);
            if (on && s + 1u == steps) {
                if (x.mismatch && s0 + steps < end && !same_as_checkpoint(seg + 1u)) {
                    atomicOr(x.mismatch + r.cidx, 1u);
                }
                if (s0 + steps == end && has_node()) {
                    // Fitness com_x = sum m x / sum m.
                    float com_x = 0.0f;
                    for (unsigned n = 0u; n < r.nodes; n++) {
                        com_x = __fmaf_rn(this->tally_of(n).x, pos(n).x, com_x);
                    }
                    com_x = __fmul_rn(com_x, r.inv_mass);
                    gmass(i) = __fmaf_rn(__fmul_rn(weight, r.inv_mass), pos(i).x - com_x, gmass(i));
                }
            }
            __syncwarp();
        }
        for (unsigned s = most; s-- > 0u;) {
            const Hidden h = hide(s >= steps);
            const float t_now = __fmul_rn((float)(s0 + s), C::dt);
            this->demands(t_now);
            Entry now = entry_of(s * 16u + 15u);
            for (unsigned q = 16u; q-- > 0u;) {
                const unsigned k = s * 16u + q;
                // The entry before comes while this substep is worked on.
                const Entry next = q > 0u ? entry_of(k - 1u) : now;
                reverse_substep(k, now.state, kept_of(k, now));
                now = next;
            }
            demands_back(t_now);
            show(h);
            __syncwarp();
        }
        if (!live || seg == 0u) {
            return false;
        }
        seg--;
        return true;
    }
};

template <class W, int RATE>
__global__ void __launch_bounds__(kTeamBlock, kTeamAdjointMinBlocks)
    team_adjoint_kernel(const KernelArgs a, const ce_params p, const TeamAdjointArgs x, unsigned warp_bytes) {
    extern __shared__ float4 smem[];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5u;
    const W w{};
    LaneRegs r;
    const Physics<W, RATE> f{w, p, r};
    TeamBackward<W, RATE> t(f, a, r, x);
    TeamClaim claim(a, lane, warp, gridDim.x * (blockDim.x >> 5u));
    char* const mem = reinterpret_cast<char*>(smem) + (threadIdx.x >> 5u) * warp_bytes;
    float* const tape = x.tape + (size_t)warp * team_tape_warp_floats(a.rows, a.mm);
    t.settle(lane, claim.lanes, mem, tape);
    bool live = false;
    for (;;) {
        const unsigned got = claim.next(!live && t.i == 0u);
        const unsigned mine = __shfl_sync(kFull, got, t.base);
        const bool fresh = !live && mine != kNone;
        if (__any_sync(kFull, fresh)) {
            const unsigned cidx = fresh ? (a.order ? __ldg(a.order + mine) : p.base + mine) : 0u;
            const bool usable = t.start(fresh, cidx);
            if (fresh && !usable) {
                t.leave();
            }
            live = live || (fresh && usable);
            if (!__any_sync(kFull, live)) {
                continue;
            }
        }
        if (!__any_sync(kFull, live)) {
            if (!claim.next_group()) {
                break;
            }
            t.settle(lane, claim.lanes, mem, tape);
            continue;
        }
        const bool was = live;
        live = t.segment(live);
        if (was && !live) {
            t.finish();
            t.leave();
        }
    }
}

unsigned team_adjoint_warp_bytes(unsigned first_n, unsigned rows, unsigned mm) {
    unsigned most = 0u;
    for (unsigned lanes = team_lanes(first_n); lanes <= team_lanes(rows); lanes *= 2u) {
        const unsigned bytes =
            32u / lanes * (TeamLayout::make(lanes, mm, false).bytes + TeamAdjointLayout::make(lanes, mm).bytes);
        if (bytes > most) most = bytes;
    }
    return most;
}

template <class F>
cudaError_t with_gradient_world(uint32_t flags, int rate, F&& go) {
    const auto at = [&](auto w) -> cudaError_t {
        if (rate == 60) return go(w, std::integral_constant<int, 60>{});
        if (rate == 120) return go(w, std::integral_constant<int, 120>{});
        return cudaErrorInvalidValue;
    };
    switch (flags) {
        case kWorldCalm: return at(StaticWorld<kWorldCalm>{});
        case kWorldEffects: return at(StaticWorld<kWorldEffects>{});
        case kWorldEffectsQuake: return at(StaticWorld<kWorldEffectsQuake>{});
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

size_t team_adjoint_tape_bytes(unsigned blocks, unsigned rows, unsigned mm) {
    return (size_t)blocks * (kTeamBlock / 32u) * team_tape_warp_floats(rows, mm) * 4u;
}

cudaError_t team_adjoint_blocks(unsigned rows, unsigned mm, uint32_t flags, int rate, unsigned sms, size_t warps,
                                unsigned* blocks) {
    const size_t smem = (size_t)team_adjoint_warp_bytes(2u, rows, mm) * (kTeamBlock / 32u);
    return with_gradient_world(flags, rate, [&](auto w, auto rt) -> cudaError_t {
        auto kern = team_adjoint_kernel<decltype(w), decltype(rt)::value>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)kTeamBlock, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
        const size_t need = (warps + kTeamBlock / 32u - 1u) / (kTeamBlock / 32u), full = (size_t)per_sm * sms;
        *blocks = (unsigned)(need < 1u ? 1u : need < full ? need : full);
        return cudaSuccess;
    });
}

cudaError_t launch_team_adjoint(const TeamSpec& s, const KernelArgs& a, const ce_params& p, float* tape, float* grads,
                                const float* weights, uint32_t* mismatch) {
    const unsigned warp_bytes = team_adjoint_warp_bytes(2u, a.rows, a.mm);
    const TeamAdjointArgs x{tape, grads, weights, mismatch};
    return with_gradient_world(s.flags, s.rate, [&](auto w, auto rt) -> cudaError_t {
        auto kern = team_adjoint_kernel<decltype(w), decltype(rt)::value>;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        kern<<<s.blocks, kTeamBlock, (size_t)warp_bytes * (kTeamBlock / 32u), s.stream>>>(a, p, x, warp_bytes);
        return cudaGetLastError();
    });
}

}  // namespace cek

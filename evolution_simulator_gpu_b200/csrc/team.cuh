// The creature kernel for launches whose time is one creature's: several
// lanes a creature.
//
// With one creature a lane (trial.cuh) a substep is a serial chain over all
// of a body's muscles, bones, joints and nodes. A launch of a few thousand
// creatures, or the last creatures of a large one, takes as long as that
// chain however empty the GPU is. Here a team of T lanes (8, 16 or 32: the
// least power of two that gives every node a lane) runs one creature:
//
// * lane i holds node i, the bone that ends there and that bone's joint, with
//   their constants in registers and its state in shared memory;
// * the muscles go round the lanes; their forces meet in shared memory and
//   each node's lane adds up its own in the muscles' order (a list built when
//   the trial begins), so a sum has the serial pass's rounding;
// * the bones' drag and lengths, which update two nodes each in bone order,
//   run in levels: a bone goes when every earlier bone at its nodes has. Levels
//   are the depth of the body's left-child right-sibling tree (3 to 6 for 6
//   to 10 nodes) instead of its bone count. The damping runs in levels too,
//   over the joints that share a node;
// * the joint ranges are tested all at once. A joint whose test saw no pushed
//   node keeps its verdict; only those after a push on their nodes are tested
//   again.
//
// Every operation and every order of operations on a value is the serial
// pass's, so the results are the same to the bit (Physics holds the
// arithmetic of both).
#pragma once
#include "team_physics.cuh"
#include "trial.cuh"

namespace cek {

// Shared memory of one creature: offsets in bytes. A team's regions lie an
// odd multiple of 64 bytes apart, so the 8-byte accesses of two teams of 8
// lanes meet in no bank.
struct TeamLayout {
    unsigned vel, tally, pull0, pull1, store, force, offset, entries, words, shown, kept, bytes;
    __host__ __device__ static TeamLayout make(unsigned lanes, unsigned mm, bool record) {
        TeamLayout s;
        s.vel = 8u * lanes;                 // after the positions
        s.tally = s.vel + 8u * lanes;       // (mass, radius) of each node
        s.pull0 = s.tally + 8u * lanes;     // the muscles' two pull lines
        s.pull1 = s.pull0 + 16u * mm;
        s.store = s.pull1 + 16u * mm;       // (energy store, demand)
        s.force = s.store + 8u * mm;        // (fx, fy)
        s.entries = s.force + 8u * mm;      // (weight, muscle) of each node's forces
        s.offset = s.entries + 32u * mm;    // touchdown offsets
        s.words = s.offset + 4u * mm;       // result and tallies
        s.shown = s.words + 4u * 32u;       // RECORD: pulls
        s.kept = s.shown + (record ? 4u * mm : 0u);
        const unsigned end = s.kept + (record ? 4u * 20u : 0u);
        s.bytes = ((end + 63u) / 128u) * 128u + 64u;
        return s;
    }
};

// Lanes of the team of a body with `nodes` nodes.
__host__ __device__ inline unsigned team_lanes(unsigned nodes) { return nodes <= 8u ? 8u : nodes <= 16u ? 16u : 32u; }

// Which creatures the warp's teams take next: as Claim, from the queues of
// the node counts that one team size serves. A warp whose queues run dry
// goes on with the next team size once its creatures are done. Queues go
// from the largest body down, so the longest trials start first.
struct TeamClaim {
    const KernelArgs& a;
    const unsigned lane, warps_total;
    unsigned lanes = 0u;  // of a team
    unsigned group = 0u, tried = 0u, q_lo = 0u, q_hi = 0u, win_cur = 0u, win_end = 0u;
    bool drained = true;

    __device__ __forceinline__ unsigned queues() const { return a.queues > 0u ? a.queues : 1u; }
    // The positions of queue q: the launch's queues, or the states of a tail
    // by team size.
    __device__ __forceinline__ unsigned start(unsigned q) const {
        return a.resume ? q * a.tail.most : a.queues > 0u ? a.bounds[q] : 0u;
    }
    __device__ __forceinline__ unsigned size(unsigned q) const {
        return a.resume ? a.tail.counters[kTailWritten + q] : a.queues > 0u ? a.bounds[q + 1u] - a.bounds[q] : a.count;
    }
    // Queues of team size g: node counts up to 8, 16, 32.
    __device__ __forceinline__ unsigned first_queue(unsigned g) const {
        const unsigned n = g == 0u ? 0u : g == 1u ? 9u : g == 2u ? 17u : CE_MAX_NODES + 1u;
        return min(n > a.first_n ? n - a.first_n : 0u, queues());
    }
    __device__ __forceinline__ void enter(unsigned g) {
        group = g;
        if (a.resume) {
            lanes = 8u << g;
            q_lo = g;
            q_hi = g + 1u;
        } else if (a.queues == 0u) {
            lanes = team_lanes(a.rows);
            q_lo = 0u;
            q_hi = 1u;
        } else {
            lanes = 8u << g;
            q_lo = first_queue(g);
            q_hi = first_queue(g + 1u);
        }
        drained = false;
    }
    // The next team size with work; false when all have been served.
    __device__ __forceinline__ bool next_group() {
        if (a.queues == 0u && !a.resume) return false;
        if (++tried >= 3u) return false;
        enter(group == 2u ? 0u : group + 1u);
        return true;
    }

    __device__ __forceinline__ TeamClaim(const KernelArgs& args, unsigned lane_, unsigned warp, unsigned warps)
        : a(args), lane(lane_), warps_total(warps) {
        if (a.queues == 0u && !a.resume) {
            enter(0u);
            return;
        }
        // Warps each team size needs to run all its creatures at once. When
        // they all fit each gets that many; else they share the warps by
        // estimated work times lanes.
        unsigned long long need[3], load[3], needs = 0ull, loads = 0ull;
#pragma unroll
        for (unsigned g = 0u; g < 3u; g++) {
            const unsigned per = 4u >> g;
            if (a.resume) {
                need[g] = (size(g) + per - 1u) / per;
                load[g] = need[g];
            } else {
                const unsigned q0 = first_queue(g), q1 = first_queue(g + 1u);
                need[g] = (a.bounds[q1] - a.bounds[q0] + per - 1u) / per;
                load[g] = (a.work[q1] - a.work[q0]) * (8ull << g);
            }
            needs += need[g];
            loads += load[g];
        }
        unsigned g = 2u;
        if (needs <= warps_total) {
            g = warp < need[2] ? 2u : warp < need[2] + need[1] ? 1u : 0u;
        } else {
            const unsigned long long at = loads * (2ull * warp + 1ull) / (2ull * warps_total);
            g = at < load[2] ? 2u : at < load[2] + load[1] ? 1u : 0u;
        }
        enter(g);
    }

    // The next position of the order for each leader lane that `wants` one.
    __device__ __forceinline__ unsigned next(bool wants) {
        const unsigned below = (1u << lane) - 1u;
        unsigned need = __ballot_sync(kFull, wants);
        unsigned mine = kNone;
        while (need != 0u) {
            if (win_cur >= win_end) {
                if (drained) {
                    break;
                }
                unsigned c0 = kNone, c1 = 0u;
                if (lane == 0u) {
                    for (unsigned q = q_hi; q-- > q_lo;) {
                        const unsigned lo = start(q), n = size(q);
                        const unsigned seen = *reinterpret_cast<volatile unsigned*>(a.counter + q);
                        if (seen >= n) {
                            continue;
                        }
                        const unsigned want = min((unsigned)__popc(need), max((n - seen) / warps_total, 1u));
                        const unsigned got = atomicAdd(a.counter + q, want);
                        if (got >= n) {
                            continue;
                        }
                        // From the queue's end: its muscle counts ascend.
                        c1 = lo + n - got;
                        c0 = lo + n - min(got + want, n);
                        break;
                    }
                }
                c0 = __shfl_sync(kFull, c0, 0);
                c1 = __shfl_sync(kFull, c1, 0);
                if (c0 == kNone) {
                    drained = true;
                    break;
                }
                win_cur = c0;
                win_end = c1;
            }
            const unsigned rank = (unsigned)__popc(need & below);
            const bool take = ((need >> lane) & 1u) != 0u && rank < win_end - win_cur;
            if (take) {
                mine = win_cur + rank;
            }
            const unsigned taken = __ballot_sync(kFull, take);
            need &= ~taken;
            win_cur += (unsigned)__popc(taken);
        }
        return mine;
    }
};

template <class W, bool RECORD, int RATE, bool CKPT>
struct Team {
    using C = Clock<RATE>;
    using P = Physics<W, RATE>;
    using Joint = typename P::Joint;
    const P& f;
    const KernelArgs& a;
    LaneRegs& r;

    // This lane's place: its team's size, first lane and lanes' bits, and its
    // index i in the team.
    unsigned T = 8u, base = 0u, i = 0u, mask = 0xffu;
    char* mem = nullptr;  // its creature's shared memory
    TeamLayout S;

    // Node i, bone i - 1 (pivot to node i), its joint.
    float4 nr, ba, bb, ra, rb;
    float2 shown_force;                  // RECORD: contact forces summed over a step
    unsigned e0 = 0u, e1 = 0u;           // the node's entries
    unsigned level = 0u, damp_level = 0u;  // 0: no bone, no joint
    unsigned before = 0u;                // lanes whose joints this one's test depends on
    unsigned levels = 0u, damp_levels = 0u;  // the warp's most
    unsigned rhythm_at = 0u;             // the creature's muscle records
    bool distinct = true;                // every joint of the warp's bodies joins three nodes

    __device__ __forceinline__ float2& pos(unsigned n) const { return reinterpret_cast<float2*>(mem)[n]; }
    __device__ __forceinline__ float2& vel(unsigned n) const { return reinterpret_cast<float2*>(mem + S.vel)[n]; }
    __device__ __forceinline__ float2& tally_of(unsigned n) const {
        return reinterpret_cast<float2*>(mem + S.tally)[n];
    }
    __device__ __forceinline__ float4& pull0(unsigned k) const { return reinterpret_cast<float4*>(mem + S.pull0)[k]; }
    __device__ __forceinline__ float4& pull1(unsigned k) const { return reinterpret_cast<float4*>(mem + S.pull1)[k]; }
    __device__ __forceinline__ float2& store(unsigned k) const { return reinterpret_cast<float2*>(mem + S.store)[k]; }
    __device__ __forceinline__ float2& force(unsigned k) const { return reinterpret_cast<float2*>(mem + S.force)[k]; }
    __device__ __forceinline__ float& offset(unsigned k) const { return reinterpret_cast<float*>(mem + S.offset)[k]; }
    __device__ __forceinline__ float2& entry(unsigned e) const { return reinterpret_cast<float2*>(mem + S.entries)[e]; }
    __device__ __forceinline__ float* words() const { return reinterpret_cast<float*>(mem + S.words); }
    __device__ __forceinline__ float& shown(unsigned k) const { return reinterpret_cast<float*>(mem + S.shown)[k]; }
    __device__ __forceinline__ float* kept() const { return reinterpret_cast<float*>(mem + S.kept); }

    __device__ __forceinline__ float from(float x, unsigned n) const { return __shfl_sync(kFull, x, base + n); }
    __device__ __forceinline__ unsigned from(unsigned x, unsigned n) const { return __shfl_sync(kFull, x, base + n); }
    __device__ __forceinline__ unsigned votes(bool x) const { return (__ballot_sync(kFull, x) >> base) & mask; }

    // `extra`: bytes of a creature's memory behind its own (a multiple of 128).
    __device__ __forceinline__ void place(unsigned lane, unsigned lanes, char* warp_mem, unsigned extra = 0u) {
        T = lanes;
        i = lane & (T - 1u);
        base = lane - i;
        mask = T == 32u ? kFull : (1u << T) - 1u;
        S = TeamLayout::make(T, a.mm, RECORD);
        mem = warp_mem + (base / T) * (S.bytes + extra);
        nr = make_float4(1.0f, 1.0f, 0.0f, 0.0f);
        ba = bb = ra = rb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        shown_force = make_float2(0.0f, 0.0f);
        r = LaneRegs{};
        leave();
    }
    // No creature on this team.
    __device__ __forceinline__ void leave() {
        r.nodes = 0u;
        r.muscles = 0u;
        level = 0u;
        damp_level = 0u;
        e0 = e1 = 0u;
        before = 0u;
        ra.x = __uint_as_float(kNone);
    }

    __device__ __forceinline__ bool has_node() const { return i < r.nodes; }
    __device__ __forceinline__ bool has_bone() const { return i != 0u && i < r.nodes; }

    // Starts creature `cidx` on the teams whose lanes are `fresh` (Trial::begin).
    // The whole warp calls it.
    __device__ __forceinline__ void begin(bool fresh, unsigned cidx, unsigned slot) {
        const ce_params& pr = f.p;
        const uint32_t* rec = nullptr;
        const float* mus = nullptr;
        [[maybe_unused]] float4 new_nr = nr, new_ba = ba, new_bb = bb, new_ra = ra, new_rb = rb;
        unsigned pivot = 0u;
        bool foot = false;
        if (fresh) {
            const uint4 h0 = __ldcs(&a.heads[2u * cidx]);
            const uint4 h1 = __ldcs(&a.heads[2u * cidx + 1u]);
            r.cidx = cidx;
            r.rec_slot = slot;
            r.nodes = h0.x & 255u;
            r.muscles = h0.y;
            rec = a.records + h0.w;
            rhythm_at = h1.x;
            mus = a.muscles + h1.x;
            r.inv_mass = __uint_as_float(h1.z);
            r.flags = h1.w >> 16u;
            r.period_f = h2f(h1.w & 0xffffu);
            if (f.w.has(CE_FLAG_QUAKE)) {
                r.qphase = (float)(h0.z & 0xffffu) * (1.0f / 65536.0f);
                r.amp = pr.terrain + pr.quake * (0.6f + (float)((h0.z >> 16u) & 0xffffu) * (0.8f / 65536.0f));
            } else {
                r.qphase = 0.0f;
                r.amp = pr.terrain;
            }
            r.limp = false;
            r.scoring = true;
            r.step = 0u;
            new_nr = make_float4(1.0f, 1.0f, 0.0f, 0.0f);
            if (has_node()) {
                const uint32_t* q = rec + i * CE_NODE_WORDS;
                const float m = __uint_as_float(__ldcs(q + 0));
                new_nr = make_float4(m, 1.0f / m, __uint_as_float(__ldcs(q + 1)), __uint_as_float(__ldcs(q + 2)));
                pos(i) = make_float2(__uint_as_float(__ldcs(q + 3)), __uint_as_float(__ldcs(q + 4)));
                vel(i) = make_float2(0.0f, 0.0f);
                foot = (__ldcs(q + 5) & 1u) != 0u;
                tally_of(i) = make_float2(new_nr.x, new_nr.z);
            }
            shown_force = make_float2(0.0f, 0.0f);
        }
        const unsigned feet = votes(foot);
        if (fresh) r.feet = feet;
        // The bone that ends at node i and its joint.
        unsigned far = 0u;
        new_ra.x = fresh ? __uint_as_float(kNone) : new_ra.x;
        uint32_t length = 0u, pj = kNone, lo = 0u, hi = 0u, parent_pivot = 0u;
        if (fresh && has_bone()) {
            const uint32_t* bone_rec = rec + r.nodes * CE_NODE_WORDS;
            const uint32_t* q = bone_rec + (i - 1u) * CE_BONE_WORDS;
            pivot = __ldcs(q + 0);
            length = __ldcs(q + 1);
            pj = __ldcs(q + 2);
            lo = __ldcs(q + 3);
            hi = __ldcs(q + 4);
            if (i > 1u && pj != kNone) {
                parent_pivot = __ldcs(bone_rec + pj * CE_BONE_WORDS);
                far = pivot == parent_pivot ? pj + 1u : parent_pivot;
            }
        }
        const float n0x = from(new_nr.x, pivot), n0y = from(new_nr.y, pivot), n0z = from(new_nr.z, pivot);
        const float far_inv = from(new_nr.y, far);
        unsigned writes = 0u, reads = 0u;
        if (fresh) {
            nr = new_nr;
            ba = bb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            ra = make_float4(__uint_as_float(kNone), 0.0f, 0.0f, 0.0f);
            rb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (has_bone()) {
                const float len = __uint_as_float(length);
                const float width = n0z + nr.z;
                const float bone_mass = n0x + nr.x;
                ba = make_float4(__uint_as_float(pivot), len, n0y, nr.y);
                bb = make_float4(kAirDrag * len * width, 0.5f * bone_mass * C::inv_h, 0.5f * C::h * n0y,
                                 0.5f * C::h * nr.y);
                if (i > 1u && pj != kNone) {
                    const bool at_head = pivot == parent_pivot;
                    const unsigned topo = pivot | ((pj + 1u) << 5u) | (parent_pivot << 10u) | (far << 15u) |
                                          ((at_head ? 1u : 0u) << 20u);
                    const float l = __uint_as_float(lo), h = __uint_as_float(hi);
                    ra = make_float4(__uint_as_float(topo), l, h, 0.5f * (l + h));
                    rb = make_float4(nr.y, far_inv, n0y, 0.0f);
                    writes = (1u << i) | (1u << far) | (1u << pivot);
                    reads = (1u << i) | (1u << pivot) | (1u << (pj + 1u)) | (1u << parent_pivot);
                }
            }
            for (unsigned k = i; k < r.muscles; k += T) {
                const float4* q = reinterpret_cast<const float4*>(mus + k * CE_MUSCLE_FIELDS);
                pull0(k) = __ldcs(q + 0);
                pull1(k) = __ldcs(q + 1);
                store(k) = make_float2(1.0f, 0.0f);
                offset(k) = 0.0f;
                if (RECORD) {
                    shown(k) = 0.0f;
                }
            }
            if (i == 0u) {
                float lw[36];
                start_words(lw, pos(0u));
                for (unsigned q = 0u; q < 32u; q++) {
                    words()[q] = lw[q];
                }
            }
        }
        __syncwarp();
        if (!RECORD && !CKPT && a.resume != 0u) {
            resume(fresh, slot);
            __syncwarp();
        }
        // The node's forces in muscle order: a muscle acts on a0 and a1 with
        // 1 - anchor_a and anchor_a, on b0 and b1 with minus the same of
        // anchor_b. A weight of zero adds a zero, which changes no sum but
        // with an infinite force, and is left out here (see gather()).
        unsigned mine = 0u;
        if (fresh && has_node()) {
            for (unsigned k = 0u; k < r.muscles; k++) {
                mine += entries_of(k, [](float) {});
            }
        }
        unsigned upto = mine;
        for (unsigned o = 1u; o < 32u; o <<= 1u) {
            const unsigned x = __shfl_up_sync(kFull, upto, o);
            if (o < T && i >= o) upto += x;
        }
        if (fresh) {
            e0 = upto - mine;
            e1 = upto;
            if (has_node()) {
                unsigned e = e0;
                for (unsigned k = 0u; k < r.muscles; k++) {
                    entries_of(k, [&](float weight) { entry(e++) = make_float2(weight, __uint_as_float(k)); });
                }
            }
        }
        // Levels: an item's is one past the largest of the earlier items that
        // share a node with it.
        const bool bone = fresh && has_bone(), joint = fresh && writes != 0u;
        unsigned level_now = bone ? 1u : 0u, damp_now = joint ? 1u : 0u, anc = 0u;
        const unsigned ends = bone ? (1u << i) | (1u << pivot) : 0u;
        for (unsigned s = 1u; s < T; s++) {
            const unsigned ls = from(level_now, s), ds = from(damp_now, s), as = from(anc, s);
            const unsigned es = from(ends, s), ws = from(writes, s), rs = from(reads, s);
            if (s < i && (es & ends) != 0u) {
                level_now = max(level_now, ls + 1u);
            }
            if (s < i && joint && ws != 0u) {
                if (((ws & reads) | (rs & writes)) != 0u) {
                    anc |= as | (1u << s);
                }
                if ((ws & writes) != 0u) {
                    damp_now = max(damp_now, ds + 1u);
                }
            }
        }
        if (fresh) {
            level = level_now;
            damp_level = damp_now;
            before = anc;
        }
        levels = __reduce_max_sync(kFull, level);
        damp_levels = __reduce_max_sync(kFull, damp_level);
        const unsigned topo = __float_as_uint(ra.x);
        distinct = __all_sync(kFull, !has_joint() || (((topo >> 15u) & 31u) != i &&
                                                      ((topo >> 15u) & 31u) != (topo & 31u) && (topo & 31u) != i));
        __syncwarp();
        if (RECORD) {
            for (unsigned t = 0u; t <= C::settle; t++) {
                record_frame(t, fresh);
            }
        }
    }

    // The state that a lane wrote down (Trial::hand_over) over the start's.
    __device__ __forceinline__ const float* tail_state(unsigned slot) const {
        return a.tail.state + (size_t)slot * tail_floats(a.rows, a.mm);
    }
    __device__ __forceinline__ void resume(bool fresh, unsigned slot) {
        if (!fresh) {
            return;
        }
        const float* s = tail_state(slot);
        if (has_node()) {
            pos(i) = make_float2(s[4u * i], s[4u * i + 1u]);
            vel(i) = make_float2(s[4u * i + 2u], s[4u * i + 3u]);
        }
        s += 4u * a.rows;
        for (unsigned k = i; k < r.muscles; k += T) {
            store(k).x = s[2u * k];
            offset(k) = s[2u * k + 1u];
        }
        s += 2u * a.mm;
        for (unsigned q = i; q < 32u; q += T) {
            words()[q] = s[q];
        }
        r.step = __float_as_uint(s[33]);
    }

    // Calls `put(weight)` for each weight of muscle k that acts on node i, in
    // the pass's order, but for zeros; returns how many.
    template <class F>
    __device__ __forceinline__ unsigned entries_of(unsigned k, F&& put) const {
        const float4 q0 = pull0(k);
        const unsigned nodes = __float_as_uint(q0.x);
        unsigned n = 0u;
        const float weights[4] = {1.0f - q0.y, q0.y, -(1.0f - q0.z), -q0.z};
#pragma unroll
        for (unsigned e = 0u; e < 4u; e++) {
            if (((nodes >> (8u * e)) & 255u) == i && weights[e] != 0.0f) {
                put(weights[e]);
                n++;
            }
        }
        return n;
    }

    // Frame t of a recording (Trial::record_frame), on the teams with `on`.
    __device__ __forceinline__ void record_frame(unsigned t, bool on) const {
        const unsigned long long broken = broken_joints();
        if (!on) {
            return;
        }
        const unsigned stride = f.p.stride;
        const size_t k = a.count;
        float2* fr = a.frames + (size_t)t * stride * k + r.rec_slot;
        if (has_node()) {
            fr[i * k] = pos(i);
            fr[(CE_MAX_NODES + r.muscles + i) * k] = shown_force;
        }
        for (unsigned m = i; m < r.muscles; m += T) {
            fr[(CE_MAX_NODES + m) * k] = make_float2(store(m).x, shown(m));
        }
        if (i == 0u) {
            fr[(stride - 1u) * k] =
                make_float2(__uint_as_float((unsigned)broken), __uint_as_float((unsigned)(broken >> 32)));
        }
    }

    // Checkpoint n of the creature (Trial::save_checkpoint).
    __device__ __forceinline__ void save_checkpoint(unsigned n) const {
        const size_t count = a.count;
        float* c = a.ckpt + (size_t)n * checkpoint_floats(a.rows, a.mm) * count + r.cidx;
        if (has_node()) {
            const float2 p = pos(i), v = vel(i);
            __stcs(c + (2u * i) * count, p.x);
            __stcs(c + (2u * i + 1u) * count, p.y);
            __stcs(c + (2u * a.rows + 2u * i) * count, v.x);
            __stcs(c + (2u * a.rows + 2u * i + 1u) * count, v.y);
        }
        for (unsigned k = i; k < r.muscles; k += T) {
            __stcs(c + (4u * a.rows + k) * count, store(k).x);
        }
    }

    __device__ __forceinline__ bool has_joint() const { return __float_as_uint(ra.x) != kNone; }
    // The joint of this lane from the positions in shared memory, its angle,
    // and how far that is past its range (0 within it).
    __device__ __forceinline__ Joint joint() const {
        const unsigned topo = __float_as_uint(ra.x);
        return P::joint_at(i - 1u, ra, rb, pos((topo >> 5u) & 31u), pos((topo >> 10u) & 31u), pos(i),
                           pos(topo & 31u));
    }
    __device__ __forceinline__ float angle() const {
        const unsigned topo = __float_as_uint(ra.x);
        return P::angle_at(ra, pos((topo >> 5u) & 31u), pos((topo >> 10u) & 31u), pos(i), pos(topo & 31u));
    }
    __device__ __forceinline__ float joint_error() const {
        const float x = angle();
        float error = 0.0f;
        if (x < ra.y) {
            error = x - ra.y;
        }
        if (x > ra.z) {
            error = x - ra.z;
        }
        return error;
    }
    // Moves the joint's three nodes in `table` along its gradients.
    __device__ __forceinline__ void push(const Joint& k, float lambda, float2* table) const {
        float2& tip = table[k.tip];
        float2& far = table[k.far];
        float2& hub = table[k.hub];
        float2 e = tip;
        if (!distinct) {
            // Two of the three may be one node: one after the other.
            tip = make_float2(__fmaf_rn(__fmul_rn(k.w_tip, lambda), k.g_tip.x, e.x),
                              __fmaf_rn(__fmul_rn(k.w_tip, lambda), k.g_tip.y, e.y));
            e = far;
            far = make_float2(__fmaf_rn(__fmul_rn(k.w_far, lambda), k.g_far.x, e.x),
                              __fmaf_rn(__fmul_rn(k.w_far, lambda), k.g_far.y, e.y));
            e = hub;
            hub = make_float2(__fmaf_rn(__fmul_rn(k.w_hub, lambda), k.g_hub.x, e.x),
                              __fmaf_rn(__fmul_rn(k.w_hub, lambda), k.g_hub.y, e.y));
            return;
        }
        float2 g = far, h = hub;
        e.x = __fmaf_rn(__fmul_rn(k.w_tip, lambda), k.g_tip.x, e.x);
        e.y = __fmaf_rn(__fmul_rn(k.w_tip, lambda), k.g_tip.y, e.y);
        g.x = __fmaf_rn(__fmul_rn(k.w_far, lambda), k.g_far.x, g.x);
        g.y = __fmaf_rn(__fmul_rn(k.w_far, lambda), k.g_far.y, g.y);
        h.x = __fmaf_rn(__fmul_rn(k.w_hub, lambda), k.g_hub.x, h.x);
        h.y = __fmaf_rn(__fmul_rn(k.w_hub, lambda), k.g_hub.y, h.y);
        tip = e;
        far = g;
        hub = h;
    }

    // Bits of the joints past their range (Creature::broken_joints), from the
    // positions in shared memory.
    __device__ __forceinline__ unsigned long long broken_joints() const {
        bool broken = false;
        if (has_joint()) {
            const float x = angle();
            broken = x < ra.y - kJointBreak || x > ra.z + kJointBreak;
        }
        return (unsigned long long)(votes(broken) >> 1u);
    }

    // Each muscle's demand for the step (Creature::muscle_demands).
    __device__ __forceinline__ void demands(float t_now) const {
        if (r.nodes == 0u) {
            return;
        }
        const float4* mus = reinterpret_cast<const float4*>(a.muscles + rhythm_at);
        for (unsigned k = i; k < r.muscles; k += T) {
            store(k).y = f.demand_at(t_now, __ldg(mus + 5u * k + 2u), __ldg(mus + 5u * k + 3u), offset(k));
        }
    }

    // The muscles' forces (Creature::muscle_forces), from the state in shared
    // memory, into `sum`, this lane's node's.
    __device__ __forceinline__ float2 muscles() const {
        bool finite = true;
        for (unsigned k = i; k < r.muscles; k += T) {
            const float4 q0 = pull0(k);
            const unsigned nodes = __float_as_uint(q0.x);
            const float2 ms = store(k);
            const auto at = [&](unsigned n) {
                const float2 x = pos(n), u = vel(n);
                return make_float4(x.x, x.y, u.x, u.y);
            };
            const typename P::Pull g = f.muscle_at(q0, pull1(k), ms, at(nodes & 255u), at((nodes >> 8u) & 255u),
                                                   at((nodes >> 16u) & 255u), at(nodes >> 24u));
            store(k).x = g.energy;
            force(k) = make_float2(g.fx, g.fy);
            if (RECORD) {
                shown(k) = g.pull;
            }
            finite = finite && fabsf(g.fx) < 1e38f && fabsf(g.fy) < 1e38f;
        }
        const bool all_finite = __all_sync(kFull, finite);
        __syncwarp();
        float2 sum = make_float2(0.0f, 0.0f);
        if (all_finite) {
            for (unsigned e = e0; e < e1; e++) {
                const float2 w = entry(e);
                const float2 g = force(__float_as_uint(w.y));
                sum.x = __fmaf_rn(g.x, w.x, sum.x);
                sum.y = __fmaf_rn(g.y, w.x, sum.y);
            }
        } else if (has_node()) {
            // An infinite force times a weight of zero is no zero: all four
            // weights of every muscle.
            for (unsigned k = 0u; k < r.muscles; k++) {
                const float4 q0 = pull0(k);
                const unsigned nodes = __float_as_uint(q0.x);
                const float2 g = force(k);
                const float weights[4] = {1.0f - q0.y, q0.y, -(1.0f - q0.z), -q0.z};
                for (unsigned e = 0u; e < 4u; e++) {
                    if (((nodes >> (8u * e)) & 255u) == i) {
                        sum.x = __fmaf_rn(g.x, weights[e], sum.x);
                        sum.y = __fmaf_rn(g.y, weights[e], sum.y);
                    }
                }
            }
        }
        return sum;
    }

    // A pass over the bones in their order, each updating its two ends' values
    // in `table`: `item(x0, x1)` on the pivot's and the node's.
    template <class F>
    __device__ __forceinline__ void bones(float2* table, F&& item) const {
        float2& pivot = table[__float_as_uint(ba.x) & 31u];
        for (unsigned l = 1u; l <= levels; l++) {
            if (level == l) {
                float2 x0 = pivot, x1 = table[i];
                item(x0, x1);
                pivot = x0;
                table[i] = x1;
            }
            __syncwarp();
        }
    }

    // What the reverse of a substep reads of this lane's node, bone and joint:
    // the values that each sequential pass saw, the muscles' force and the
    // contact.
    struct Kept {
        float2 pulls, landing;           // muscle force; position before the ground pass
        float2 drag0, drag1, bone0, bone1;  // the bone's ends before its drag and its projection
        float2 pt, pp, ct, ch;           // positions that the joint's push saw
        float2 vt, vf, vh;               // velocities that its damping saw
        Joint k;                         // its damping's gradients and
        float wgt;                       // their weight
        bool pushed, touched, slid;
    };

    // One substep (Creature::substep). The positions and velocities are in
    // shared memory at its start and end. `KEEP`: what the reverse reads goes
    // to `kept`.
    template <bool KEEP = false>
    __device__ __forceinline__ void substep(Kept* kept = nullptr) {
        const float2 pulls = muscles();
        if (KEEP) {
            kept->pulls = pulls;
            kept->pushed = kept->touched = kept->slid = false;
        }
        const bool node = has_node();
        const float2 start = node ? pos(i) : make_float2(0.0f, 0.0f);
        // Drag.
        typename P::Wet wet{0.0f, 0.0f, 0.0f};
        if (f.w.has(CE_FLAG_WATER)) {
            const unsigned pivot = has_bone() ? __float_as_uint(ba.x) : 0u;
            const float r0 = from(nr.z, pivot);
            if (has_bone()) {
                wet = f.wet_at(ba, r0, nr.z, pos(pivot), start);
            }
        }
        bones(&vel(0u), [&](float2& v0, float2& v1) {
            if (KEEP) {
                kept->drag0 = v0;
                kept->drag1 = v1;
            }
            f.drag_at(bb, wet, v0, v1);
        });
        // World forces, velocities and predicted positions.
        if (node) {
            const float2 v = vel(i);
            float4 s = make_float4(start.x, start.y, v.x, v.y);
            f.integrate_at(i, nr, pulls, s);
            pos(i) = make_float2(s.x, s.y);
        }
        __syncwarp();
        bones(&pos(0u), [&](float2& p0, float2& p1) {
            if (KEEP) {
                kept->bone0 = p0;
                kept->bone1 = p1;
            }
            P::bone_at(ba, p0, p1);
        });
        // Joint ranges.
        bool open = has_joint();
        for (;;) {
            // A NaN angle gives no error, as in the serial pass.
            const float error = open ? joint_error() : 0.0f;
            const unsigned past = __ballot_sync(kFull, error != 0.0f);
            if (past == 0u) {
                break;
            }
            if (open && (before & (past >> base)) == 0u) {
                if (error != 0.0f) {
                    const Joint k = joint();
                    const float wgt = P::joint_weight(k);
                    if (wgt > 0.0f) {
                        if (KEEP) {
                            const unsigned topo = __float_as_uint(ra.x);
                            kept->pushed = true;
                            kept->pt = pos((topo >> 5u) & 31u);
                            kept->pp = pos((topo >> 10u) & 31u);
                            kept->ct = pos(i);
                            kept->ch = pos(topo & 31u);
                        }
                        push(k, -error / wgt, &pos(0u));
                    }
                }
                open = false;
            }
            __syncwarp();
        }
        // Ground contact and the velocity of the move.
        if (node) {
            float2 p = pos(i);
            float depth, back;
            bool slid;
            if (KEEP) {
                kept->landing = p;
            }
            if (f.ground_at(nr, p, start, depth, back, slid)) {
                if (KEEP) {
                    kept->touched = true;
                    kept->slid = slid;
                }
                if (RECORD) {
                    shown_force.x += nr.x * depth * C::inv_h * C::inv_h;
                    shown_force.y += nr.x * back * C::inv_h * C::inv_h;
                }
            }
            pos(i) = p;
            vel(i) = make_float2((p.x - start.x) * C::inv_h, (p.y - start.y) * C::inv_h);
        }
        __syncwarp();
        // Damping.
        const float share = fminf(C::h * kInvJointDamping, 1.0f);
        Joint k;
        float wgt = 0.0f;
        if (has_joint()) {
            k = joint();
            wgt = P::joint_weight(k);
        }
        for (unsigned l = 1u; l <= damp_levels; l++) {
            if (damp_level == l) {
                const float2 vt = vel(k.tip), vf = vel(k.far), vh = vel(k.hub);
                if (KEEP) {
                    kept->vt = vt;
                    kept->vf = vf;
                    kept->vh = vh;
                }
                const float rate = P::joint_rate(k, vt, vf, vh);
                if (wgt > 0.0f) {
                    push(k, __fmul_rn(-share, rate) / wgt, &vel(0u));
                }
            }
            __syncwarp();
        }
        if (KEEP) {
            kept->k = k;
            kept->wgt = wgt;
        }
    }

    // What score() reads and writes, for the team's first lane.
    struct Words {
        const Team& t;
        unsigned& down;
        __device__ __forceinline__ float2 pos(unsigned n) const { return t.pos(n); }
        __device__ __forceinline__ float energy(unsigned k) const { return t.store(k).x; }
        __device__ __forceinline__ void load(float* lw) const {
#pragma unroll
            for (unsigned q = 0u; q < 32u; q++) {
                lw[q] = t.words()[q];
            }
        }
        __device__ __forceinline__ void store(const float* lw) const {
#pragma unroll
            for (unsigned q = 0u; q < 32u; q++) {
                t.words()[q] = lw[q];
            }
        }
        __device__ __forceinline__ void touchdown(unsigned nodes, float) const { down = nodes; }
        __device__ __forceinline__ void keep(const float* m) const {
            for (unsigned q = 0u; q < 19u; q++) {
                t.kept()[q] = m[q];
            }
        }
    };

    // One step of every team's creature (Trial::step); `live` teams whose
    // trial ends return false.
    __device__ __forceinline__ bool step(bool live) {
        const float t_now = __fmul_rn((float)r.step, C::dt);
        shown_force = make_float2(0.0f, 0.0f);
        if (CKPT && live && (r.step & 15u) == 0u) {
            save_checkpoint(r.step >> 4u);
        }
        demands(t_now);
        __syncwarp();
        for (unsigned s = 0u; s < 16u; s++) {
            substep();
        }
        if (RECORD) {
            shown_force.x *= 1.0f / 16u;
            shown_force.y *= 1.0f / 16u;
        }
        // The step's tallies: the nodes' tests on their lanes, the sums in
        // node order on the first.
        const bool broken = broken_joints() != 0ull;
        const bool node = has_node();
        const float2 p = node ? pos(i) : make_float2(0.0f, 0.0f);
        const bool failed = votes(!(fabsf(p.x) <= 1e6f && fabsf(p.y) <= 1e6f)) != 0u;
        bool touches = false, lifts = false;
        if (node && f.w.has(CE_FLAG_GROUND)) {
            const float2 g = ground_tally(f.w, p.x, r.amp, r.qphase, f.p);
            const float floor_y = __fmaf_rn(nr.z, sqrtf(__fmaf_rn(g.y, g.y, 1.0f)), g.x);
            touches = p.y <= floor_y + kContactSlack;
            lifts = p.y > floor_y + kLiftClearance;
        }
        const unsigned touching = votes(touches), lifted = votes(lifts);
        unsigned down = 0u;
        bool over = false;
        if (live && i == 0u) {
            Tally y{failed, 0.0f, 0.0f, 1e20f, -1e20f, touching, lifted};
            for (unsigned n = 0u; n < r.nodes; n++) {
                const float2 q = pos(n), mr = tally_of(n);
                y.center_y += q.y;
                y.com_x += mr.x * q.x;
                y.low = fminf(y.low, q.y - mr.y);
                y.high = fmaxf(y.high, q.y + mr.y);
            }
            over = score<RECORD, CKPT, RATE>(Words{*this, down}, r, a, f.p, y, broken);
        }
        __syncwarp();
        down = from(down, 0u);
        over = from(over ? 1u : 0u, 0u) != 0u;
        if (RECORD) {
            r.limp = from(r.limp ? 1u : 0u, 0u) != 0u;
            r.scoring = from(r.scoring ? 1u : 0u, 0u) != 0u;
        }
        if (live && down != 0u) {
            // Touch sensors among the nodes `down` restart their muscles.
            const float next = t_now + C::dt;
            const float4* mus = reinterpret_cast<const float4*>(a.muscles + rhythm_at);
            for (unsigned k = i; k < r.muscles; k += T) {
                const unsigned sensor = __float_as_uint(__ldg(mus + 5u * k + 4u).x);
                if (sensor != kNone && ((down >> sensor) & 1u)) {
                    const float4 r0 = __ldg(mus + 5u * k + 2u), r1 = __ldg(mus + 5u * k + 3u);
                    offset(k) = fracf(r1.w - (next * r0.y + r0.z));
                }
            }
        }
        if (RECORD) {
            record_frame(C::settle + r.step + 1u, live);
            if (live && r.step + 1u >= f.p.steps) {
                if (i == 0u) {
                    float* out = reinterpret_cast<float*>(a.results + r.cidx);
                    for (unsigned q = 0u; q < 19u; q++) {
                        out[q] = kept()[q];
                    }
                }
                over = true;
            }
        }
        r.step++;
        __syncwarp();
        return live && !over;
    }
};

template <class W, bool RECORD, int RATE, bool CKPT>
__global__ void __launch_bounds__(kTeamBlock, kTeamMinBlocks) team_kernel(const KernelArgs a, const ce_params p,
                                                                          const W w, unsigned warp_bytes) {
    extern __shared__ float4 smem[];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5u;
    LaneRegs r;
    const Physics<W, RATE> f{w, p, r};
    Team<W, RECORD, RATE, CKPT> t{f, a, r};
    TeamClaim claim(a, lane, warp, gridDim.x * (blockDim.x >> 5u));
    char* const mem = reinterpret_cast<char*>(smem) + (threadIdx.x >> 5u) * warp_bytes;
    t.place(lane, claim.lanes, mem);
    bool live = false;
    for (;;) {
        const unsigned got = claim.next(!live && t.i == 0u);
        const unsigned mine = __shfl_sync(kFull, got, t.base);
        const bool fresh = !live && mine != kNone;
        if (__any_sync(kFull, fresh)) {
            unsigned cidx = 0u, slot = mine;
            if (fresh && a.resume != 0u) {
                slot = a.tail.order[mine];
                cidx = __float_as_uint(t.tail_state(slot)[4u * a.rows + 2u * a.mm + 32u]);
            } else if (fresh) {
                cidx = a.order ? __ldg(a.order + mine) : p.base + mine;
            }
            t.begin(fresh, cidx, slot);
            live = live || fresh;
        }
        if (!__any_sync(kFull, live)) {
            if (!claim.next_group()) {
                break;
            }
            t.place(lane, claim.lanes, mem);
            continue;
        }
        const bool was = live;
        live = t.step(live);
        if (was && !live) {
            t.leave();
        }
    }
}

}  // namespace cek

// The rung audit of one batch on the device, from its resident results:
// Audit::note over every trial (src/rungs.rs:510-525) and GenAudit::of over
// the audit rows (src/rungs.rs:319-345), the rows that record_rungs files
// (src/storage.rs:672-708): trials of creatures flagged AUDIT whose trace is
// not empty, in batch order. Each rung's class A (reached the 5 s bar) and
// class B get Sums::add's float64 sums (src/rungs.rs:286-299) of the six
// features (src/rungs.rs:224-235), and class A's feature words are listed.
//
// The sums are order dependent in float64, so they are added in row order,
// one thread a sum: the rows are first compacted in order (a count and an
// ordered write), then a block a (rung, class) walks them in chunks: 30 warps
// stage the next chunk's features of its class while the first 43 threads add
// one column each (a count, 6 sums, 36 products) of the last one.
// Built with no fused multiply-adds, so every sum equals the reference's to
// the bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "../../include/creature_engine.h"
#include "host_model.h"

namespace {

constexpr uint32_t kAudit = 1u, kExempt = 2u;  // rungs::AUDIT, rungs::EXEMPT (src/rungs.rs:18-22)
constexpr unsigned kFeatures = 6u;
constexpr unsigned kTile = 256u;                 // threads of the count and write kernels
constexpr unsigned kColumns = 1u + kFeatures + kFeatures * kFeatures;  // count, sums, products: 43
constexpr unsigned kAdders = 64u;                // threads of a sum block that add: a column each
constexpr unsigned kChunk = 960u;                // its others, which stage a row each
constexpr unsigned kAhead = 8u;                  // rows whose products are formed ahead of the additions
constexpr unsigned kStaged = (kChunk + kAhead) * (kFeatures + 1u);  // doubles; the last kAhead rows are read, not added
constexpr size_t kSumBytes = 2u * kStaged * sizeof(double);

__device__ __forceinline__ uint32_t bits(float f) { return __float_as_uint(f); }

// The seven trace words of a result (RungTrace, src/creature_kernel.rs:
// 120-218).
struct Trace {
    uint32_t w[7];
    __device__ explicit Trace(const ce_result& r)
        : w{bits(r.contact_hi), bits(r.lift_hi), bits(r.ground_hi), bits(r.previous_center_y),
            bits(r.vertical_extremum), bits(r.vertical_trend), bits(r.gait_turns)} {}
    __device__ uint32_t steps() const { return w[2] >> 16; }
    __device__ uint32_t stopped_by() const { return (w[2] >> 6) & 3u; }
};

// IEEE half to single precision (exact).
__device__ float half_to_float(uint32_t h) {
    const uint32_t sign = (h >> 15) << 31, exponent = (h >> 10) & 0x1fu, mantissa = h & 0x3ffu;
    uint32_t out;
    if (exponent == 0u && mantissa == 0u) {
        out = sign;
    } else if (exponent == 0u) {
        const uint32_t shift = (uint32_t)__clz(mantissa) - 21u;
        out = sign | ((113u - shift) << 23) | (((mantissa << shift) & 0x3ffu) << 13);
    } else if (exponent == 31u) {
        out = sign | 0x7f800000u | (mantissa ? (0x00400000u | (mantissa << 13)) : 0u);
    } else {
        out = sign | ((exponent + 112u) << 23) | (mantissa << 13);
    }
    return __uint_as_float(out);
}

// Single to half precision, rounding to nearest even (the kernel's
// conversion, src/creature_kernel.rs:220-260).
__device__ uint32_t float_to_half(float v) {
    const uint32_t b = __float_as_uint(v);
    const uint32_t sign = (b >> 16) & 0x8000u, mantissa = b & 0x7fffffu;
    const int exponent = (int)((b >> 23) & 0xffu);
    if (exponent == 0xff) return sign | 0x7c00u | (mantissa ? 0x200u : 0u);
    const int e = exponent - 127 + 15;
    if (e >= 31) return sign | 0x7c00u;
    if (e <= 0) {
        if (e < -10) return sign;
        const uint32_t m = mantissa | 0x800000u, shift = (uint32_t)(14 - e);
        const uint32_t half = 1u << (shift - 1u), rest = m & ((1u << shift) - 1u);
        uint32_t out = m >> shift;
        if (rest > half || (rest == half && (out & 1u))) out += 1u;
        return sign | out;
    }
    const uint32_t rest = mantissa & 0x1fffu;
    uint32_t out = ((uint32_t)e << 10) | (mantissa >> 13);
    if (rest > 0x1000u || (rest == 0x1000u && (out & 1u))) out += 1u;
    return sign | out;
}

__device__ __forceinline__ float half_of(uint32_t w, bool high) { return half_to_float(high ? w >> 16 : w & 0xffffu); }

struct Inputs {
    const ce_result* results;
    const ce_genome* genomes;
    const ce_muscle_gene* muscles;
    const float* bars;
    size_t count;
    size_t tile;  // creatures a block of the count and write kernels
};

__device__ __forceinline__ bool is_row(const Inputs& in, size_t i, const Trace& t) {
    return (in.genomes[i].flags & kAudit) != 0u && t.steps() != 0u;
}

// Audit::note's tallies and the audit rows of each block's tile, added up over
// the warp before they meet in shared memory (one 64-bit shared atomic a
// thread and tally had most of the kernel's time: 43 -> 9 us at 300,007).
__global__ void __launch_bounds__(kTile) audit_count_kernel(const Inputs in, uint32_t* tile_rows, ce_audit* out) {
    __shared__ unsigned long long s_steps[kTile / 32u];
    __shared__ unsigned s_counts[4][kTile / 32u];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const size_t lo = (size_t)blockIdx.x * in.tile, hi = min(lo + in.tile, in.count);
    unsigned long long steps = 0ull;
    unsigned counts[4] = {0u, 0u, 0u, 0u};  // stops, rows
    for (size_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const ce_result& r = in.results[i];
        const Trace t(r);
        steps += t.steps();
        if (r.screened > 0.0f) {
            const uint32_t k = t.stopped_by();
            counts[k == 1u ? 0 : (k == 2u ? 1 : 2)] += 1u;
        }
        counts[3] += is_row(in, i, t) ? 1u : 0u;
    }
    for (unsigned d = 16u; d > 0u; d >>= 1) steps += __shfl_down_sync(0xffffffffu, steps, d);
#pragma unroll
    for (unsigned q = 0u; q < 4u; q++) counts[q] = __reduce_add_sync(0xffffffffu, counts[q]);
    if (lane == 0u) {
        s_steps[warp] = steps;
#pragma unroll
        for (unsigned q = 0u; q < 4u; q++) s_counts[q][warp] = counts[q];
    }
    __syncthreads();
    if (threadIdx.x < 5u) {
        unsigned long long all = 0ull;
        for (unsigned v = 0u; v < kTile / 32u; v++) {
            all += threadIdx.x == 4u ? s_steps[v] : (unsigned long long)s_counts[threadIdx.x][v];
        }
        if (threadIdx.x == 3u) {
            tile_rows[blockIdx.x] = (uint32_t)all;
        } else if (all != 0ull) {
            uint64_t* const to = threadIdx.x == 4u ? &out->steps : &out->stops[threadIdx.x];
            atomicAdd(reinterpret_cast<unsigned long long*>(to), all);
        }
    }
}

// Each tile writes its rows' indices in order, behind those of the tiles
// before it, whose counts it adds up itself: a block-wide ordered compaction,
// 256 creatures at a time. The last tile has the batch's totals.
__global__ void __launch_bounds__(kTile) audit_write_kernel(const Inputs in, const uint32_t* tile_rows,
                                                            uint32_t* row_index, ce_audit* out) {
    __shared__ unsigned warp_rows[kTile / 32u];
    __shared__ unsigned base;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned ahead = 0u;
    for (unsigned k = threadIdx.x; k < blockIdx.x; k += blockDim.x) ahead += tile_rows[k];
    ahead = __reduce_add_sync(0xffffffffu, ahead);
    if (lane == 0u) warp_rows[warp] = ahead;
    __syncthreads();
    if (threadIdx.x == 0u) {
        unsigned all = 0u;
        for (unsigned k = 0u; k < blockDim.x / 32u; k++) all += warp_rows[k];
        base = all;
        if (blockIdx.x + 1u == gridDim.x) {
            out->rows = all + tile_rows[blockIdx.x];
            out->creatures = in.count;
        }
    }
    const size_t lo = (size_t)blockIdx.x * in.tile, hi = min(lo + in.tile, in.count);
    for (size_t start = lo; start < hi; start += blockDim.x) {
        const size_t i = start + threadIdx.x;
        const bool row = i < hi && is_row(in, i, Trace(in.results[i]));
        const unsigned ballot = __ballot_sync(0xffffffffu, row);
        __syncthreads();  // `base` and `warp_rows` of the last round are read
        if (lane == 0u) warp_rows[warp] = __popc(ballot);
        __syncthreads();
        unsigned before = base;
        for (unsigned k = 0u; k < warp; k++) before += warp_rows[k];
        if (row) row_index[before + __popc(ballot & ((1u << lane) - 1u))] = (uint32_t)i;
        __syncthreads();
        if (threadIdx.x == 0u) {
            unsigned all = 0u;
            for (unsigned k = 0u; k < blockDim.x / 32u; k++) all += warp_rows[k];
            base += all;
        }
    }
}

// GenAudit::of over the compacted rows, in order, a block a (rung, class).
// Each chunk's rows of the class are staged in row order as float64 with a
// constant 1 behind their features, and thread c < 43 adds its column over
// them: c = 0 the count, 1-6 feature c - 1 times the constant 1 (an exact
// product, so the sum is Sums::add's), 7-42 the product of features
// (c - 7) / 6 and (c - 7) % 6. Every column is one row-ordered chain of
// float64 multiply and add, with no branch on the row.
//
// Bound by the gathers of a row (its index, then its result, genome and bar,
// then its muscle) and by the chain of additions. One block for all four
// groups that staged 256 rows, then added them, took 103 us for 2,344 rows;
// 960 rows at a time, staged while the last ones are added, 50 us, and with
// the next rows' products formed under the chain (8 cycles an addition, 19
// with its loads in line) 25 us. 480 and 256 rows at a time are 2 and 8 us
// slower, products of 4 rows ahead 29 us, of 16 no faster.
__global__ void __launch_bounds__(kAdders + kChunk) audit_sum_kernel(const Inputs in, const uint32_t* row_index,
                                                                     ce_audit* out, uint16_t* a_words, size_t a_cap) {
    extern __shared__ double feat[];  // [2][kChunk + kAhead][kFeatures + 1]
    __shared__ unsigned warp_count[kChunk / 32u], staged[2];
    const unsigned r = blockIdx.x >> 1, k = blockIdx.x & 1u, lane = threadIdx.x & 31u;
    const unsigned col = threadIdx.x;
    const unsigned fa = col == 0u ? kFeatures : (col <= kFeatures ? col - 1u : (col - 1u - kFeatures) / kFeatures);
    const unsigned fb = col <= kFeatures ? kFeatures : (col - 1u - kFeatures) % kFeatures;
    const uint32_t rows = out->rows;
    const uint32_t chunks = rows / kChunk + (rows % kChunk ? 1u : 0u);
    double acc = 0.0;
    unsigned long long n = 0ull;
    uint32_t index = threadIdx.x >= kAdders && threadIdx.x - kAdders < rows ? row_index[threadIdx.x - kAdders] : 0u;
    for (uint32_t c = 0u; c <= chunks; c++) {
        if (threadIdx.x >= kAdders && c < chunks) {
            const unsigned t = threadIdx.x - kAdders, warp = t >> 5;
            const size_t row = (size_t)c * kChunk + t;
            float f[kFeatures] = {};
            bool mine = false;
            if (row < rows) {
                const uint32_t i = index;
                if (row + kChunk < rows) index = row_index[row + kChunk];
                const ce_result& res = in.results[i];
                const Trace tr(res);
                const ce_genome& g = in.genomes[i];
                const float bar = in.bars[i];
                const bool counted = (g.flags & kExempt) == 0u && isfinite(bar);
                const float period = g.muscle_count > 0u ? in.muscles[g.muscle_start].period : 0.0f;
                f[0] = half_of(tr.w[0], r == 1u);
                f[1] = half_of(tr.w[3], r == 1u);
                f[2] = half_of(r == 0u ? tr.w[4] : tr.w[5], false);
                f[3] = half_of(tr.w[6], r == 1u);
                f[4] = half_of(r == 0u ? tr.w[4] : tr.w[5], true);
                f[5] = half_to_float(float_to_half(period));
                bool finite = true;
#pragma unroll
                for (unsigned x = 0u; x < kFeatures; x++) finite = finite && isfinite(f[x]);
                // rungs::RUNG_STEPS: R1 at step 60, R2 at 150.
                mine = counted && tr.steps() > (r == 0u ? 60u : 150u) && finite && (res.screen_x >= bar) == (k == 0u);
            }
            // The class's rows in row order: a ballot a warp, then the
            // counts of the warps before.
            const unsigned ballot = __ballot_sync(0xffffffffu, mine);
            if (lane == 0u) warp_count[warp] = __popc(ballot);
            asm volatile("bar.sync 1, %0;" ::"n"(kChunk) : "memory");
            const unsigned have = lane < kChunk / 32u ? warp_count[lane] : 0u;
            const unsigned all = __reduce_add_sync(0xffffffffu, have);
            const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? have : 0u);
            if (mine) {
                const unsigned j = before + __popc(ballot & ((1u << lane) - 1u));
                double* const to = feat + (c & 1u) * kStaged + j * (kFeatures + 1u);
#pragma unroll
                for (unsigned x = 0u; x < kFeatures; x++) to[x] = (double)f[x];
                to[kFeatures] = 1.0;
                if (k == 0u && a_words && n + j < a_cap) {  // class A's feature words
                    uint16_t* const w = a_words + ((size_t)r * a_cap + n + j) * kFeatures;
#pragma unroll
                    for (unsigned x = 0u; x < kFeatures; x++) w[x] = (uint16_t)float_to_half(f[x]);
                }
            }
            // Rows of zeros fill up the last kAhead: no sum is -0, so they add nothing.
            if (t < kAhead && all + t < (all + kAhead - 1u) / kAhead * kAhead) {
                double* const to = feat + (c & 1u) * kStaged + (all + t) * (kFeatures + 1u);
#pragma unroll
                for (unsigned x = 0u; x <= kFeatures; x++) to[x] = 0.0;
            }
            if (t == 0u) staged[c & 1u] = all;
            n += all;
        } else if (col < kColumns && c > 0u) {
            const unsigned len = staged[(c - 1u) & 1u];
            const double* at = feat + ((c - 1u) & 1u) * kStaged;
            double now[kAhead], next[kAhead];
#pragma unroll
            for (unsigned x = 0u; x < kAhead; x++) now[x] = at[x * (kFeatures + 1u) + fa] * at[x * (kFeatures + 1u) + fb];
            for (unsigned j = 0u; j < len; j += kAhead) {
                at += kAhead * (kFeatures + 1u);
#pragma unroll
                for (unsigned x = 0u; x < kAhead; x++) {
                    next[x] = at[x * (kFeatures + 1u) + fa] * at[x * (kFeatures + 1u) + fb];
                }
#pragma unroll
                for (unsigned x = 0u; x < kAhead; x++) acc += now[x];
#pragma unroll
                for (unsigned x = 0u; x < kAhead; x++) now[x] = next[x];
            }
            n += len;
        }
        __syncthreads();
    }
    if (col < kColumns) {
        ce_audit_sums& s = k == 0u ? out->a[r] : out->b[r];
        if (col == 0u) s.n = n;
        else if (col <= kFeatures) s.sum[col - 1u] = acc;
        else s.xx[(col - 1u - kFeatures) / kFeatures][(col - 1u - kFeatures) % kFeatures] = acc;
    }
}

}  // namespace

extern "C" size_t ce_audit_scratch_bytes(size_t count) {
    return 4096ull * sizeof(uint32_t) + count * sizeof(uint32_t);
}

extern "C" ce_status ce_audit_device(const ce_result* results, const ce_genome* genomes, const ce_muscle_gene* muscles,
                                     const float* bars, size_t count, void* scratch, size_t scratch_bytes,
                                     ce_audit* out, uint16_t* a_words, size_t a_cap, void* stream) {
    if (!out || (count && (!results || !genomes || !muscles || !bars || !scratch))) {
        ce::set_error("ce_audit_device: null argument");
        return CE_ERR_INVALID;
    }
    if (count > 0xffffffffull) {
        ce::set_error("ce_audit_device: at most 2^32 - 1 trials a call");
        return CE_ERR_INVALID;
    }
    if (scratch_bytes < ce_audit_scratch_bytes(count)) {
        ce::set_error("ce_audit_device: scratch smaller than ce_audit_scratch_bytes");
        return CE_ERR_INVALID;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(ce_audit), st);
    if (e != cudaSuccess) {
        ce::set_error(std::string("ce_audit_device: ") + cudaGetErrorString(e));
        return CE_ERR_DEVICE;
    }
    if (count == 0) return CE_OK;  // every tally and sum is zero
    uint32_t* tile_rows = static_cast<uint32_t*>(scratch);
    uint32_t* row_index = tile_rows + 4096;
    const unsigned tiles = (unsigned)std::min<size_t>(148u * 8u, std::max<size_t>(1u, (count + kTile - 1u) / kTile));
    Inputs in{results, genomes, muscles, bars, count, (count + tiles - 1u) / tiles};
    if (in.tile == 0u) in.tile = 1u;
    audit_count_kernel<<<tiles, kTile, 0, st>>>(in, tile_rows, out);
    audit_write_kernel<<<tiles, kTile, 0, st>>>(in, tile_rows, row_index, out);
    e = cudaFuncSetAttribute(audit_sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumBytes);
    if (e == cudaSuccess) {
        audit_sum_kernel<<<4, kAdders + kChunk, kSumBytes, st>>>(in, row_index, out, a_words, a_cap);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        ce::set_error(std::string("ce_audit_device: launch: ") + cudaGetErrorString(e));
        return CE_ERR_DEVICE;
    }
    return CE_OK;
}

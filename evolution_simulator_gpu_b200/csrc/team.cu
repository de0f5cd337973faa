// Plain trials on teams of lanes (team.cuh).
#include "team_launch.cuh"

namespace cek {

cudaError_t launch_team(const TeamSpec& s, const KernelArgs& a, const ce_params& p) {
    return s.rate == 60 ? team_in_world<false, 60>(s, a, p)
           : s.rate == 120 ? team_in_world<false, 120>(s, a, p)
                           : cudaErrorInvalidValue;
}

// Blocks of a launch that would give every creature its team at once.
unsigned team_blocks(unsigned rows, size_t count) {
    // Each team size may leave one warp partly filled.
    const size_t blocks = (count * team_lanes(rows) + 3u * 32u + kTeamBlock - 1u) / kTeamBlock;
    return (unsigned)(blocks < 0x7fffffffu ? blocks : 0x7fffffffu);
}

size_t team_smem_bytes(unsigned first_n, unsigned rows, unsigned mm) {
    KernelArgs a{};
    a.queues = kQueues;
    a.first_n = first_n;
    a.rows = rows;
    a.mm = mm;
    return (size_t)team_warp_bytes(a, false) * (kTeamBlock / 32u);
}

namespace {
size_t align256(size_t b) { return (b + 255u) & ~(size_t)255u; }
}  // namespace

size_t tail_bytes(unsigned rows, unsigned mm, unsigned most) {
    return align256(kTailCounters * 4u) + align256((size_t)3u * most * 4u) +
           align256((size_t)most * tail_floats(rows, mm) * 4u);
}

namespace {
// One warp, a node count a lane. The lanes of a launch hand over when its
// count less the trials that ended is at most tail.most: for a smaller number
// the ended trials start below zero.
__global__ void tail_start_kernel(const Tail tail, const uint32_t* bounds, const unsigned long long* work,
                                  uint32_t count, double budget) {
    const unsigned lane = threadIdx.x;
    double cost = 0.0;
    for (unsigned n = lane; n < kQueues; n += 32u) {
        const double have = bounds[n + 1u] - bounds[n];
        if (have > 0.0 && n >= 2u) {
            const double muscles = ((double)(work[n + 1u] - work[n]) / have - (186.0 * n - 260.0)) / 75.0;
            const double turns = muscles / (n <= 8u ? 8.0 : n <= 16u ? 16.0 : 32.0) + 0.5;
            cost += have * team_cost(n, turns > 1.0 ? turns : 1.0);
        }
    }
    for (unsigned o = 16u; o > 0u; o >>= 1u) cost += __shfl_down_sync(0xffffffffu, cost, o);
    if (lane == 0u) {
        const double fit = budget * (double)count / (cost > 0.0 ? cost : 1.0);
        tail.counters[kTailDone] = fit < (double)tail.most ? (uint32_t)fit - tail.most : 0u;
    } else if (lane < kTailCounters) {
        tail.counters[lane] = 0u;
    }
}
}  // namespace

cudaError_t launch_tail_start(const Tail& tail, const uint32_t* bounds, const unsigned long long* work,
                              uint32_t count, double budget, cudaStream_t stream) {
    tail_start_kernel<<<1, 32, 0, stream>>>(tail, bounds, work, count, budget);
    return cudaGetLastError();
}

Tail tail_layout(void* area, unsigned most) {
    char* p = static_cast<char*>(area);
    Tail t;
    t.counters = reinterpret_cast<uint32_t*>(p);
    p += align256(kTailCounters * 4u);
    t.order = reinterpret_cast<uint32_t*>(p);
    p += align256((size_t)3u * most * 4u);
    t.state = reinterpret_cast<float*>(p);
    t.most = most;
    return t;
}

}  // namespace cek

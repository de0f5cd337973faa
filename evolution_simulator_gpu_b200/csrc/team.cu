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

// The launchers of the team kernels (team.cuh), for the files that compile
// them: plain trials, recordings and checkpointed forward runs.
#pragma once
#include <type_traits>

#include "team.cuh"

namespace cek {

// Shared memory of a warp of a launch whose bodies have first_n to rows nodes.
inline unsigned team_warp_bytes(const KernelArgs& a, bool record) {
    unsigned most = 0u;
    for (unsigned lanes = 8u; lanes <= 32u; lanes *= 2u) {
        const bool used = a.queues == 0u ? lanes == team_lanes(a.rows)
                                         : lanes >= team_lanes(a.first_n) && lanes <= team_lanes(a.rows);
        const unsigned bytes = 32u / lanes * TeamLayout::make(lanes, a.mm, record).bytes;
        if (used && bytes > most) most = bytes;
    }
    return most;
}

template <class W, bool RECORD, int RATE, bool CKPT>
cudaError_t team_occupancy_one(unsigned warp_bytes, int* blocks) {
    auto kern = team_kernel<W, RECORD, RATE, CKPT>;
    const size_t smem = (size_t)warp_bytes * (kTeamBlock / 32u);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kern, (int)kTeamBlock, smem);
}

// Launches the kernel on as many blocks as fit.
template <class W, bool RECORD, int RATE, bool CKPT>
cudaError_t team_one(const W& w, const TeamSpec& s, const KernelArgs& a, const ce_params& p) {
    const unsigned warp_bytes = team_warp_bytes(a, RECORD);
    int per_sm = 0;
    const cudaError_t e = team_occupancy_one<W, RECORD, RATE, CKPT>(warp_bytes, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const unsigned grid = s.blocks < (unsigned)per_sm * s.sms ? s.blocks : (unsigned)per_sm * s.sms;
    team_kernel<W, RECORD, RATE, CKPT>
        <<<grid > 0u ? grid : 1u, kTeamBlock, (size_t)warp_bytes * (kTeamBlock / 32u), s.stream>>>(a, p, w, warp_bytes);
    return cudaGetLastError();
}

template <bool RECORD, int RATE>
cudaError_t team_in_world(const TeamSpec& s, const KernelArgs& a, const ce_params& p) {
    const auto go = [&](auto w) {
        return team_one<decltype(w), RECORD, RATE, false>(w, s, a, p);
    };
    switch (s.flags) {
        case kWorldCalm: return go(StaticWorld<kWorldCalm>{});
        case kWorldEffects: return go(StaticWorld<kWorldEffects>{});
        case kWorldEffectsQuake: return go(StaticWorld<kWorldEffectsQuake>{});
        case kWorldAll: return go(StaticWorld<kWorldAll>{});
        default: return go(RuntimeWorld{s.flags});
    }
}

}  // namespace cek

// Checkpointed forward runs of the gradients' worlds on teams of lanes
// (team.cuh).
#include "team_launch.cuh"

namespace cek {

cudaError_t launch_team_ckpt(const TeamSpec& s, const KernelArgs& a, const ce_params& p) {
    const auto go = [&](auto w) -> cudaError_t {
        if (s.rate == 60) return team_one<decltype(w), false, 60, true>(w, s, a, p);
        if (s.rate == 120) return team_one<decltype(w), false, 120, true>(w, s, a, p);
        return cudaErrorInvalidValue;
    };
    switch (s.flags) {
        case kWorldCalm: return go(StaticWorld<kWorldCalm>{});
        case kWorldEffects: return go(StaticWorld<kWorldEffects>{});
        case kWorldEffectsQuake: return go(StaticWorld<kWorldEffectsQuake>{});
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace cek

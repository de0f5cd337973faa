// Recordings on teams of lanes (team.cuh).
#include "team_launch.cuh"

namespace cek {

cudaError_t launch_team_record(const TeamSpec& s, const KernelArgs& a, const ce_params& p) {
    return s.rate == 60 ? team_in_world<true, 60>(s, a, p)
           : s.rate == 120 ? team_in_world<true, 120>(s, a, p)
                           : cudaErrorInvalidValue;
}

}  // namespace cek

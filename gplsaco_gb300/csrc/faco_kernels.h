// faco_kernels.h -- kernel declarations shared by faco_kernels.cu and the
// host engine.
#pragma once

#include <cstdint>

#include "faco_ant.cuh"
#include "faco_control.cuh"

namespace faco {

// Ants (warps) per block of the ant kernel, and the resident blocks per SM
// the register budget of each variant is sized for.  Panels that fill the GPU
// trade registers for resident warps (72 registers without room to spare: 8
// blocks spill); elsewhere an iteration lasts as long as its slowest ants, and
// the compiler's longer overlaps (up to 96 and 128 registers) pay more than
// warps that are not there.  One GB300, whole runs in ms, by blocks:
//   full panels: 256 x 32 ants at N=1000, 320 iterations, 5 / 6 / 7 / 8: 113.2 /
//     110.6 / 108.6 / 122.9; with Or-opt (more registers), 160 iterations, 4 / 5
//     / 6 / 7: 79.2 / 71.3 / 76.4 / 80.9.
//   others, 4 / 5 / 6 / 7 / 8: the uneven batch (4,096 ant warps, N 200-1000, 400
//     iterations) 87.1 / 81.6 / 86.0 / 91.0 / 109.2, with Or-opt 163.8 / 159.5 /
//     174.5 / 193.6 / 225.6; 128 x 32 at N=1000-2000, 640 iterations, 146.4 /
//     146.3 / 152.0 / 158.2 / 182.9; 32 x 128 at N=537, 100 iterations, 26.0 /
//     25.6 / 27.1 / 28.1 / 30.6; one N=100 colony, 64 iterations, 4.45 / 4.43 /
//     4.60 / 4.79 / 5.01.
//   global-memory workspace: the large panel (80 x 64 ants, N 5000-10000, 80
//     iterations), 2 / 3 / 4 / 5 / 6: 2-opt 61.6 / 53.2 / 53.0 / 59.3 / 63.2, with
//     Or-opt 82.6 / 71.8 / 72.4 / 81.5 / 88.1.
//   FACO_FOLLOW_OFF has no build for full panels: 256 x 32 at N=1000, 320
//     iterations, 4 / 5 / 6 / 7 / 8 blocks 161 / 136-145 / 133.6 / 135.3 / 141.1.
constexpr std::uint32_t kMaxWarpsPerBlock = 4;
constexpr std::uint32_t ant_blocks_per_sm(int mode) {
    return dense_mode(mode) ? (mode & kOrOptOnly ? 5 : 7) : global_mode(mode) || !engine_mode(mode) ? 4 : 5;
}

struct ColonyParams {
    std::uint32_t ants;
    std::uint32_t mne_target;
    double retention;
    float retention_f;
    double p_root;                   // p_best^(1/k), computed once on the host
    double epoch_source_probability;
    std::uint32_t controlled;        // GP controllers choose MNE, start region and restarts
    std::uint32_t total_iterations;  // T of the evaluation (iteration-fraction feature)
    float log2k;                     // log2(k) by the engine's own log2
    std::uint32_t ref_control;       // 1: the 12-feature controller (feature spec 2)
    std::uint32_t zero_fingerprints; // diagnostic: every tour fingerprint 0 (forced collisions)
    unsigned long long ls_limit;     // LS evaluation budget per ant (LS-work feedback)
    DecisionCapture capture;         // decisions to record (count 0: none)
    const std::uint32_t* prior_rows; // per colony: 1 = the prior re-ranks departures only (device; may be null)
    std::uint32_t trail_blocks;      // > 1: colony_trails_kernel updates the trails with this many blocks per
                                     // colony, after the colony update (uncontrolled evaluations only)
};

// Candidate rows of registration on the GPU (faco_knn.cu): per node its
// `needed` nearest nodes in (EUC_2D length, id) order, ids and lengths
// [n][needed]; needed <= kKnnMaxNeeded and < n, shared memory 8 n bytes.
constexpr std::uint32_t kKnnMaxNeeded = 256;
std::uint32_t knn_smem_bytes(std::uint32_t n);
cudaError_t launch_knn(const int2* xy, std::uint32_t n, std::uint32_t needed, node_t* near_ids,
                       std::int32_t* near_dist, cudaStream_t stream);

// Host-side launchers (the kernels are defined in faco_kernels.cu).
cudaError_t prepare_ant_kernel(int mode, std::uint32_t ls_mode, std::uint32_t smem_bytes);
// (`overlapped`: the kernel's prologue may start while the kernel before it on
// the stream still runs)
cudaError_t launch_ant_kernel(int mode, const AntLaunch& L, std::uint32_t blocks, std::uint32_t warps,
                              std::uint32_t smem_bytes, cudaStream_t stream, bool overlapped = false);

__global__ void colony_init_kernel(const InstanceView* instances, const ColonyView* colonies, ColonyState* states,
                                   ColonyParams P, std::uint32_t colony_count);
__global__ void prior_rows_kernel(const InstanceView* instances, const ColonyView* colonies,
                                  const std::uint32_t* modes);
__global__ void fingerprint_kernel(const ColonyView* colonies, const std::uint32_t* list, std::uint32_t ants,
                                   std::uint32_t colony_count, std::uint32_t zero);
// colony_update_kernel of `blocks` colonies (those of `list`, or all when null)
cudaError_t launch_colony_update(const InstanceView* instances, const ColonyView* colonies, ColonyState* states,
                                 const ColonyParams& P, TraceRow* trace, const std::uint32_t* list,
                                 std::uint32_t blocks, std::uint32_t colony_count, std::uint32_t trace_cap,
                                 cudaStream_t stream, bool overlapped = false);
__global__ void colony_trails_kernel(const InstanceView* instances, const ColonyView* colonies,
                                     const ColonyState* states, ColonyParams P, const std::uint32_t* list);
__global__ void pheromone_step_kernel(std::uint32_t n, std::uint32_t k, const node_t* primary,
                                      const std::uint32_t* parent_nbr, float ret, float tmin, float tmax, float inc,
                                      const float* eta, float* trails, float* products);
// (one warp per colony, four per block; kErrFeature in *error where a feature is outside [0, 1])
__global__ void score_controllers_kernel(const Program* trees, const std::uint32_t* kinds, std::uint32_t replicas,
                                         const float* features, const std::uint32_t* masks, float* scores,
                                         std::int32_t* actions, std::uint32_t colonies, unsigned* error);
__global__ void score_kernel(const Program* programs, std::uint32_t replicas, const float* features,
                             const std::uint32_t* masks, float* scores, std::int32_t* actions,
                             std::uint32_t colonies, unsigned* error);

}  // namespace faco

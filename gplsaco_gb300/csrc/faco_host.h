// faco_host.h -- host-side helpers of the engine (no CUDA types).
#pragma once

#include <cstdint>
#include <vector>

namespace faco {

float host_log2(float x);
void host_regions(const std::vector<std::int32_t>& xy, std::uint32_t n, std::uint32_t offsets[5],
                  std::vector<std::uint16_t>& list);
std::int32_t host_euc2d(std::int64_t x0, std::int64_t y0, std::int64_t x1, std::int64_t y1);
std::int64_t host_tour_length(const std::vector<std::int32_t>& xy, const std::uint32_t* order, std::uint32_t n);
void host_candidates(const std::vector<std::int32_t>& xy, std::uint32_t n, std::uint32_t k, std::uint32_t b,
                     std::uint32_t w, std::vector<std::uint16_t>& primary, std::vector<std::uint16_t>& backup,
                     std::vector<std::uint16_t>& ls, std::vector<std::int32_t>& ls_dist, std::vector<float>& eta,
                     double beta);
std::vector<std::uint32_t> host_nearest_neighbour_tour(const std::vector<std::int32_t>& xy, std::uint32_t n);
// Rows and eta from sorted near lists ([n][needed] ids and lengths).
void host_rows_from_near(const std::vector<std::uint16_t>& near, const std::vector<std::int32_t>& near_dist,
                         std::uint32_t n, std::uint32_t needed, std::uint32_t k, std::uint32_t b, std::uint32_t w,
                         double beta, std::vector<std::uint16_t>& primary, std::vector<std::uint16_t>& backup,
                         std::vector<std::uint16_t>& ls, std::vector<std::int32_t>& ls_dist, std::vector<float>& eta);
// The nearest-neighbour tour using the near lists; a full scan only when
// every listed node is already visited.
std::vector<std::uint32_t> host_nearest_neighbour_tour_near(const std::vector<std::int32_t>& xy, std::uint32_t n,
                                                            const std::vector<std::uint16_t>& near,
                                                            std::uint32_t needed);
// Alpha-nearness (length minus the longest edge on the minimum spanning
// tree path between the ends) of every primary candidate entry, [n][k].
void host_alpha(const std::vector<std::int32_t>& xy, std::uint32_t n, std::uint32_t k,
                const std::vector<std::uint16_t>& primary, std::uint32_t b, const std::vector<std::uint16_t>& backup,
                std::uint32_t w, const std::vector<std::uint16_t>& ls, std::vector<float>& alpha);
void host_distance_order(const std::vector<std::int32_t>& xy, std::uint32_t n, std::uint32_t w,
                         const std::uint32_t* rows, std::vector<std::uint16_t>& ls,
                         std::vector<std::int32_t>& ls_dist);
// The inverse of a tour (n below 65535): inverse[order[i]] = i.  False where
// `order` is not a permutation of 0 .. n-1.
bool host_inverse(const std::uint16_t* order, std::uint32_t n, std::uint16_t* inverse);
// Construction steps per ant and iteration of a colony's run so far: what a
// restored colony starts from in place of its last iteration's walk, which a
// snapshot does not hold.
std::uint32_t host_mean_walk(std::uint64_t construction_steps, std::uint32_t iterations, std::uint32_t ants);

// The construction steps per ant from which a colony takes parent-following
// steps in batches (FACO_FOLLOW_AUTO), as walked in its last iteration (the
// ant kernel reads it); below, the batches' setup costs more than the few
// steps they take at once.  A line per launch, by the placement of its own
// ants: one line for all, the highest, kept the small instances of a mixed
// panel on single steps (256 x 32 ants of N 500-2500, 200 iterations: 115.4
// ms, now 113.4).  Measured in us per iteration, one at a time / in
// batches: the uneven batch (4,096 ant warps) 179 / 211 at 23 steps, 224 /
// 226 at 31, 297 / 251 at 44; 256 x 32 ants at N=1000 340 / 416 at 33 steps,
// 438 / 448 at 51, 601 / 500 at 80; the large panel in the global-memory
// workspace (2-opt) 1814 / 1857 at 54, 2195 / 1994 at 80.  The curves are flat
// near the lines; all three moved by a fifth down / up / by half up: the uneven
// batch (400 iterations) 81.3 / 82.2 / 83.6 ms against 81.6, 128 x 32 ants at
// N=1000-2000 145.3 / 147.5 / 149.4 against 146.3, 256 x 32 at N=1000 108.2 /
// 110.1 / 112.4 against 108.6, the large panel 52.8 / 52.7 / 53.1 against 53.0.
constexpr std::uint32_t kBatchFromOneWave = 30, kBatchFromFull = 48, kBatchFromGlobal = 60;
// `always`: FACO_FOLLOW_ON; `full`: more ant warps than one wave of the GPU.
constexpr std::uint32_t host_batch_from(bool always, bool full, bool global_workspace) {
    return always ? 0u : global_workspace ? kBatchFromGlobal : full ? kBatchFromFull : kBatchFromOneWave;
}

// The factor on a class's time with its ants in shared memory, against the
// global-memory workspace, when the tuner compares the two: it times a class
// alone, from the initial tours, and a full panel's other chains change which
// is faster.  By the blocks of four ants that fit on an SM (228 KB, 1 KB of it
// the driver's per block):
//   3 and more (N up to about 3,300): nearly as many ants as the workspace's
//     registers admit, without its L2 reads.  60 iterations of 80 x 64 ants at
//     N=2200 / 2600 / 3000: 12.3 / 14.8 / 15.7 ms in shared memory, 17.8 / 19.0
//     / 19.9 in the workspace; the ants above N=2048 of 256 x 32 with N 500-2500
//     timed the same in both, and the panel ran 81 or 115 ms.
//   2: alike in a panel of one size (N=3500 / 4000 / 4500: 21.4 / 22.8 / 23.7 ms,
//     in the workspace 21.2 / 22.3 / 24.0); 120 x 64 ants of N 3773-4485, timed
//     faster in shared memory, ran 37.3 instead of 32.4 ms.
//   1 (N from about 4,600 on): a block holds the SM.  At N 5000-8166 (40
//     colonies x 64 ants) shared memory timed 0-11 % faster than the workspace
//     in five panels, and the two panels that took it ran 120 instead of 107 ms.
constexpr float host_shared_factor(bool full, std::uint32_t block_bytes) {
    return !full ? 1.0f : 3 * (block_bytes + 1024u) <= 228u * 1024u ? 0.8f : 1.15f;
}

}  // namespace faco

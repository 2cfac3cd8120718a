// faco_common.cuh -- device types and primitives shared by the FACO kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace faco {

using node_t = std::uint16_t;   // node ids on the device (n <= 65535)
constexpr std::uint32_t kMaxNodes = 65535;
constexpr std::uint32_t kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// Device error word bits (the host turns a non-zero word into FACO_EDEVICE).
enum DeviceError : unsigned {
    kErrNone = 0,
    kErrQueueOverflow = 1u << 0,
    kErrBadChoice = 1u << 1,
    kErrLoopCap = 1u << 2,
    kErrShape = 1u << 3,
    kErrTensorWait = 1u << 4,   // a tcgen05 MMA completion wait ran out
    kErrFeature = 1u << 5,      // a controller feature outside [0, 1]
};

// TSPLIB EUC_2D: round(sqrt(dx^2+dy^2)) with halves up.  sqrt(s) is never a
// half-integer for integer s, so the result is the unique m with
// m*m - m < s <= m*m + m (m > 0) -- found from an FP32 estimate and at most
// a few exact int64 corrections.  Equal to floor(sqrt((double)s) + 0.5)
// for lengths below 2^25, which covers every instance registration admits
// (coordinate spans below 2^24 per axis).
// The estimate comes from 32-bit dx, dy in FP32 (GB300 runs 64-bit
// integer/float conversions on its narrow FP64 pipe, so none are used) and is
// within 7 of the length (relative error below 2^-21.5, lengths below
// 2^24.5), so the residual t = s - m^2 fits 32 bits and is exact in modular
// arithmetic.  t decides the length when the estimate is off by at most one:
// m + 1 when t > m, m - 1 when t <= -m.  Estimates further off (lengths above
// about 2^21) take the 64-bit loops.  Lengths of 10^4 to 10^5 miss by one in
// 1-5 % of the pairs, so in a warp of 32 lanes every other call: correcting in
// line took the N=1000 panel (256 x 32 ants, 320 iterations) from 124.5 to
// 122.8 ms.
__device__ __forceinline__ float sqrt_estimate(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ int euc2d(int2 p, int2 q) {
    const int dx = p.x - q.x, dy = p.y - q.y;  // |dx|, |dy| < 2^27
    const float fx = (float)dx, fy = (float)dy;
    const int m = __float2int_rn(sqrt_estimate(fx * fx + fy * fy));
    const int t = (int)((unsigned)dx * (unsigned)dx + (unsigned)dy * (unsigned)dy - (unsigned)m * (unsigned)m);
    int r = m + (t > m ? 1 : 0) - (t <= -m ? 1 : 0);
    // off by at most one: -3 m + 3 <= t <= 3 m + 2
    if ((unsigned)(t + 3 * m - 3) >= (unsigned)(6 * m)) {
        const long long s = (long long)dx * dx + (long long)dy * dy;
        r = m;
        while (s > (long long)r * r + r) ++r;
        while (r > 0 && s <= (long long)r * r - r) --r;
    }
    return r;
}

// Programmatic dependent launch: lets the next kernel of the stream start its
// prologue now; waits until the previous one is complete and its writes are
// visible.  Both without effect in an ordinary launch.
__device__ __forceinline__ void start_next_kernel() {
#ifdef __CUDACC__
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}
__device__ __forceinline__ void wait_previous_kernel() {
#ifdef __CUDACC__
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// A load of what another kernel of the stream writes while this one may already
// be resident (a colony's parent, neighbours and products).  Not by __ldg: that
// is for memory constant over the kernel's life, so it may move above
// wait_previous_kernel() and need not see the writes.
template <class T>
__device__ __forceinline__ T load_written(const T* p) {
#ifdef __CUDACC__
    __builtin_assume(__isGlobal(p));   // ld.global, not a generic load
#endif
    return *p;
}

// Philox4x32 with 10 rounds (Salmon, Moraes, Dror, Shaw, SC'11).
struct uint4v { std::uint32_t x, y, z, w; };
__device__ __forceinline__ uint4v philox4x32(std::uint32_t c0, std::uint32_t c1, std::uint32_t c2,
                                             std::uint32_t c3, std::uint32_t k0, std::uint32_t k1) {
#pragma unroll
    for (int round = 0; round < 10; ++round) {
        const std::uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const std::uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        c0 = hi1 ^ c1 ^ k0; c1 = lo1; c2 = hi0 ^ c3 ^ k1; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return {c0, c1, c2, c3};
}

// The same generator with its rounds in a loop: fewer instructions in the
// code, for call sites where code size matters more than the loop overhead.
__device__ __forceinline__ uint4v philox4x32_rolled(std::uint32_t c0, std::uint32_t c1, std::uint32_t c2,
                                                    std::uint32_t c3, std::uint32_t k0, std::uint32_t k1) {
#pragma unroll 1
    for (int round = 0; round < 10; ++round) {
        const std::uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const std::uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        c0 = hi1 ^ c1 ^ k0; c1 = lo1; c2 = hi0 ^ c3 ^ k1; c3 = lo0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return {c0, c1, c2, c3};
}

__device__ __forceinline__ double u53(std::uint32_t hi, std::uint32_t lo) {
    return (double)(((((unsigned long long)hi) << 32) | lo) >> 11) * 0x1.0p-53;
}

// Counter layout: (step, ant, batch, tag).  tag 0 construction uniform,
// 1 start node, 2 colony source draw (ant = 0xffffffff).
__device__ __forceinline__ double source_uniform(unsigned long long key, std::uint32_t batch) {
    const uint4v r = philox4x32(0, 0xffffffffu, batch, 2, (std::uint32_t)key, (std::uint32_t)(key >> 32));
    return u53(r.x, r.y);
}

// One registered instance resident on the device.
struct InstanceView {
    std::uint32_t n;
    std::uint32_t k, b, w;         // primary / backup / LS widths (clipped to n)
    const int2* xy;                // [n]
    const node_t* primary;         // [n][k]
    const node_t* backup;          // [n][b]
    const node_t* ls;              // [n][w], distance ordered
    const int* ls_dist;            // [n][w]
    const float* eta;              // [n][k]
    const node_t* initial;         // [n]
    long long initial_cost;
    const node_t* region_list;     // nodes grouped by quadrant of the bounding box
    std::uint32_t region_offsets[5];
    float mean_nn;                 // mean nearest-neighbour distance (prior features)
    // 12-feature controller (feature spec 2)
    const node_t* samples;         // min(n, 64) sample nodes drawn from the instance key
    std::uint32_t sample_count;
    const double* local_scale;     // [n] mean of the min(8, n-1) nearest lengths
    double scale_epsilon;          // 1e-12 * max(coordinate span, 1)
    const float* alpha;            // [n][k] alpha-nearness of the primary entries (prior features)
};

// GP program (postfix IR; device mirror of faco_program).
struct Program {
    std::uint16_t ir_version, numeric_spec_id, feature_spec_id, length, constants_count;
    std::uint8_t opcode[63];
    std::uint8_t operand[63];
    float constants[63];
};

// Start node from a start region (quadrant) when one is set and non-empty,
// else uniform over all nodes; the same Philox draw either way.
__device__ __forceinline__ std::uint32_t region_start(unsigned long long key, std::uint32_t batch,
                                                      std::uint32_t ant, const InstanceView* in,
                                                      std::uint32_t region) {
    const uint4v r = philox4x32(0, ant, batch, 1, (std::uint32_t)key, (std::uint32_t)(key >> 32));
    if (region < 4) {
        const std::uint32_t lo = in->region_offsets[region], size = in->region_offsets[region + 1] - lo;
        if (size) return in->region_list[lo + (std::uint32_t)(((unsigned long long)r.x * size) >> 32)];
    }
    return (std::uint32_t)(((unsigned long long)r.x * in->n) >> 32);
}

// Per-colony mutable state (one per work item of an evaluation).
struct ColonyState {
    long long epoch_cost, global_cost, parent_cost;
    long long iteration_best_cost;
    float tau_min, tau_max, default_trail;
    std::uint32_t iteration;       // completed batches
    std::uint32_t iteration_best;
    std::uint32_t source_is_epoch;
    std::uint32_t mne_target;
    std::int32_t action;
    unsigned long long construction_steps, ls_evaluations, reversed_elements;
    // controller state (GP-controlled evaluations)
    std::uint32_t region;          // start region of the next iteration (4 = all nodes, 5 = the controller's start list)
    std::uint32_t restarts, last_improvement, last_restart;
};

struct RefControl;

// Per-colony constant view.
struct ColonyView {
    std::uint32_t instance;        // index into the instance table
    std::uint32_t n;
    unsigned long long key;        // Philox key
    float* trails;                 // [n][k]
    float* products;               // [n][k]
    float* eta;                    // [n][k] heuristic of this colony (instance eta, or reweighted by the prior)
    node_t* parent;                // [n_pad] (16-byte aligned)
    std::uint32_t* parent_nbr;     // [n]: parent successor | predecessor << 16
    node_t* epoch;                 // [n]
    node_t* global;                // [n]
    node_t* ant_tours;             // [ants][n_pad] (16-byte aligned rows)
    std::uint32_t n_pad;           // row stride of ant_tours (n rounded up to 8)
    long long* ant_costs;          // [ants] final (after LS)
    long long* ant_ccosts;         // [ants] after construction
    unsigned* ant_counts;          // [ants][3]: construction steps, LS evaluations, moved elements
    const Program* program;        // GP controller of this colony: 3 tree slots (null: plain FACO)
    std::uint32_t action_mask;     // legal actions
    std::uint32_t controller_kind; // 0 joint_single (slot 0), 1 conditional_three (slots 0-2 = roles)
    // 12-feature controller (feature spec 2; null otherwise)
    RefControl* control;
    node_t* archive;               // [2 sides][4 slots][tour, positions][n_pad]
    unsigned long long* ant_ids;   // [ants][2] fingerprints of the batch's tours
    std::uint32_t* ant_p0;         // [ants] position of node 0 in each tour
    std::uint32_t* walk;           // construction steps per ant of the last iteration
    node_t* parent_pos;            // [n_pad] inverse of `parent` (null: not kept, the ants build their own)
};

struct TraceRow {
    long long iteration_best_cost, global_cost, parent_cost;
    std::uint32_t iteration_best, source_is_epoch;
    float tau_min, tau_max;
    std::uint32_t mne_target;
    std::int32_t action;
    unsigned long long construction_steps, ls_evaluations;
};

}  // namespace faco

// faco_ant.cuh -- one warp runs one ant: focused construction from the
// colony's parent tour, then checklist local search.
//
// Semantics follow the reference's fused kernel construct_and_search
// (cuda/faco_device.cuh:100-501) and its CPU restatement
// (cpp/src/faco_cpu.cpp:82-294): relocation steps until the MNE target,
// candidate-row roulette with backup and global fallbacks, then FIFO
// checklist 2-opt with best-gain moves and the reference's tie, cap and
// reversal rules.  The GB300 design differs throughout:
//   - every per-ant scalar is warp-uniform and lives in registers of all 32
//     lanes (no shared State struct, no lane-0 serial sections beyond the
//     single store of a queue slot or flag word);
//   - the tour and its inverse live in shared memory as 16-bit nodes, the
//     visited/pending flags as bitsets; coordinates are staged once per
//     block for all its ants (one colony per block); the checklist ring
//     lives in the ant's own output-tour slot in global memory (L1-cached),
//     which nothing reads before the ant writes its final tour there;
//   - distances are exact EUC_2D integers computed on the fly, so gains and
//     tour lengths are exact int64 and ties are decided by index only;
//   - the roulette decides from an FP32 warp scan whenever a proven error
//     margin allows and otherwise recomputes the reference's ordered FP64
//     prefix sums, so the choice is always the FP64 one (GB300 runs FP64 at
//     a small fraction of its FP32 rate);
//   - relocation shifts run as register-staged warp chunks, reversals as
//     disjoint swap pairs, the best move by __reduce_max_sync, and the local
//     search packs the candidates of several pending nodes into one warp pass.
#pragma once

#include <climits>

#include "faco_common.cuh"

namespace faco {

enum AntMode : int {
    kModeEngine = 0,    // Philox choices, colony parent (production path)
    kModeVisits = 1,    // explicit visit orders (diagnostic)
    kModeUniforms = 2,  // injected uniforms + given products (diagnostic)
    kModePrepare = 3,   // no construction; LS over the whole tour (registration)
    kModeEngineGlobal = 4,  // kModeEngine with tour/inverse in global memory and
                            // coordinates read from global (large instances)
    kModeEngineFollow = 5,        // kModeEngine with batched parent-following steps (follow_batch)
    kModeEngineGlobalFollow = 6,  // kModeEngineGlobal with batched parent-following steps
    // kModeEngineFollow with fewer registers, for panels beyond one wave of
    // the GPU (ant_blocks_per_sm)
    kModeEngineFollowDense = 7,
};

// An engine variant compiled for one local search (or'ed to the mode).  With
// both in one kernel the register budget of the larger one spills in the
// other: 256 x 32 ants at N=1000 ran 122.5 ms instead of 115.4.
constexpr int kTwoOptOnly = 16, kOrOptOnly = 32, kModeMask = 15;

__host__ __device__ constexpr bool engine_mode(int mode) {
    const int m = mode & kModeMask;
    return m == kModeEngine || m == kModeEngineGlobal || m == kModeEngineFollow || m == kModeEngineGlobalFollow ||
           m == kModeEngineFollowDense;
}
__host__ __device__ constexpr bool global_mode(int mode) {
    const int m = mode & kModeMask;
    return m == kModeEngineGlobal || m == kModeEngineGlobalFollow;
}
__host__ __device__ constexpr bool dense_mode(int mode) { return (mode & kModeMask) == kModeEngineFollowDense; }
__host__ __device__ constexpr bool follow_mode(int mode) {
    const int m = mode & kModeMask;
    return m == kModeEngineFollow || m == kModeEngineGlobalFollow || m == kModeEngineFollowDense;
}
// The batched variant of an engine mode (`dense`: the build for panels
// beyond one wave, where there is one).
__host__ __device__ constexpr int with_follow(int mode, bool dense = false) {
    return mode == kModeEngineGlobal ? kModeEngineGlobalFollow
           : mode == kModeEngine     ? (dense ? kModeEngineFollowDense : kModeEngineFollow)
                                     : mode;
}

struct AntLaunch {
    // instance (all ants of a block share one instance)
    const InstanceView* instances;
    // engine mode
    const ColonyView* colonies;
    ColonyState* states;
    const uint2* work;            // per block: (colony, first ant)
    node_t* workspace;            // kModeEngineGlobal: tour + inverse per ant, laid out
                                  // like the colonies' ant_tours with rows of 2 x n_pad
    const node_t* ant_tours_base; // start of the buffer the colonies' ant_tours point into
    std::uint32_t ants;           // ants per colony
    std::uint32_t warps;          // warps per block
    std::uint32_t n_max;          // smem layout size
    unsigned long long ls_limit;
    std::uint32_t ls_mode;
    std::uint32_t batch_from;     // batched variants: colonies whose ants walked at least this many steps
                                  // in their last iteration (ColonyView::walk; 0: all) use the batches
    // diagnostic modes: tasks on instance 0
    std::uint32_t tasks;
    const node_t* task_tours;        // [tasks][n]
    const std::uint32_t* task_nbr;   // [tasks][n] parent successor | predecessor << 16
    const long long* task_costs;     // [tasks]
    const node_t* task_visits;       // [tasks][n]
    const double* task_uniforms;     // [tasks][n]
    const std::uint32_t* task_starts;
    const std::uint32_t* task_targets;
    const float* task_products;      // [n][k]
    // diagnostic outputs (may be null)
    node_t* out_construction;     // [tasks][n]
    node_t* out_tours;            // [tasks][n]; required: also each task's checklist ring during the run
    node_t* out_pos;              // [tasks][n]
    node_t* out_selected;         // [tasks][n]
    std::uint32_t* out_checklist; // [tasks][checklist_cap]
    std::uint32_t checklist_cap;
    long long* out_costs;         // [tasks][2]
    unsigned long long* out_counters;  // [tasks][10]
    unsigned* error;
};

__host__ __device__ inline std::uint32_t pad8(std::uint32_t n) { return (n + 7u) & ~7u; }

// Per-warp shared-memory workspace: tour and inverse (16-bit), visited and
// pending bitsets.
__host__ __device__ inline std::uint32_t ant_smem_bytes(std::uint32_t n) {
    return (4u * pad8(n) + 8u * ((n + 31u) / 32u) + 15u) & ~15u;
}
__host__ __device__ inline std::uint32_t block_smem_bytes(std::uint32_t n, std::uint32_t warps) {
    return ((8u * n + 15u) & ~15u) + warps * ant_smem_bytes(n);
}
// Global-workspace variant: only the two bitsets per ant stay in shared memory.
__host__ __device__ inline std::uint32_t ant_bitset_bytes(std::uint32_t n) {
    return (8u * ((n + 31u) / 32u) + 15u) & ~15u;
}
__host__ __device__ inline std::uint32_t block_smem_bytes_global(std::uint32_t n, std::uint32_t warps) {
    return warps * ant_bitset_bytes(n);
}

struct AntSmem {
    node_t* tour;                 // shared
    node_t* pos;                  // shared
    node_t* ring;                 // global: the ant's checklist ring (n entries)
    std::uint32_t* visited;       // shared
    std::uint32_t* queued;        // shared
    __device__ static AntSmem at(unsigned char* base, std::uint32_t n_max, node_t* ring) {
        const std::uint32_t np = pad8(n_max), words = (n_max + 31u) / 32u;
        return {reinterpret_cast<node_t*>(base), reinterpret_cast<node_t*>(base + 2 * np), ring,
                reinterpret_cast<std::uint32_t*>(base + 4 * np),
                reinterpret_cast<std::uint32_t*>(base + 4 * np) + words};
    }
    // tour/inverse at `global` (2 x n_pad nodes), bitsets at `bits` (shared)
    __device__ static AntSmem split(node_t* global, std::uint32_t n_pad, unsigned char* bits,
                                    std::uint32_t n_max, node_t* ring) {
        const std::uint32_t words = (n_max + 31u) / 32u;
        return {global, global + n_pad, ring, reinterpret_cast<std::uint32_t*>(bits),
                reinterpret_cast<std::uint32_t*>(bits) + words};
    }
};

__device__ __forceinline__ bool test_bit(const std::uint32_t* bits, std::uint32_t v) {
    return (bits[v >> 5] >> (v & 31u)) & 1u;
}

struct Checklist {
    std::uint32_t head, tail, pending, pushed;  // ring indices and counters (warp-uniform)
};

// Appends the nodes of lanes 0, 1, ... (each lane its own `v`, taken when
// `want`) that are not pending, in lane order: what one append_if_absent
// after the other does (cuda/faco_device.cuh:81-92).  The wanted nodes are
// distinct.  Returns the number appended.
__device__ __forceinline__ std::uint32_t push_lanes(const AntSmem& s, Checklist& q, std::uint32_t n, std::uint32_t v,
                                                    bool want, std::uint32_t lane, std::uint32_t* log,
                                                    std::uint32_t log_cap) {
    const bool absent = want && !test_bit(s.queued, v);
    const unsigned m = __ballot_sync(kFull, absent);   // every lane has read its flag before one is set
    if (absent) {
        const std::uint32_t rank = __popc(m & ((1u << lane) - 1u));
        std::uint32_t at = q.tail + rank;
        if (at >= n) at -= n;
        atomicOr(&s.queued[v >> 5], 1u << (v & 31u));
        s.ring[at] = (node_t)v;
        if (log && q.pushed + rank < log_cap) log[q.pushed + rank] = v;
    }
    const std::uint32_t count = __popc(m);
    q.tail += count;
    if (q.tail >= n) q.tail -= n;
    q.pending += count;
    q.pushed += count;
    __syncwarp();
    return count;
}

struct AntResult {
    long long construction_cost, final_cost;
    std::uint32_t mne, steps, nonidentity;
    // below 2^32: at most a few pops per accepted move, n moves, 5 w evaluations per pop
    std::uint32_t processed, checks, evaluations, accepted, reactivations;
    std::uint32_t moved;  // tour elements rewritten by relocations and reversals, modulo 2^32 (as reported)
    std::uint32_t limit_reached, checklist;
};

// Rounds of a shift, reversal or copy taken as one, all loads before the first
// store.  In the global-memory workspace a round waits for L2: three in one cut
// the large panel (80 colonies x 64 ants, N 5000-10000) from 90 to 73 ms (two
// 78; four 78, with spills).  In shared memory the longer code and its
// registers cost more than the shorter wait (two in one: 256 x 32 ants at
// N=1000 158 instead of 109 ms).
template <bool kGlobal>
constexpr std::uint32_t kRound = kGlobal ? 3u : 1u;

// Moves `node` right after `target` (CpuTour::relocate): shifts the closed
// interval between their positions by one, register-staged per chunk (two
// elements per lane and round) so that every read of a chunk precedes its
// writes; chunks run away from the vacated end.
template <bool kGlobal>
__device__ __forceinline__ void relocate_shift(const AntSmem& s, std::uint32_t lane, std::uint32_t tpos,
                                               std::uint32_t npos, std::uint32_t node) {
    constexpr std::uint32_t kEach = 2 * kRound<kGlobal>;
    std::uint32_t v[kEach];
    if (tpos < npos) {
        // new[tpos+1] = node, new[i] = old[i-1] for i in (tpos+1, npos]
        const int lo = (int)tpos + 1;
        for (int base = (int)npos; base >= lo; base -= 32 * (int)kEach) {
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const int i = base - (int)lane - 32 * (int)u;
                if (i >= lo) v[u] = i == lo ? node : s.tour[i - 1];
            }
            __syncwarp();
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const int i = base - (int)lane - 32 * (int)u;
                if (i >= lo) { s.tour[i] = (node_t)v[u]; s.pos[v[u]] = (node_t)i; }
            }
            __syncwarp();
        }
    } else {
        // new[i] = old[i+1] for i in [npos, tpos), new[tpos] = node
        for (std::uint32_t base = npos; base <= tpos; base += 32 * kEach) {
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const std::uint32_t i = base + lane + 32 * u;
                if (i <= tpos) v[u] = i == tpos ? node : s.tour[i + 1];
            }
            __syncwarp();
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const std::uint32_t i = base + lane + 32 * u;
                if (i <= tpos) { s.tour[i] = (node_t)v[u]; s.pos[v[u]] = (node_t)i; }
            }
            __syncwarp();
        }
    }
}

// Swaps the pairs (l, r) = ends(o), o in [0, pairs), of disjoint tour
// positions, with the inverse.
template <bool kGlobal, class Ends>
__device__ __forceinline__ void swap_pairs(const AntSmem& s, std::uint32_t lane, std::uint32_t pairs, Ends ends) {
    constexpr std::uint32_t kEach = kRound<kGlobal>;
    for (std::uint32_t first = lane; first < pairs; first += 32 * kEach) {
        node_t a[kEach], b[kEach];
#pragma unroll
        for (std::uint32_t u = 0; u < kEach; ++u) {
            if (first + 32 * u >= pairs) continue;
            const uint2 at = ends(first + 32 * u);
            a[u] = s.tour[at.x];
            b[u] = s.tour[at.y];
        }
#pragma unroll
        for (std::uint32_t u = 0; u < kEach; ++u) {
            if (first + 32 * u >= pairs) continue;
            const uint2 at = ends(first + 32 * u);
            s.tour[at.x] = b[u]; s.tour[at.y] = a[u];
            s.pos[b[u]] = (node_t)at.x; s.pos[a[u]] = (node_t)at.y;
        }
    }
    __syncwarp();
}

// Reverses tour[lo..hi] (inclusive, lo <= hi, no wrap) with the inverse.
template <bool kGlobal>
__device__ __forceinline__ void reverse_range(const AntSmem& s, std::uint32_t lane, std::uint32_t lo,
                                              std::uint32_t hi) {
    swap_pairs<kGlobal>(s, lane, (hi - lo + 1) / 2, [&](std::uint32_t o) { return uint2{lo + o, hi - o}; });
}

// A run of relocations deferred during construction.  Once trails converge
// an ant mostly follows parent edges: after it takes a node x from its place
// to after the current node, its next nodes are x's old tour neighbours,
// taken one at a time from the same place -- each relocation shifting the
// whole span between the two places again.  A run starts at a relocation:
// it keeps the tour as it is before the node moves (`ph`, the node y_1 at
// p, the current node at t) and the number m of nodes taken since
// (y_j = ph[p + dir (j-1)], j = 1..m), and reads the relocated tour through
// a position map; apply() rewrites the span once, by the single shift when
// m == 1, else with two or three reversals.  The tour it reads equals the one the
// relocations one by one would have left (CpuTour::relocate,
// cpp/src/faco_cpu.cpp:82-112):
//   p < t: the taken nodes sit at [t-m+1, t] in order, the span between
//          them and their source moved left by m;
//   p > t: the taken nodes sit at [t+1, t+m] in order, the span moved
//          right by m.
// An ant defers its relocations on instances of more than kDeferAllFrom
// nodes, and on the others after kDeferFromStep construction steps (early,
// short walks rarely continue a run: there a deferred single relocation
// costs more than an immediate one; measured at N=1000 and N=5000-10000).
constexpr std::uint32_t kDeferFromStep = 24;
constexpr std::uint32_t kDeferAllFrom = 2048;

struct RelocationRun {
    std::uint32_t m = 0;   // 0: no run
    std::uint32_t p = 0, t = 0;
    int dir = 1;           // +1: sources taken rightwards; -1: leftwards (either while m == 1)

    // node at position i of the relocated tour
    __device__ __forceinline__ std::uint32_t read(const AntSmem& s, std::uint32_t i) const {
        if (p < t) {
            const std::uint32_t first = t - m + 1;
            if (i >= first && i <= t) return s.tour[dir > 0 ? p + (i - first) : p - (i - first)];
            const std::uint32_t lo = dir > 0 ? p : p - m + 1;
            if (i >= lo && i < first) return s.tour[i + m];
        } else {
            const std::uint32_t last = t + m;
            if (i > t && i <= last) return s.tour[dir > 0 ? p + (i - t - 1) : p - (i - t - 1)];
            const std::uint32_t hi = dir > 0 ? p + m - 1 : p;
            if (i > last && i <= hi) return s.tour[i - m];
        }
        return s.tour[i];
    }
    // position of the current node (the last one taken)
    __device__ __forceinline__ std::uint32_t current_pos() const { return p < t ? t : t + m; }
    // Direction in which a node at position q of ph continues the run (the
    // next source, p + dir m), or 0: not next to the sources, past a tour
    // end, or out of the span between the sources and the taken nodes.
    __device__ __forceinline__ int continues(std::uint32_t q) const {
        if (q + m == p && (p < t || q > t) && (m == 1 || dir < 0)) return -1;
        if (q == p + m && (p > t || q < t) && (m == 1 || dir > 0)) return 1;
        return 0;
    }
    // position of that node in the relocated tour
    __device__ __forceinline__ std::uint32_t source_pos(int d) const {
        return (p < t) == (d < 0) ? (d < 0 ? p - m : p + m) : p;
    }
    // Rewrites the span so that the tour holds the relocated order; the run
    // ends.  `last` is the node taken last (the ant's current node).
    template <bool kGlobal>
    __device__ void apply(const AntSmem& s, std::uint32_t lane, std::uint32_t last) {
        if (m == 1) {
            relocate_shift<kGlobal>(s, lane, t, p, last);   // reads before its first write, after a warp barrier
            m = 0;
            return;
        }
        __syncwarp();
        if (p < t) {
            // [sources | span] -> [span | taken in order]
            const std::uint32_t lo = dir > 0 ? p : p - m + 1, span = t - lo + 1 - m;
            reverse_range<kGlobal>(s, lane, lo, t);
            if (span > 1) reverse_range<kGlobal>(s, lane, lo, lo + span - 1);
            if (dir > 0) reverse_range<kGlobal>(s, lane, t - m + 1, t);
        } else {
            // [span | sources] -> [taken in order | span]
            const std::uint32_t hi = dir > 0 ? p + m - 1 : p, span = hi - t - m;
            reverse_range<kGlobal>(s, lane, t + 1, hi);
            if (dir > 0) reverse_range<kGlobal>(s, lane, t + 1, t + m);
            if (span > 1) reverse_range<kGlobal>(s, lane, t + m + 1, hi);
        }
        m = 0;
    }
};

// Construction steps that follow the parent tour, evaluated 16 or 32 at a
// time, one lane per step.  Once trails converge an ant mostly takes a
// parent-tour neighbour of its current node (no new edge): either the node
// after it in its tour (an identity step) or, after a jump, the old tour
// neighbours of the node it jumped to, pulled one by one from their place
// (a relocation run).  Both paths are known before the draws are: lane i
// assumes the walk followed that path for i steps and decides step i's
// roulette on its own -- candidates of its node, available unless visited
// or earlier on the path, its own uniform -- with a serial FP32 sum and a
// proven margin (sequential FP32 prefixes of at most 32 non-negative terms
// are within 31 roundings of the exact ones, the threshold within 33, so
// 2^-17 of the total separates the FP64 decision with room to spare);
// undecided lanes end the batch.  The leading lanes whose choice is their
// hypothesised node are then applied as one: visited bits, counters, the
// run extended by their number (or, for identity steps, nothing else), and
// the exact six-edge deltas of every step summed.  The tour, costs and
// counters equal those of the steps one by one; the first lane that is not
// taken is left to the caller's serial step.  All 32 steps are decided at
// once, so a long walk along the parent tour costs a few steps' latency:
// the variant for panels that leave the GPU under-filled, where an
// iteration lasts as long as its longest walk.
//
// Hypotheses: with a run of m >= 2 nodes, its direction (32 lanes); with a
// run of one node, both directions (lanes 0-15 rightwards, 16-31
// leftwards); with no run, lanes 0-15 the parent successor of the current
// node and 16-31 its parent predecessor -- an identity walk along the tour
// when that node follows the current one, else the start of a run.
// Returns the number of steps taken (0: nothing changed); `full` is set when
// every lane of the chosen hypothesis was taken (the walk may go on).
__device__ __forceinline__ bool on_segment(int lo, int hi, int q) { return q >= lo && q <= hi; }

// Whether one lane's step in follow_batch draws `sel`: the candidates of
// `row` still open to the walk (unvisited, and neither on the identity walk
// nor on the relocation run taken by the earlier lanes), their FP32 weights
// summed serially in candidate order.  The first prefix at or above uf *
// total is sel's own, by the decision margin on both sides, exactly when the
// prefix before sel is certainly below the threshold and the one with sel
// certainly above it; so one pass over the row decides, with the total and
// those two prefixes.  False where the margin leaves it open (the one-step
// path then decides).  Rows of a multiple of four candidates are read four
// at a time (8 + 16 bytes), one group ahead of the sums; the caller has read
// the first one (x, p).
__device__ __forceinline__ bool follow_takes(const AntSmem& s, const node_t* row, const float* prow, std::uint32_t n,
                                             std::uint32_t k, std::uint32_t sel, std::uint32_t rel, std::uint32_t t0,
                                             bool identity, int lo, int hi, float uf, uint2 x, float4 p) {
    float total = 0.0f, before = 0.0f, upto = -1.0f;
    bool any = false, earlier = false;
    // (adding zero for a closed candidate leaves the sum as it is)
    const auto add = [&](std::uint32_t x, float weight) {
        const std::uint32_t px = s.pos[x];
        const std::uint32_t dx = px >= t0 ? px - t0 : px + n - t0;   // tour positions after the start
        const bool on_path = identity ? dx - 1u < rel : on_segment(lo, hi, (int)px);
        const bool open = !(test_bit(s.visited, x) | (rel && on_path)), mine = open && x == sel;
        before = mine ? total : before;
        earlier = mine ? any : earlier;
        total += open ? weight : 0.0f;
        upto = mine ? total : upto;
        any |= open;
    };
    if ((k & 3u) == 0) {
        const uint2* rows = reinterpret_cast<const uint2*>(row);
        const float4* weights = reinterpret_cast<const float4*>(prow);
#pragma unroll 1
        for (std::uint32_t g = 1; g <= k / 4; ++g) {
            const uint2 xg = x;
            const float4 pg = p;
            if (g < k / 4) {
                x = __ldg(rows + g);
                p = load_written(weights + g);
            }
            add(xg.x & 0xffffu, pg.x);
            add(xg.x >> 16, pg.y);
            add(xg.y & 0xffffu, pg.z);
            add(xg.y >> 16, pg.w);
        }
    } else {
#pragma unroll 1
        for (std::uint32_t j = 0; j < k; ++j) add(__ldg(row + j), load_written(prow + j));
    }
    if (!(total >= 0x1p-100f)) return false;
    const float threshold = uf * total, delta = total * 0x1p-17f;
    return (!earlier || before - threshold < -delta) && upto - threshold > delta;
}

__device__ inline std::uint32_t follow_batch(const AntSmem& s, const int2* xy, const InstanceView& in,
                                             const float* products, const std::uint32_t* parent_nbr, std::uint32_t n,
                                             std::uint32_t lane, unsigned long long key, std::uint32_t batch,
                                             std::uint32_t ant, std::uint32_t& current, AntResult& r,
                                             long long& cost, RelocationRun& run, std::uint32_t& draw_base,
                                             std::uint32_t& draw_hi, std::uint32_t& draw_lo, bool& full) {
    const std::uint32_t k = in.k;
    const std::uint32_t m0 = run.m;
    const bool split = m0 <= 1;
    const std::uint32_t half = split ? lane >> 4 : 0u, rel = split ? lane & 15u : lane;
    // the draws of the next 32 steps, lane i holding step base + i (the
    // caller's layout, which it reuses afterwards)
    const std::uint32_t base = r.steps + 1;
    if (base != draw_base) {
        const uint4v rb = philox4x32_rolled(base + lane, ant, batch, 0, (std::uint32_t)key, (std::uint32_t)(key >> 32));
        draw_base = base;
        draw_hi = rb.x;
        draw_lo = rb.y;
    }
    const std::uint32_t rhi = __shfl_sync(kFull, draw_hi, rel);
    const float uf = __uint2float_rn(rhi) * 0x1p-32f;

    // this lane's hypothesis: the node it stands on (cur) and the node it
    // must draw (sel), with the run geometry of its step
    bool identity = false;
    int p = 0, t = 0, D = 1;
    std::uint32_t t0 = 0;
    if (m0 >= 1) {
        p = (int)run.p;
        t = (int)run.t;
        D = m0 >= 2 ? run.dir : (half ? -1 : 1);
    } else {
        const std::uint32_t pn = load_written(parent_nbr + current);
        const std::uint32_t y = half ? pn >> 16 : pn & 0xffffu;
        t0 = s.pos[current];
        const std::uint32_t ty = s.pos[y];
        if (ty == (t0 + 1 == n ? 0u : t0 + 1)) {
            identity = true;
        } else {
            p = (int)ty;
            t = (int)t0;
            D = half ? -1 : 1;
        }
    }
    const std::uint32_t mr = m0 + rel;   // run nodes taken before this lane's step
    bool ok = rel + 1 < n - r.steps;     // the loop's step budget: steps + rel + 1 < n
    std::uint32_t cur = current, sel = n;
    int lo = 0, hi = -1;                 // path positions taken by the earlier lanes
    if (identity) {
        if (rel) cur = s.tour[(t0 + rel) % n];
        sel = s.tour[(t0 + rel + 1) % n];
    } else {
        const int q = p + D * (int)mr;
        ok = ok && q >= 0 && q < (int)n && (mr == 0 || (D < 0 ? (p < t || q > t) : (p > t || q < t)));
        if (ok) {
            sel = s.tour[q];
            if (rel) cur = s.tour[q - D];
        }
        if (rel) {
            const int a = p + D * (int)m0, b = q - D;
            lo = a < b ? a : b;
            hi = a < b ? b : a;
        }
    }
    // the first candidates of the lane's row, before what decides whether they are needed
    const node_t* row = in.primary + (size_t)cur * k;
    const float* prow = products + (size_t)cur * k;
    uint2 x = {0, 0};
    float4 p4 = {0.0f, 0.0f, 0.0f, 0.0f};
    if ((k & 3u) == 0) {
        x = __ldg(reinterpret_cast<const uint2*>(row));
        p4 = load_written(reinterpret_cast<const float4*>(prow));
    }
    if (ok) {
        const std::uint32_t pn = load_written(parent_nbr + cur);
        ok = (sel == (pn & 0xffffu) || sel == (pn >> 16)) && !test_bit(s.visited, sel);
    }
    // the run as it stands before this lane's step (m = mr): a step onto the
    // node after the current one is an identity step, not a relocation
    RelocationRun v;
    v.m = mr;
    v.p = (std::uint32_t)p;
    v.t = (std::uint32_t)t;
    v.dir = D;
    std::uint32_t tpos = 0, target_after = n;
    if (ok && !identity) {
        tpos = v.current_pos();
        target_after = v.read(s, tpos + 1 == n ? 0 : tpos + 1);
        ok = target_after != sel;
    }
    // the roulette of this lane's step: serial FP32 sums in candidate order
    if (ok) ok = follow_takes(s, row, prow, n, k, sel, rel, t0, identity, lo, hi, uf, x, p4);
    // the leading run of taken steps
    const unsigned okm = __ballot_sync(kFull, ok);
    std::uint32_t f, first_lane;
    if (split) {
        const unsigned m_lo = okm & 0xffffu, m_hi = okm >> 16;
        const std::uint32_t f_lo = __ffs(~m_lo) - 1, f_hi = __ffs(~m_hi) - 1;   // trailing ones, <= 16
        first_lane = f_lo ? 0u : 16u;
        f = f_lo ? f_lo : f_hi;
    } else {
        first_lane = 0;
        f = okm == kFull ? 32u : (std::uint32_t)(__ffs(~okm) - 1);
    }
    full = f == (split ? 16u : 32u);
    if (f == 0) return 0;
    const bool taken = lane >= first_lane && lane < first_lane + f;
    // identity lanes of the chosen half all agree on `identity`
    const std::uint32_t last_lane = first_lane + f - 1;
    const bool ident = __shfl_sync(kFull, identity ? 1 : 0, first_lane) != 0;
    const std::uint32_t last = __shfl_sync(kFull, sel, last_lane);
    if (!ident) {
        // The six-edge deltas of CpuTour::relocate over the steps telescope:
        // with s_1 .. s_f the nodes taken after c, T the node after c, X
        // beside s_1 on the near side of the sources and Y beside s_f on the
        // far side (each read through the run of its own step), they add up to
        // (X,Y) + (c,s_1) + (s_f,T) - (X,s_1) - (s_f,Y) - (c,T): one length
        // per lane instead of six in each.
        const std::uint32_t npos = v.source_pos(D);
        const std::uint32_t right = npos + 1 == n ? 0 : npos + 1, left = npos == 0 ? n - 1 : npos - 1;
        std::uint32_t near_end = n, far_end = n, moved = 0;
        if (taken) {
            near_end = v.read(s, D > 0 ? left : right);
            far_end = v.read(s, D > 0 ? right : left);
            moved = tpos < npos ? npos - tpos : tpos - npos + 1;
        }
        const std::uint32_t X = __shfl_sync(kFull, near_end, first_lane), T = __shfl_sync(kFull, target_after, first_lane);
        const std::uint32_t Y = __shfl_sync(kFull, far_end, last_lane), first = __shfl_sync(kFull, sel, first_lane);
        int term = 0;
        if (lane < 6) {
            const std::uint32_t ea = lane == 0 || lane == 3 ? X : lane == 1 || lane == 5 ? current : last;
            const std::uint32_t eb = lane == 0 || lane == 4 ? Y : lane == 1 || lane == 3 ? first : T;
            const int dd = euc2d(xy[ea], xy[eb]);
            term = lane < 3 ? dd : -dd;
        }
        cost += __reduce_add_sync(kFull, term);
        r.moved += __reduce_add_sync(kFull, moved);
        r.nonidentity += f;
        run.p = (std::uint32_t)__shfl_sync(kFull, p, first_lane);
        run.t = (std::uint32_t)__shfl_sync(kFull, t, first_lane);
        run.dir = __shfl_sync(kFull, D, first_lane);
        run.m = m0 + f;
    }
    if (taken) atomicOr(&s.visited[sel >> 5], 1u << (sel & 31u));
    current = last;
    r.steps += f;
    __syncwarp();
    return f;
}

// flip_without_cost (cpp/src/faco_cpu.cpp:114-135) between the tour positions
// of its two end nodes, as disjoint swap pairs.  Returns the number of
// elements in the reversed segment.  Every lane has read what it needs of the
// tour before the call's barrier.
template <bool kGlobal>
__device__ __forceinline__ std::uint32_t flip(const AntSmem& s, std::uint32_t n, std::uint32_t lane,
                                              std::uint32_t first, std::uint32_t last) {
    if (first > last) { const std::uint32_t t = first; first = last; last = t; }
    const std::uint32_t length = last - first;
    const bool straight = length <= n - length || first == 0;
    const std::uint32_t count = straight ? length : n - length, begin = straight ? first : last;
    __syncwarp();
    swap_pairs<kGlobal>(s, lane, count / 2, [&](std::uint32_t o) {
        uint2 at{begin + o, begin + count - 1 - o};
        if (at.x >= n) at.x -= n;
        if (at.y >= n) at.y -= n;
        return at;
    });
    return count;
}

// Checklist 2-opt, best gain per popped node, reference tie/cap rules
// (cpp/src/faco_cpu.cpp:148-217; cuda/faco_device.cuh:295-478).
//
// Up to kPopNodes nodes from the head of the checklist are evaluated
// together.  About two pops in three find no move and then leave the tour as
// it is, so the nodes up to and including the first one with a move are the
// pops one by one, with the same tours, checklist order and counts; the
// nodes after it stay pending and are evaluated again.  A node's candidates
// worth a gain (those nearer than its tour neighbour, a prefix of its row
// for each of the two kinds) are few -- 6.5 per pop of 2 x 20 on the N=1000
// panel -- so the prefixes of all nodes are packed one per lane:
//   lanes 2i + kind   node i's neighbour of that kind and its length
//   all lanes         the prefix lengths of the 2 x kPopNodes segments, by
//                     one ballot each over the node's row
//   lane t            the t-th candidate of the concatenated segments
// Nodes whose segments end past lane 31 wait for the next pass; a first node
// that fills more than a warp alone (both kinds wide) takes two rounds.
//
// Bound by the ant's chain of dependent instructions (one warp issues every
// ~6 cycles; a length takes ~150 cycles, a shuffle 36, a ballot 44); a pass
// resolves about two pops for the chain of one.  One GB300, against one pop
// per pass: one N=100 colony, 64 iterations 8.78 -> 7.46 ms; 256 x 32 ants at
// N=1000, 320 iterations 151 -> 136 ms; the uneven batch (N 200-1000, 400
// iterations) 145 -> 122 ms; 128 x 32 at N=1000-2000, 640 iterations 228 ->
// 205 ms.  The winner by one reduction of (node, gain), its payload in two
// words and the reversal's ends by position: a further 3-6 %.
constexpr std::uint32_t kPopNodes = 4;

template <bool kGlobal>
__device__ __forceinline__ void checklist_two_opt(const AntSmem& s, const int2* xy, const InstanceView& in,
                                                  std::uint32_t n, std::uint32_t lane, Checklist& q,
                                                  unsigned long long cap, AntResult& r, long long& gain_sum,
                                                  std::uint32_t* log, std::uint32_t log_cap) {
    const std::uint32_t w = in.w;
    const std::uint32_t limit = cap < 0xffffffffull ? (std::uint32_t)cap : 0xffffffffu;
    std::uint32_t evaluations = 0;
    const std::uint32_t kind = lane & 1u;
    while (q.pending > 0 && r.accepted < n) {
        if (evaluations >= limit) { r.limit_reached = 1; break; }
        // lane 2i + kind: node i (the first one again where fewer are pending), its neighbour and edge length
        const std::uint32_t i = (lane >> 1) & (kPopNodes - 1);
        const bool live = i < q.pending;
        std::uint32_t at = live ? q.head + i : q.head;
        if (at >= n) at -= n;
        const std::uint32_t a = s.ring[at];
        std::uint32_t head[kPopNodes], row_b[kPopNodes];
        int row_ab[kPopNodes];
#pragma unroll
        for (std::uint32_t t = 0; t < kPopNodes; ++t) {
            head[t] = __shfl_sync(kFull, a, 2 * t);
            const std::size_t row = (std::size_t)head[t] * w + lane;
            row_b[t] = n;
            row_ab[t] = INT_MAX;
            if (lane < w) {
                row_b[t] = __ldg(in.ls + row);
                row_ab[t] = __ldg(in.ls_dist + row);
            }
        }
        const std::uint32_t pa = s.pos[a];
        const std::uint32_t pend = kind ? (pa == 0 ? n - 1 : pa - 1) : (pa + 1 == n ? 0 : pa + 1);
        const std::uint32_t end = s.tour[pend];
        const int cur = live ? euc2d(xy[a], xy[end]) : -1;
        const std::uint32_t ends = a | end << 16;
        // segment ends: off[2i + kind + 1]
        std::uint32_t off[2 * kPopNodes + 1];
        off[0] = 0;
#pragma unroll
        for (std::uint32_t g = 0; g < 2 * kPopNodes; ++g) {
            const int c = __shfl_sync(kFull, cur, g);
            off[g + 1] = off[g] + __popc(__ballot_sync(kFull, c > row_ab[g >> 1] && row_b[g >> 1] < n));
        }
        std::uint32_t nodes = 1;
#pragma unroll
        for (std::uint32_t t = 2; t <= kPopNodes; ++t)
            if (off[2 * t] <= 32u) nodes = t;
        nodes = nodes < q.pending ? nodes : q.pending;
        std::uint32_t total = off[2];
#pragma unroll
        for (std::uint32_t t = 2; t <= kPopNodes; ++t)
            if (nodes == t) total = off[2 * t];
        if (total >= limit - evaluations) {
            // the budget may end here: the first node alone, cut where the budget ends
            nodes = 1;
            total = off[2];
            const std::uint32_t left = limit - evaluations, f0 = off[1], f1 = off[2] - off[1];
            const bool cut0 = left < f0, cut1 = !cut0 && left - f0 < f1;
            if (cut0 || cut1) {
                evaluations += left;
                r.checks += left + 1 + (cut1 && f0 < w ? 1 : 0);
                ++r.processed;
                r.limit_reached = 1;
                break;
            }
        }
        // lane t: the t-th candidate of the segments; its best move so far:
        // the gain, with the first nodes' moves above the others' (lengths
        // are below 2^25, gains below 2^26)
        constexpr std::uint32_t kNodeShift = 26;
        std::uint32_t best = 0, best_ends = 0, best_at = 0;
        for (std::uint32_t base = 0; base < total; base += 32) {
            const std::uint32_t t = base + lane;
            const bool on = t < total;
            // the segment of t, by halving
            const bool h2 = t >= off[4];
            const std::uint32_t e1 = h2 ? off[6] : off[2];
            const bool h1 = t >= e1;
            const std::uint32_t e0 = h2 ? (h1 ? off[7] : off[5]) : (h1 ? off[3] : off[1]);
            const bool h0 = t >= e0;
            const std::uint32_t seg = on ? (h2 ? 4u : 0u) + (h1 ? 2u : 0u) + (h0 ? 1u : 0u) : 0u;
            const std::uint32_t j = on ? t - (h0 ? e0 : h1 ? e1 : h2 ? off[4] : 0u) : 0u;
            const std::uint32_t own = __shfl_sync(kFull, ends, seg), node = own & 0xffffu, close = own >> 16;
            const int edge = __shfl_sync(kFull, cur, seg);
            std::uint32_t b = __shfl_sync(kFull, row_b[0], j);
            int ab = __shfl_sync(kFull, row_ab[0], j);
#pragma unroll
            for (std::uint32_t x = 1; x < kPopNodes; ++x) {
                const std::uint32_t bx = __shfl_sync(kFull, row_b[x], j);
                const int abx = __shfl_sync(kFull, row_ab[x], j);
                if ((seg >> 1) == x) { b = bx; ab = abx; }
            }
            if (on) {
                const std::uint32_t pb = s.pos[b];
                const std::uint32_t pnb = seg & 1u ? (pb == 0 ? n - 1 : pb - 1) : (pb + 1 == n ? 0 : pb + 1);
                const std::uint32_t nb = s.tour[pnb];
                const int2 nxy = xy[nb];
                const int g = nb == node || b == close ? 0 : edge - ab + euc2d(xy[b], nxy) - euc2d(xy[close], nxy);
                const std::uint32_t rank = ((kPopNodes - 1 - (seg >> 1)) << kNodeShift) + (std::uint32_t)g;
                if (g > 0 && rank > best) {
                    best = rank;
                    best_ends = b | nb << 16;
                    best_at = (seg & 1u ? pb : pnb) | seg << 16 | t << 19;   // second end of the reversal, segment, t
                }
            }
        }
        // the pops: up to the first node with a move, else all
        const std::uint32_t top = __reduce_max_sync(kFull, best);
        const std::uint32_t popped = top ? kPopNodes - (top >> kNodeShift) : nodes;
        std::uint32_t done = off[2];
#pragma unroll
        for (std::uint32_t t = 2; t <= kPopNodes; ++t)
            if (popped == t) done = off[2 * t];
        evaluations += done;
        r.processed += popped;
        r.checks += done;
#pragma unroll
        for (std::uint32_t g = 0; g < 2 * kPopNodes; ++g)
            r.checks += (g >> 1) < popped && off[g + 1] - off[g] < w ? 1 : 0;
        q.head += popped;
        if (q.head >= n) q.head -= n;
        q.pending -= popped;
        // pending flags of the pops, each by the lane of its node; lanes that
        // share a word clear the same bits of it
        std::uint32_t bits = 0;
#pragma unroll
        for (std::uint32_t t = 0; t < kPopNodes; ++t)
            if (t < popped && (head[t] >> 5) == (a >> 5)) bits |= 1u << (head[t] & 31u);
        if (lane < 2 * popped && kind == 0) s.queued[a >> 5] &= ~bits;
        if (top) {
            // the lowest candidate with that gain, in (kind, rank) order
            const unsigned ties = __ballot_sync(kFull, best == top);
            std::uint32_t src = __ffs(ties) - 1;
            if (total > 32) src = __reduce_min_sync(kFull, best == top ? best_at >> 19 : 0xffu) & 31u;
            const std::uint32_t move = __shfl_sync(kFull, best_ends, src), at1 = __shfl_sync(kFull, best_at, src);
            const std::uint32_t seg = (at1 >> 16) & 7u, p1 = at1 & 0xffffu, bj = move & 0xffffu, nbj = move >> 16;
            const std::uint32_t own = __shfl_sync(kFull, ends, seg), p0 = __shfl_sync(kFull, kind ? pa : pend, seg);
            const std::uint32_t node = own & 0xffffu, close = own >> 16;
            const bool back = seg & 1u;
            // all four ends become pending, in this order; reversed between the first two
            const std::uint32_t m0 = back ? node : close, m1 = back ? bj : nbj;
            const std::uint32_t m2 = back ? close : node, m3 = back ? nbj : bj;
            r.moved += flip<kGlobal>(s, n, lane, p0, p1);
            r.reactivations += push_lanes(s, q, n, lane == 0 ? m0 : lane == 1 ? m1 : lane == 2 ? m2 : m3, lane < 4,
                                          lane, log, log_cap);
            ++r.accepted;
            gain_sum -= (long long)(top & ((1u << kNodeShift) - 1u));
        }
        __syncwarp();
    }
    r.evaluations += evaluations;
}

// Checklist local search with first-improvement 2-opt then Or-opt (segments
// of 1-3 nodes starting at the popped node).  The reference has no Or-opt;
// the move order, pruning and counting rules are this engine's own (stated in
// full beside the CPU restatement).
//
// As in checklist_two_opt, up to kPopNodes pops are evaluated together and
// those up to the first with a move are taken: lanes 8i + r hold node i's
// tour neighbourhood (the nodes at positions -1 .. +3 around it, r = 0 .. 4)
// and its five scans (r = 0, 1: the 2-opt kinds; 2-4: the Or-opt lengths).
// Every move is the same expression: a candidate c of the node's row joins
// its tour neighbour nb on one side of it,
//   gain = base + d(c, nb) - d(a, c) - d(X, nb),
// base and X belonging to the scan.  The 2-opt scans of all nodes go one
// candidate per lane; then, node by node up to the first one with a 2-opt
// move, its Or-opt scans, one (candidate, side) per lane in scan order, so
// that the lowest lane with a gain is the first improvement.  On instances
// in the global-memory workspace a pop is a chain of five L2 reads, which the
// nodes of a pass share.  One GB300, the large panel (80 colonies x 64 ants,
// N 5000-10000, 80 iterations): 132 -> 110 ms.
template <bool kGlobal>
__device__ __forceinline__ void checklist_ls_first(const AntSmem& s, const int2* xy, const InstanceView& in,
                                                   std::uint32_t n, std::uint32_t lane, Checklist& q,
                                                   unsigned long long cap, AntResult& r, long long& gain_sum,
                                                   std::uint32_t* log, std::uint32_t log_cap) {
    const std::uint32_t w = in.w;
    const std::uint32_t limit = cap < 0xffffffffull ? (std::uint32_t)cap : 0xffffffffu;
    const std::uint32_t lengths = n < 6 ? n - 3 : 3u;   // Or-opt lengths L with n >= L + 3
    std::uint32_t evaluations = 0;
    const std::uint32_t role = lane & 7u, first = lane & 24u;
    // scan tests of a row whose first f candidates pass
    const auto scanned = [&](std::uint32_t f) { return f + (f < w ? 1u : 0u); };
    while (q.pending > 0 && r.accepted < n) {
        if (evaluations >= limit) { r.limit_reached = 1; break; }
        const bool live = (lane >> 3) < q.pending;
        std::uint32_t at = live ? q.head + (lane >> 3) : q.head;
        if (at >= n) at -= n;
        const std::uint32_t a = s.ring[at];
        std::uint32_t head[kPopNodes], row_b[kPopNodes];
        int row_ab[kPopNodes];
#pragma unroll
        for (std::uint32_t t = 0; t < kPopNodes; ++t) {
            head[t] = __shfl_sync(kFull, a, 8 * t);
            const std::size_t row = (std::size_t)head[t] * w + lane;
            row_b[t] = n;
            row_ab[t] = INT_MAX;
            if (lane < w) {
                row_b[t] = __ldg(in.ls + row);
                row_ab[t] = __ldg(in.ls_dist + row);
            }
            if (row_b[t] >= n) row_ab[t] = INT_MAX;   // right padding
        }
        // tour nodes t0 .. t4 at positions -1 .. +3, roles 0 .. 4
        std::uint32_t at_tour = s.pos[a] + n - 1 + (role < 5 ? role : 1u);
        if (at_tour >= n) at_tour -= n;
        if (at_tour >= n) at_tour -= n;
        const std::uint32_t near = s.tour[at_tour];
        const int2 near_xy = xy[near];
        // roles 0-3: d(t_r, t_r+1); roles 4-6: d(t0, t_r-2)
        const std::uint32_t from = first + (role < 4 ? role : 0u), to = first + (role < 4 ? role + 1 : role < 7 ? role - 2 : 0u);
        const int2 p = make_int2(__shfl_sync(kFull, near_xy.x, from), __shfl_sync(kFull, near_xy.y, from));
        const int2 o = make_int2(__shfl_sync(kFull, near_xy.x, to), __shfl_sync(kFull, near_xy.y, to));
        const int d = euc2d(p, o);
        // scan bases: d(a, next), d(prev, a), and the removal gains
        // d(prev, a) + d(e, q) - d(prev, q) of the segments a .. e before q
        const int d0 = __shfl_sync(kFull, d, role == 0 ? first + 1 : first);
        const int deq = __shfl_sync(kFull, d, first + (role >= 2 ? role - 1 : 0u));
        const int dpq = __shfl_sync(kFull, d, first + (role >= 2 && role < 5 ? role + 2 : 0u));
        const std::uint32_t X = __shfl_sync(kFull, near, first + (role == 0 ? 2u : role == 1 ? 0u : role < 5 ? role - 1 : 0u));
        const int base = !live || role > 1 + lengths ? -1 : role < 2 ? d0 : d0 + deq - dpq;
        // the 2-opt scans, as in checklist_two_opt
        std::uint32_t off[2 * kPopNodes + 1];
        off[0] = 0;
#pragma unroll
        for (std::uint32_t g = 0; g < 2 * kPopNodes; ++g) {
            const int c = __shfl_sync(kFull, base, 8 * (g >> 1) + (g & 1u));
            off[g + 1] = off[g] + __popc(__ballot_sync(kFull, c > row_ab[g >> 1]));
        }
        std::uint32_t nodes = 1;
#pragma unroll
        for (std::uint32_t t = 2; t <= kPopNodes; ++t)
            if (off[2 * t] <= 32u) nodes = t;
        nodes = nodes < q.pending ? nodes : q.pending;
        // near the end of the budget one node at a time, cut where it ends
        const std::uint32_t left = limit - evaluations;
        const bool tight = left <= 5 * kPopNodes * 32;
        if (tight) nodes = 1;
        std::uint32_t total = off[2];
#pragma unroll
        for (std::uint32_t t = 2; t <= kPopNodes; ++t)
            if (nodes == t) total = off[2 * t];
        bool two_opt = false;
        std::uint32_t move_c = 0, move_nb = 0, move_seg = 0, move_t = 0, node_of = nodes;
        int move_gain = 0;
        for (std::uint32_t base_t = 0; base_t < total && !two_opt; base_t += 32) {
            const std::uint32_t t = base_t + lane;
            const bool on = t < total;
            const bool h2 = t >= off[4];
            const std::uint32_t e1 = h2 ? off[6] : off[2];
            const bool h1 = t >= e1;
            const std::uint32_t e0 = h2 ? (h1 ? off[7] : off[5]) : (h1 ? off[3] : off[1]);
            const bool h0 = t >= e0;
            const std::uint32_t seg = on ? (h2 ? 4u : 0u) + (h1 ? 2u : 0u) + (h0 ? 1u : 0u) : 0u;
            const std::uint32_t j = on ? t - (h0 ? e0 : h1 ? e1 : h2 ? off[4] : 0u) : 0u;
            const std::uint32_t own = 8 * (seg >> 1) + (seg & 1u);
            const std::uint32_t close = __shfl_sync(kFull, X, own), node = __shfl_sync(kFull, a, own);
            const int edge = __shfl_sync(kFull, base, own);
            std::uint32_t c = __shfl_sync(kFull, row_b[0], j);
            int ac = __shfl_sync(kFull, row_ab[0], j);
#pragma unroll
            for (std::uint32_t x = 1; x < kPopNodes; ++x) {
                const std::uint32_t cx = __shfl_sync(kFull, row_b[x], j);
                const int acx = __shfl_sync(kFull, row_ab[x], j);
                if ((seg >> 1) == x) { c = cx; ac = acx; }
            }
            int g = 0;
            std::uint32_t nb = 0;
            if (on) {
                const std::uint32_t pc = s.pos[c];
                nb = s.tour[seg & 1u ? (pc == 0 ? n - 1 : pc - 1) : (pc + 1 == n ? 0 : pc + 1)];
                const int2 nxy = xy[nb];
                g = nb == node || c == close ? 0 : edge - ac + euc2d(xy[c], nxy) - euc2d(xy[close], nxy);
            }
            const unsigned improving = __ballot_sync(kFull, g > 0);
            if (improving) {
                const std::uint32_t src = __ffs(improving) - 1;
                two_opt = true;
                move_c = __shfl_sync(kFull, c, src);
                move_nb = __shfl_sync(kFull, nb, src);
                move_seg = __shfl_sync(kFull, seg, src);
                move_t = base_t + src;
                node_of = move_seg >> 1;
                move_gain = __shfl_sync(kFull, g, src);
            }
        }
        // the Or-opt scans of the nodes before it (of all, without one)
        bool or_opt = false;
        std::uint32_t or_c = 0, or_nb = 0, or_len = 0, or_side = 0, or_done = 0, or_node = 0;
        std::uint32_t f1 = 0, f2 = 0, f3 = 0, checks = 0;
        int or_gain = 0;
        for (std::uint32_t i = 0; i < node_of && !or_opt; ++i) {
            std::uint32_t rb = row_b[0], ai = head[0];
            int rab = row_ab[0];
#pragma unroll
            for (std::uint32_t x = 1; x < kPopNodes; ++x)
                if (i == x) { rb = row_b[x]; rab = row_ab[x]; ai = head[x]; }
            const std::uint32_t own = 8 * i + 2;
            const int g1 = __shfl_sync(kFull, base, own), g2 = __shfl_sync(kFull, base, own + 1);
            const int g3 = __shfl_sync(kFull, base, own + 2);
            const std::uint32_t s2 = __shfl_sync(kFull, near, own), s3 = __shfl_sync(kFull, near, own + 1);
            f1 = __popc(__ballot_sync(kFull, g1 > rab));
            f2 = __popc(__ballot_sync(kFull, g2 > rab));
            f3 = __popc(__ballot_sync(kFull, g3 > rab));
            const std::uint32_t o1 = 2 * f1, o2 = o1 + 2 * f2, o3 = o2 + 2 * f3;
            for (std::uint32_t base_t = 0; base_t < o3 && !or_opt; base_t += 32) {
                const std::uint32_t t = base_t + lane;
                const bool on = t < o3;
                const std::uint32_t len = on ? (t >= o1 ? 1u : 0u) + (t >= o2 ? 1u : 0u) : 0u;   // L - 1
                const std::uint32_t rest = on ? t - (len == 0 ? 0u : len == 1 ? o1 : o2) : 0u;
                const std::uint32_t j = rest >> 1, side = rest & 1u;   // side 0: between c and its successor
                const std::uint32_t c = __shfl_sync(kFull, rb, j), e = __shfl_sync(kFull, X, own + len);
                const int ac = __shfl_sync(kFull, rab, j), G = __shfl_sync(kFull, base, own + len);
                const auto inside = [&](std::uint32_t v) {
                    return v == ai || (len >= 1 && v == s2) || (len >= 2 && v == s3);
                };
                int g = 0;
                std::uint32_t nb = 0;
                if (on) {
                    const std::uint32_t pc = s.pos[c];
                    nb = s.tour[side ? (pc == 0 ? n - 1 : pc - 1) : (pc + 1 == n ? 0 : pc + 1)];
                    const int2 nxy = xy[nb];
                    g = inside(c) || inside(nb) ? 0 : G - ac + euc2d(xy[c], nxy) - euc2d(xy[e], nxy);
                }
                const unsigned improving = __ballot_sync(kFull, g > 0);
                if (improving) {
                    const std::uint32_t src = __ffs(improving) - 1;
                    or_opt = true;
                    or_node = i;
                    or_c = __shfl_sync(kFull, c, src);
                    or_nb = __shfl_sync(kFull, nb, src);
                    or_len = __shfl_sync(kFull, len, src) + 1;
                    or_side = __shfl_sync(kFull, side, src);
                    or_gain = __shfl_sync(kFull, g, src);
                    f3 = or_len >= 3 ? __shfl_sync(kFull, j, src) + 1 : 0u;
                    f2 = or_len == 2 ? __shfl_sync(kFull, j, src) + 1 : or_len > 2 ? f2 : 0u;
                    f1 = or_len == 1 ? __shfl_sync(kFull, j, src) + 1 : f1;
                }
            }
            or_done += f1 + f2 + f3;
            // scan tests: whole scans, the last one up to its move
            const std::uint32_t whole = or_opt ? or_len - 1 : lengths;
            checks += (whole >= 1 ? scanned(f1) : f1) + (whole >= 2 ? scanned(f2) : f2) +
                      (whole >= 3 ? scanned(f3) : f3);
        }
        // (an Or-opt move, of an earlier node, comes before the 2-opt one)
        const std::uint32_t popped = or_opt ? or_node + 1 : two_opt ? node_of + 1 : nodes;
        std::uint32_t before = 0;   // 2-opt evaluations of the pops, or up to the 2-opt move
#pragma unroll
        for (std::uint32_t t = 1; t <= kPopNodes; ++t)
            if (popped == t) before = off[2 * t];
        if (two_opt && !or_opt) before = move_t + 1;
        if (tight && before + or_done > left) {
            // the budget ends inside this node's scans
            std::uint32_t rest = left;
            const std::uint32_t f[5] = {off[1], off[2] - off[1], f1, f2, f3};
#pragma unroll
            for (std::uint32_t g = 0; g < 5; ++g) {
                if (g >= 2 + lengths || rest == 0xffffffffu) continue;
                const std::uint32_t used = rest < f[g] ? rest : f[g];
                r.checks += scanned(used);
                rest = used < f[g] ? 0xffffffffu : rest - used;
            }
            evaluations += left;
            ++r.processed;
            r.limit_reached = 1;
            break;
        }
        evaluations += before + or_done;
        r.processed += popped;
        r.checks += checks;
#pragma unroll
        for (std::uint32_t g = 0; g < 2 * kPopNodes; ++g) {
            if ((g >> 1) >= popped) continue;
            const std::uint32_t f = off[g + 1] - off[g];
            if (or_opt || !two_opt || g < move_seg) r.checks += scanned(f);
            else if (g == move_seg) r.checks += move_t + 1 - off[g];
        }
        q.head += popped;
        if (q.head >= n) q.head -= n;
        q.pending -= popped;
        // pending flags of the pops; lanes that share a word clear the same bits of it
        std::uint32_t bits = 0;
#pragma unroll
        for (std::uint32_t t = 0; t < kPopNodes; ++t)
            if (t < popped && (head[t] >> 5) == (a >> 5)) bits |= 1u << (head[t] & 31u);
        if (role == 0 && (lane >> 3) < popped) s.queued[a >> 5] &= ~bits;
        __syncwarp();
        if (or_opt) {
            const std::uint32_t own = 8 * or_node;
            const std::uint32_t prev = __shfl_sync(kFull, near, own), node = __shfl_sync(kFull, near, own + 1);
            const std::uint32_t e = __shfl_sync(kFull, near, own + or_len), next = __shfl_sync(kFull, near, own + or_len + 1);
            // (0) c, a .. e, c2: a goes after c, then each next node after the last moved
            // (1) c0, e .. a, c: e goes after c0, then each previous node
            std::uint32_t target = or_side ? or_nb : or_c;
            for (std::uint32_t t = 0; t < or_len; ++t) {
                const std::uint32_t moved = __shfl_sync(kFull, near, own + 1 + (or_side ? or_len - 1 - t : t));
                const std::uint32_t tp = s.pos[target], np = s.pos[moved];
                relocate_shift<kGlobal>(s, lane, tp, np, moved);
                r.moved += tp < np ? np - tp : tp - np + 1;
                target = moved;
            }
            const std::uint32_t v = lane == 0 ? prev : lane == 1 ? node : lane == 2 ? e : lane == 3 ? next
                                  : lane == 4 ? (or_side ? or_nb : or_c) : (or_side ? or_c : or_nb);
            bool want = lane < 6;
#pragma unroll
            for (std::uint32_t t = 0; t < 5; ++t)
                if (__shfl_sync(kFull, v, t) == v && t < lane) want = false;   // already in the list
            r.reactivations += push_lanes(s, q, n, v, want, lane, log, log_cap);
            ++r.accepted;
            gain_sum -= or_gain;
        } else if (two_opt) {
            const std::uint32_t own = 8 * node_of + (move_seg & 1u);
            const std::uint32_t node = __shfl_sync(kFull, a, own), close = __shfl_sync(kFull, X, own);
            const bool back = move_seg & 1u;
            const std::uint32_t m0 = back ? node : close, m1 = back ? move_c : move_nb;
            const std::uint32_t m2 = back ? close : node, m3 = back ? move_nb : move_c;
            r.moved += flip<kGlobal>(s, n, lane, s.pos[m0], s.pos[m1]);
            r.reactivations += push_lanes(s, q, n, lane == 0 ? m0 : lane == 1 ? m1 : lane == 2 ? m2 : m3, lane < 4,
                                          lane, log, log_cap);
            ++r.accepted;
            gain_sum -= move_gain;
        }
    }
    r.evaluations += evaluations;
}

}  // namespace faco

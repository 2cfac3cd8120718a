// faco_kernels.cu -- the FACO iteration kernels for sm_103a.
//
//   ant_kernel<mode>        construction + local search, one warp per ant
//   colony_init_kernel      reset_colony + initialize_products
//                           (cuda/colony_state.cuh:72-110)
//   colony_update_kernel    reduce_and_select + update_pheromone fused, one
//                           block per colony (cuda/colony_state.cuh:148-229),
//                           with the controllers' per-batch work
//   fingerprint_kernel      tour fingerprints for the 12-feature controller,
//                           one warp per ant (cuda/control_state.cuh:45-64)
//   pheromone_step_kernel   the trail update alone (parity hook)
//   score_kernel            GP controller scoring, warp per colony
//                           (cuda/gp_score.cuh:64-102)
#include <mutex>
#include <climits>
#include <type_traits>

#include "faco_ant.cuh"
#include "faco_kernels.h"

namespace faco {

// ---------------------------------------------------------------------------
// Ant kernel
// ---------------------------------------------------------------------------
// Copies a parent tour into the warp's tour/inverse.  Engine parents are
// 16-byte aligned with padded rows, so lanes move 8 nodes per load.  In the
// global-memory workspace the inverse, which the colony's update writes once,
// is copied the same way: scattered to global memory by every ant it was an
// eighth of an ant's time (the large panel 107 -> 90 ms).  In shared memory the
// scatter is the cheaper one (the uneven batch 82 ms, copied 85).
__device__ __forceinline__ void load_parent(const AntSmem& s, const node_t* parent, const node_t* inverse,
                                            std::uint32_t n, std::uint32_t lane, bool aligned) {
    if (aligned && inverse) {
        const uint4 *tour = reinterpret_cast<const uint4*>(parent), *pos = reinterpret_cast<const uint4*>(inverse);
        constexpr std::uint32_t kEach = kRound<true>;
        for (std::uint32_t first = lane; first * 8 < n; first += 32 * kEach) {
            uint4 a[kEach], b[kEach];
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const std::uint32_t c = first + 32 * u;
                if (c * 8 >= n) continue;
                a[u] = load_written(tour + c);
                b[u] = load_written(pos + c);
            }
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u) {
                const std::uint32_t c = first + 32 * u;
                if (c * 8 >= n) continue;
                reinterpret_cast<uint4*>(s.tour)[c] = a[u];
                reinterpret_cast<uint4*>(s.pos)[c] = b[u];
            }
        }
    } else if (aligned) {
        const uint4* src = reinterpret_cast<const uint4*>(parent);
        uint4* dst = reinterpret_cast<uint4*>(s.tour);
        for (std::uint32_t c = lane; c * 8 < n; c += 32) {
            const uint4 v = load_written(src + c);
            dst[c] = v;
            const std::uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const std::uint32_t i = c * 8 + t;
                if (i < n) s.pos[(words[t >> 1] >> (16 * (t & 1))) & 0xffffu] = (node_t)i;
            }
        }
    } else {
        for (std::uint32_t i = lane; i < n; i += 32) {
            const std::uint32_t v = parent[i];
            s.tour[i] = (node_t)v;
            s.pos[v] = (node_t)i;
        }
    }
}

// the variant's own budget, inside the kernel template
#define kAntBlocksPerSM (ant_blocks_per_sm(MODE))

template <int MODE>
__global__ void __launch_bounds__(kMaxWarpsPerBlock * 32, kAntBlocksPerSM) ant_kernel(const AntLaunch L) {
    constexpr bool kEngine = engine_mode(MODE), kGlobalWs = global_mode(MODE), kFollow = follow_mode(MODE);
    extern __shared__ __align__(16) unsigned char smem[];
    const std::uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    std::uint32_t colony = 0, ant = 0, task = 0;
    bool active;
    if (kEngine) {
        const uint2 job = L.work[blockIdx.x];
        colony = job.x;
        ant = job.y + warp;
        active = ant < L.ants;
    } else {
        task = blockIdx.x * L.warps + warp;
        ant = task;
        active = task < L.tasks;
    }
    const InstanceView* in_ptr = L.instances + (kEngine ? L.colonies[colony].instance : 0);
    const InstanceView in = *in_ptr;
    const std::uint32_t n = in.n;
    const int2* xy;
    if (kGlobalWs) {
        xy = in.xy;
    } else {
        int2* staged = reinterpret_cast<int2*>(smem);
        for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) staged[i] = in.xy[i];
        __syncthreads();
        xy = staged;
    }
    // the previous iteration's update: its parent, trails and state from here on
    wait_previous_kernel();
    if (!active) return;

    node_t* ring = kEngine ? L.colonies[colony].ant_tours + (size_t)ant * L.colonies[colony].n_pad
                           : L.out_tours + (size_t)task * n;
    AntSmem s;
    if (kGlobalWs) {
        const std::uint32_t n_pad = L.colonies[colony].n_pad;
        node_t* ws = L.workspace + 2 * ((size_t)(L.colonies[colony].ant_tours - L.ant_tours_base) +
                                        (size_t)ant * n_pad);
        s = AntSmem::split(ws, n_pad, smem + warp * ant_bitset_bytes(L.n_max), L.n_max, ring);
    } else {
        s = AntSmem::at(smem + ((8u * L.n_max + 15u) & ~15u) + warp * ant_smem_bytes(L.n_max), L.n_max, ring);
    }
    const node_t* parent;
    const std::uint32_t* parent_nbr;
    long long cost;
    std::uint32_t target, batch = 0, region = 4;
    unsigned long long key = 0;
    ColonyView cv{};
    if (kEngine) {
        cv = L.colonies[colony];
        const ColonyState& st = L.states[colony];
        parent = cv.parent;
        parent_nbr = cv.parent_nbr;
        cost = st.parent_cost;
        target = st.mne_target;
        batch = st.iteration;
        region = st.region;
        key = cv.key;
    } else {
        parent = L.task_tours + (size_t)task * n;
        parent_nbr = L.task_nbr + (size_t)task * n;
        cost = L.task_costs[task];
        target = MODE == kModePrepare ? 0 : L.task_targets[task];
    }
    load_parent(s, parent, kGlobalWs ? cv.parent_pos : nullptr, n, lane, kEngine);
    const std::uint32_t words = (n + 31) / 32;
    for (std::uint32_t i = lane; i < words; i += 32) {
        s.visited[i] = 0;
        s.queued[i] = MODE == kModePrepare ? ~0u : 0u;
    }
    __syncwarp();

    std::uint32_t* log = L.out_checklist ? L.out_checklist + (size_t)task * L.checklist_cap : nullptr;
    const std::uint32_t log_cap = L.checklist_cap;
    Checklist q{0, 0, 0, 0};
    AntResult r{};

    if (MODE == kModePrepare) {
        // registration: every node pending, in tour order (prepared_problem.cpp:160-162)
        for (std::uint32_t i = lane; i < n; i += 32) {
            s.ring[i] = s.tour[i];
            if (log && i < log_cap) log[i] = s.tour[i];
        }
        q.tail = 0;
        q.pending = n;
        q.pushed = n;
        __syncwarp();
    } else {
        // ---------------- focused construction ----------------
        std::uint32_t current;
        if (kEngine) current = region == 5 ? list_start(key, batch, ant, cv.control->start_nodes,
                                                        cv.control->start_count)
                                           : region_start(key, batch, ant, in_ptr, region);
        else if (MODE == kModeVisits) current = L.task_visits[(size_t)task * n];
        else current = L.task_starts[task];
        if (L.out_selected && lane == 0) L.out_selected[(size_t)task * n] = (node_t)current;
        if (lane == 0) s.visited[current >> 5] |= 1u << (current & 31u);
        __syncwarp();
        const float* products = kEngine ? cv.products : L.task_products;
        const std::uint32_t k = in.k;
        const unsigned long long loop_cap = 2ull * n + 2;
        unsigned long long guard = 0;
        // the construction draws of 32 consecutive steps at a time, lane i
        // holding step draw_base + i (the same counters as one draw per step)
        std::uint32_t draw_base = 0x80000000u, draw_hi = 0, draw_lo = 0;   // steps < 2^16: first step refreshes
        // the candidate row of the likely next node, loaded one step ahead:
        // once trails converge an ant mostly walks the parent tour, so the
        // next node is the parent neighbour of `current` not yet visited
        std::uint32_t next_node = n, next_pnbr = 0, next_cand = n;
        float next_p = 0.0f;
        RelocationRun run;
        // steps along the parent tour are taken in batches (follow_batch)
        // until a batch stops short of its lanes; the step it stopped at is
        // taken alone, then batches resume.  A colony whose walks are short
        // takes every step alone: the batches' setup is lost on them
        const bool batches = kFollow && (L.batch_from == 0 || *cv.walk >= L.batch_from);
        bool follow = batches;
        while (r.mne < target && r.steps + 1 < n) {
            if (++guard > loop_cap) { if (lane == 0) atomicOr(L.error, kErrLoopCap); break; }
            if (kFollow && follow) {
                bool full = false;
                const std::uint32_t f = follow_batch(s, xy, in, products, parent_nbr, n, lane, key, batch,
                                                             ant, current, r, cost, run, draw_base, draw_hi, draw_lo,
                                                             full);
                follow = full;
                if (f) continue;
            }
            follow = batches;
            const std::uint32_t step = r.steps + 1;
            if (kEngine && step - draw_base >= 32u) {
                draw_base = step;
                const uint4v rb = philox4x32(step + lane, ant, batch, 0, (std::uint32_t)key, (std::uint32_t)(key >> 32));
                draw_hi = rb.x;
                draw_lo = rb.y;
            }
            // loads that depend only on `current`, issued first
            std::uint32_t pnbr, cand = n;
            float p = 0.0f;
            if (kEngine && current == next_node) {
                pnbr = next_pnbr;
                cand = next_cand;
                p = next_p;
            } else {
                pnbr = load_written(parent_nbr + current);
                if (MODE != kModeVisits && lane < k) {
                    cand = __ldg(in.primary + (size_t)current * k + lane);
                    p = load_written(products + (size_t)current * k + lane);
                }
            }
            if (kEngine) {
                const std::uint32_t ps = pnbr & 0xffffu;
                next_node = test_bit(s.visited, ps) ? pnbr >> 16 : ps;
                next_pnbr = load_written(parent_nbr + next_node);
                next_cand = n;
                next_p = 0.0f;
                if (lane < k) {
                    next_cand = __ldg(in.primary + (size_t)next_node * k + lane);
                    next_p = load_written(products + (size_t)next_node * k + lane);
                }
            }
            std::uint32_t selected = n;
            if (MODE == kModeVisits) {
                selected = L.task_visits[(size_t)task * n + step];
            } else {
                std::uint32_t rhi = 0, rlo = 0;
                double u_given = 0.0;
                float uf;
                if (kEngine) {
                    rhi = __shfl_sync(kFull, draw_hi, step - draw_base);
                    rlo = __shfl_sync(kFull, draw_lo, step - draw_base);
                    uf = __uint2float_rn(rhi) * 0x1p-32f;
                } else {
                    u_given = L.task_uniforms[(size_t)task * n + step];
                    uf = (float)u_given;
                }
                const bool avail = cand < n && !test_bit(s.visited, cand);
                const unsigned mask = __ballot_sync(kFull, avail);
                if (mask) {
                    // FP32 inclusive scan of the available weights.  Each prefix is
                    // within 5 roundings (< 3.1e-7 relative) of the exact prefix, the
                    // threshold u*total within 4.3e-7; a choice is taken only when the
                    // first candidate not certainly below the threshold is certainly
                    // above it by delta = total * 2^-19 (> 1.9e-6), which the FP64
                    // ordered sums of the reference then decide identically.
                    const float pv = avail ? p : 0.0f;
                    float scan = pv;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float t = __shfl_up_sync(kFull, scan, o);
                        if ((int)lane >= o) scan += t;
                    }
                    const float tot = __shfl_sync(kFull, scan, 31);
                    int j = -1;
                    if (tot >= 0x1p-100f) {
                        const float thr = uf * tot, delta = tot * 0x1p-19f, diff = scan - thr;
                        const unsigned yes = __ballot_sync(kFull, avail && diff > delta);
                        const unsigned maybe = __ballot_sync(kFull, avail && diff >= -delta);
                        if (maybe != 0u && (maybe & (0u - maybe)) == (yes & (0u - yes))) j = __ffs(yes) - 1;
                    }
                    if (j < 0) {
                        // exact path: ordered FP64 prefix sums (faco_cpu.cpp:254-279)
                        const double u = kEngine ? u53(rhi, rlo) : u_given;
                        double total = 0.0, mine = 0.0;
                        for (unsigned m = mask; m; m &= m - 1) {
                            const int jj = __ffs(m) - 1;
                            total += (double)__shfl_sync(kFull, p, jj);
                            if ((int)lane == jj) mine = total;
                        }
                        if (total > 0.0) {
                            const double threshold = u * total;
                            const unsigned hit = __ballot_sync(kFull, avail && threshold < mine);
                            j = hit ? __ffs(hit) - 1 : 31 - __clz(mask);
                        } else {
                            const std::uint32_t count = __popc(mask);
                            std::uint32_t t = (std::uint32_t)(u * count);
                            if (t >= count) t = count - 1;
                            unsigned m = mask;
                            for (; t; --t) m &= m - 1;
                            j = __ffs(m) - 1;
                        }
                    }
                    selected = __shfl_sync(kFull, cand, j);
                } else {
                    const std::uint32_t b = in_ptr->b;   // rare: read where it is used
                    for (std::uint32_t base_j = 0; base_j < b && selected == n; base_j += 32) {
                        const std::uint32_t jj = base_j + lane;
                        std::uint32_t v = n;
                        bool ok = false;
                        if (jj < b) {
                            v = __ldg(in_ptr->backup + (size_t)current * b + jj);
                            ok = v < n && !test_bit(s.visited, v);
                        }
                        const unsigned m = __ballot_sync(kFull, ok);
                        if (m) selected = __shfl_sync(kFull, v, __ffs(m) - 1);
                    }
                    if (selected == n) {
                        // global nearest unvisited, lowest id on ties
                        unsigned long long bestkey = ~0ull;
                        const int2 cxy = xy[current];
                        for (std::uint32_t v = lane; v < n; v += 32) {
                            if (test_bit(s.visited, v)) continue;
                            const unsigned long long kv =
                                ((unsigned long long)(unsigned)euc2d(cxy, xy[v]) << 32) | v;
                            bestkey = kv < bestkey ? kv : bestkey;
                        }
                        for (int o = 16; o; o >>= 1) {
                            const unsigned long long other = __shfl_xor_sync(kFull, bestkey, o);
                            bestkey = other < bestkey ? other : bestkey;
                        }
                        if (bestkey != ~0ull) selected = (std::uint32_t)(bestkey & 0xffffffffu);
                    }
                }
            }
            if (selected >= n || test_bit(s.visited, selected)) {
                // no legal choice (only an invalid explicit visit order can get here)
                if (lane == 0) atomicOr(L.error, kErrBadChoice);
                break;
            }
            if (L.out_selected && lane == 0) L.out_selected[(size_t)task * n + step] = (node_t)selected;
            // positions and tour neighbours, read through the deferred run
            // when `selected` continues it, else from the rewritten tour
            std::uint32_t npos = s.pos[selected], tpos = n, previous = n, after = n, target_after = n;
            int run_dir = 0;
            bool start_run = false;
            if (run.m) {
                // the inverse is that of the tour before the run (unchanged during it)
                run_dir = run.continues(npos);
                if (run_dir) {
                    npos = run.source_pos(run_dir);
                    tpos = run.current_pos();
                    target_after = run.read(s, tpos + 1 == n ? 0 : tpos + 1);
                    if (target_after == selected) run_dir = 0;
                }
                if (run_dir) {
                    if constexpr (kFollow) {
                        // the batched-step variants are bound by instruction
                        // fetch: one copy of the run's read in their code
#pragma unroll 1
                        for (int t = 0; t < 2; ++t) {
                            const std::uint32_t x = run.read(s, t == 0 ? (npos == 0 ? n - 1 : npos - 1)
                                                                       : (npos + 1 == n ? 0 : npos + 1));
                            if (t == 0) previous = x;
                            else after = x;
                        }
                    } else {
                        previous = run.read(s, npos == 0 ? n - 1 : npos - 1);
                        after = run.read(s, npos + 1 == n ? 0 : npos + 1);
                    }
                } else {
                    run.apply<kGlobalWs>(s, lane, current);
                    npos = s.pos[selected];
                }
            }
            if (!run_dir) {
                tpos = s.pos[current];
                previous = s.tour[npos == 0 ? n - 1 : npos - 1];
                after = s.tour[npos + 1 == n ? 0 : npos + 1];
                target_after = s.tour[tpos + 1 == n ? 0 : tpos + 1];
                // relocations are deferred on large instances, and on the
                // others once the walk is long (converged trails)
                start_run = n > kDeferAllFrom || r.steps >= kDeferFromStep;
            }
            ++r.steps;
            __syncwarp();
            if (lane == 0) s.visited[selected >> 5] |= 1u << (selected & 31u);
            if (target_after != selected) {
                ++r.nonidentity;
                // six-edge delta of CpuTour::relocate, one term per lane
                int term = 0;
                if (lane < 6) {
                    // removed: (previous,selected) (selected,after) (current,target_after)
                    // added:   (previous,after) (current,selected) (selected,target_after)
                    const std::uint32_t e0 = lane == 0 || lane == 3 ? previous : lane == 2 || lane == 4 ? current
                                                                                                        : selected;
                    const std::uint32_t e1 = lane == 0 || lane == 4 ? selected : lane == 1 || lane == 3 ? after
                                                                                                        : target_after;
                    const int d = euc2d(xy[e0], xy[e1]);
                    term = lane < 3 ? -d : d;
                }
                cost += __reduce_add_sync(kFull, term);
                if (run_dir) {
                    // the run takes one more node
                    run.dir = run_dir;
                    ++run.m;
                } else if (start_run) {
                    // a deferred run, of this relocation alone so far
                    run.p = npos;
                    run.t = tpos;
                    run.m = 1;
                    run.dir = 1;
                } else {
                    relocate_shift<kGlobalWs>(s, lane, tpos, npos, selected);
                }
                r.moved += tpos < npos ? npos - tpos : tpos - npos + 1;
            }
            const bool new_edge = (pnbr & 0xffffu) != selected && (pnbr >> 16) != selected;
            if (new_edge) {
                ++r.mne;
                // (the node before `selected` is `current` itself on a step onto the next tour node)
                push_lanes(s, q, n, lane == 0 ? current : lane == 1 ? selected : previous,
                           lane < (previous == current ? 2u : 3u), lane, log, log_cap);
            }
            current = selected;
            __syncwarp();
        }
        if (run.m) run.apply<kGlobalWs>(s, lane, current);
        r.construction_cost = cost;
        if (L.out_construction)
            for (std::uint32_t i = lane; i < n; i += 32) L.out_construction[(size_t)task * n + i] = s.tour[i];
        __syncwarp();
    }
    start_next_kernel();   // the update may launch; it waits for the last ant
    // ---------------- local search ----------------
    // (the instance's and the colony's fields are read again where a phase
    // uses them: kept from the start they would hold 20 registers)
    long long gain_sum = 0;
    const InstanceView ls_in = *in_ptr;
    if ((MODE & kOrOptOnly) || (!(MODE & kTwoOptOnly) && L.ls_mode == 1)) checklist_ls_first<kGlobalWs>(s, xy, ls_in, n, lane, q, L.ls_limit, r, gain_sum, log, log_cap);
    else checklist_two_opt<kGlobalWs>(s, xy, ls_in, n, lane, q, L.ls_limit, r, gain_sum, log, log_cap);
    r.final_cost = cost + gain_sum;
    r.checklist = q.pushed;
    if (log && q.pushed > log_cap && lane == 0) atomicOr(L.error, kErrQueueOverflow);
    __syncwarp();

    if (kEngine) {
        const ColonyView& to = L.colonies[colony];
        uint4* out = reinterpret_cast<uint4*>(to.ant_tours + (size_t)ant * to.n_pad);
        const uint4* src = reinterpret_cast<const uint4*>(s.tour);
        constexpr std::uint32_t kEach = kRound<kGlobalWs>;
        for (std::uint32_t first = lane; first * 8 < n; first += 32 * kEach) {
            uint4 v[kEach];
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u)
                if ((first + 32 * u) * 8 < n) v[u] = src[first + 32 * u];
#pragma unroll
            for (std::uint32_t u = 0; u < kEach; ++u)
                if ((first + 32 * u) * 8 < n) out[first + 32 * u] = v[u];
        }
        if (lane == 0) {
            to.ant_costs[ant] = r.final_cost;
            to.ant_ccosts[ant] = r.construction_cost;
            to.ant_counts[3 * ant] = r.steps;
            to.ant_counts[3 * ant + 1] = (unsigned)r.evaluations;
            to.ant_counts[3 * ant + 2] = (unsigned)r.moved;
        }
    } else {
        if (L.out_tours)
            for (std::uint32_t i = lane; i < n; i += 32) L.out_tours[(size_t)task * n + i] = s.tour[i];
        if (L.out_pos)
            for (std::uint32_t i = lane; i < n; i += 32) L.out_pos[(size_t)task * n + i] = s.pos[i];
        if (lane == 0) {
            if (L.out_costs) {
                L.out_costs[2 * (size_t)task] = r.construction_cost;
                L.out_costs[2 * (size_t)task + 1] = r.final_cost;
            }
            if (L.out_counters) {
                unsigned long long* c = L.out_counters + 10 * (size_t)task;
                c[0] = r.mne; c[1] = r.steps; c[2] = r.nonidentity; c[3] = r.processed; c[4] = r.checks;
                c[5] = r.evaluations; c[6] = r.accepted; c[7] = r.reactivations; c[8] = r.limit_reached;
                c[9] = r.checklist;
            }
        }
    }
}

namespace {
// The dynamic shared-memory limit is a per-kernel, per-device attribute that
// every engine on the device shares, and instantiated graphs launch against
// it: it is only ever raised, so that one engine's smaller classes never
// invalidate another engine's larger ones.
template <int MODE>
cudaError_t prepare_mode(std::uint32_t smem) {
    static std::mutex lock;
    static std::uint32_t raised[64] = {};
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    std::lock_guard<std::mutex> guard(lock);
    std::uint32_t& current = raised[device & 63];
    if (smem <= current) return cudaSuccess;
    err = cudaFuncSetAttribute(ant_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess) current = smem;
    return err;
}
}  // namespace

namespace {
// f(variant) for the kernel variant of a mode and local search.
template <class F>
cudaError_t for_variant(int mode, std::uint32_t ls_mode, F&& f) {
    const auto engine = [&](auto m) {
        constexpr int kMode = decltype(m)::value;
        return ls_mode == 1 ? f(std::integral_constant<int, kMode | kOrOptOnly>{})
                            : f(std::integral_constant<int, kMode | kTwoOptOnly>{});
    };
    switch (mode) {
        case kModeEngine: return engine(std::integral_constant<int, kModeEngine>{});
        case kModeVisits: return f(std::integral_constant<int, kModeVisits>{});
        case kModeUniforms: return f(std::integral_constant<int, kModeUniforms>{});
        case kModePrepare: return f(std::integral_constant<int, kModePrepare>{});
        case kModeEngineGlobal: return engine(std::integral_constant<int, kModeEngineGlobal>{});
        case kModeEngineFollow: return engine(std::integral_constant<int, kModeEngineFollow>{});
        case kModeEngineGlobalFollow: return engine(std::integral_constant<int, kModeEngineGlobalFollow>{});
        case kModeEngineFollowDense: return engine(std::integral_constant<int, kModeEngineFollowDense>{});
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace

cudaError_t prepare_ant_kernel(int mode, std::uint32_t ls_mode, std::uint32_t smem) {
    return for_variant(mode, ls_mode, [&](auto m) { return prepare_mode<decltype(m)::value>(smem); });
}

// Launches `kernel`, with `overlapped` as a programmatic dependent of the
// kernel before it on the stream: its prologue, up to wait_previous_kernel(),
// overlaps that kernel.
template <class... Params, class... Args>
static cudaError_t launch_overlapped(bool overlapped, void (*kernel)(Params...), std::uint32_t blocks,
                                     std::uint32_t threads, std::uint32_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = overlapped ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

cudaError_t launch_ant_kernel(int mode, const AntLaunch& L, std::uint32_t blocks, std::uint32_t warps,
                              std::uint32_t smem, cudaStream_t stream, bool overlapped) {
    return for_variant(mode, L.ls_mode, [&](auto m) {
        return launch_overlapped(overlapped, ant_kernel<decltype(m)::value>, blocks, warps * 32, smem, stream, L);
    });
}

// ---------------------------------------------------------------------------
// Colony kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ void trail_limits(long long cost, double retention, double p_root, std::uint32_t k,
                                             float& tmin, float& tmax) {
    const double mx = 1.0 / ((double)cost * (1.0 - retention));
    double mn = mx * (1.0 - p_root) / (((double)k - 1.0) * p_root);
    mn = mn < mx ? mn : mx;
    tmax = (float)mx;
    tmin = (float)mn;
}

// MMAS evaporate/deposit on FP32 trails (cuda/colony_state.cuh:210-229):
// tau <- max(tau_min, tau * retention); a directed candidate entry (from, to)
// on the parent tour also gains min(tau_max, tau + 1/parent_cost); products
// are refreshed as tau * eta.  The parent-edge test reads the packed parent
// neighbours of `from`.  Threads stride over entries, four at a time when the
// row width allows 16-byte accesses.
__device__ __forceinline__ float trail_value(float tau, std::uint32_t to, std::uint32_t nb, float ret, float tmin,
                                             float tmax, float inc) {
    float v = fmaxf(tmin, tau * ret);
    if (to == (nb & 0xffffu) || to == (nb >> 16)) v = fminf(tmax, v + inc);
    return v;
}

__device__ __forceinline__ void trail_update(std::uint32_t n, std::uint32_t k, const node_t* __restrict__ primary,
                                             const std::uint32_t* __restrict__ nbr, float ret, float tmin, float tmax,
                                             float inc, const float* __restrict__ eta, float* __restrict__ trails,
                                             float* __restrict__ products, std::uint32_t first, std::uint32_t stride) {
    const std::uint32_t cells = n * k;
    if ((k & 3u) == 0) {
        // groups of four entries, two in flight; the group's row by carry
        const std::uint32_t per_row = k / 4, groups = cells / 4, step_rows = stride / per_row,
                            step_rest = stride - step_rows * per_row;
        std::uint32_t row = first / per_row, rest = first - row * per_row;
        for (std::uint32_t q = first; q < groups;) {
            float4 t[2], e[2];
            uint2 pr[2];
            std::uint32_t nb[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const std::uint32_t at = q + u * stride;
                if (at >= groups) continue;
                t[u] = reinterpret_cast<const float4*>(trails)[at];
                e[u] = reinterpret_cast<const float4*>(eta)[at];
                pr[u] = reinterpret_cast<const uint2*>(primary)[at];
                nb[u] = nbr[row];
                row += step_rows;
                rest += step_rest;
                if (rest >= per_row) { rest -= per_row; ++row; }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const std::uint32_t at = q + u * stride;
                if (at >= groups) continue;
                float4 v;
                v.x = trail_value(t[u].x, pr[u].x & 0xffffu, nb[u], ret, tmin, tmax, inc);
                v.y = trail_value(t[u].y, pr[u].x >> 16, nb[u], ret, tmin, tmax, inc);
                v.z = trail_value(t[u].z, pr[u].y & 0xffffu, nb[u], ret, tmin, tmax, inc);
                v.w = trail_value(t[u].w, pr[u].y >> 16, nb[u], ret, tmin, tmax, inc);
                reinterpret_cast<float4*>(trails)[at] = v;
                reinterpret_cast<float4*>(products)[at] = make_float4(v.x * e[u].x, v.y * e[u].y, v.z * e[u].z,
                                                                      v.w * e[u].w);
            }
            q += 2 * stride;
        }
    } else {
        for (std::uint32_t idx = first; idx < cells; idx += stride) {
            const float v = trail_value(trails[idx], primary[idx], nbr[idx / k], ret, tmin, tmax, inc);
            trails[idx] = v;
            products[idx] = v * eta[idx];
        }
    }
}

// Products of a colony whose prior re-ranks departures only: per node row,
// the parent-tour entries keep the instance heuristic (products = trail *
// eta), and the other entries take the prior's heuristic scaled so that
// their total weight equals the plain total, sum(trail * eta) over the
// non-parent entries.  An ant then leaves the parent tour as often as a
// plain ant does, and the prior only decides where it goes.  Rows over
// [first, n) with the given stride; trails are already updated.
__device__ __forceinline__ void departure_rows(const InstanceView& in, const ColonyView& cv, std::uint32_t first,
                                               std::uint32_t stride, std::uint32_t end) {
    const std::uint32_t k = in.k;
    for (std::uint32_t i = first; i < end; i += stride) {
        const std::uint32_t nb = cv.parent_nbr[i], succ = nb & 0xffffu, pred = nb >> 16;
        const std::size_t row = (std::size_t)i * k;
        float plain = 0.0f, prior = 0.0f;
        for (std::uint32_t j = 0; j < k; ++j) {
            const std::uint32_t node = in.primary[row + j];
            if (node == succ || node == pred) continue;
            const float t = cv.trails[row + j];
            plain += t * in.eta[row + j];
            prior += t * cv.eta[row + j];
        }
        const float scale = prior > 0.0f ? plain / prior : 1.0f;
        for (std::uint32_t j = 0; j < k; ++j) {
            const std::uint32_t node = in.primary[row + j];
            const float t = cv.trails[row + j];
            cv.products[row + j] = node == succ || node == pred ? t * in.eta[row + j] : t * cv.eta[row + j] * scale;
        }
    }
}

// ---------------------------------------------------------------------------
// GP controller pieces (the engine's feature spec 3; the same arithmetic is
// restated on the CPU beside the oracle colony run).
// ---------------------------------------------------------------------------
// log2 from the exponent and the atanh series of the mantissa,
// m in [sqrt(2)/2, sqrt(2)): log2 m = (2/ln 2) (t + t^3/3 + t^5/5 + t^7/7),
// t = (m-1)/(m+1).  Single-rounding FP32 operations only, so that the CPU
// computes identical bits.
__device__ __forceinline__ float own_log2(float x) {
    const std::uint32_t bits = __float_as_uint(x);
    int e = (int)((bits >> 23) & 255u) - 127;
    float m = __uint_as_float((bits & 0x7FFFFFu) | 0x3F800000u);
    if (m > 0x1.6a09e6p+0f) { m = m * 0.5f; e += 1; }
    const float t = (m - 1.0f) / (m + 1.0f), t2 = t * t;
    const float s = t * (1.0f + t2 * (0x1.555556p-2f + t2 * (0x1.99999ap-3f + t2 * 0x1.24924ap-3f)));
    return (float)e + s * 0x1.715476p+1f;
}

// Normalised Shannon entropy of one trail row, in units of 2^-20.
__device__ __forceinline__ std::uint32_t row_entropy_q(const float* tau, std::uint32_t k, float log2k) {
    float sum = 0.0f;
    for (std::uint32_t j = 0; j < k; ++j) sum = sum + tau[j];
    if (!(sum > 0.0f)) return 0;
    float h = 0.0f;
#pragma unroll 4
    for (std::uint32_t j = 0; j < k; ++j) {   // the divisions of four entries overlap, the sum stays in order
        const float p = tau[j] / sum;
        const float term = p * own_log2(p > 0.0f ? p : 1.0f);
        h = p > 0.0f ? h - term : h;
    }
    float hn = h / log2k;
    hn = hn < 0.0f ? 0.0f : hn > 1.0f ? 1.0f : hn;
    return (std::uint32_t)(hn * 1048576.0f + 0.5f);
}

__device__ __forceinline__ float apply_operation(int op, float l, float r, float t) {
    float v = 0.0f;
    switch (op) {
        case 2: v = l + r; break;
        case 3: v = l - r; break;
        case 4: v = l * r; break;
        case 5: v = fminf(l, r); break;
        case 6: v = fmaxf(l, r); break;
        case 7: v = fabsf(l); break;
        case 8: { const float q = 1.0f + r * r; v = l * (1.0f / sqrtf(q)); break; }
        case 9: v = fabsf(r) < 1e-6f ? 1.0f : l / r; break;
        case 10: v = l > 0.0f ? r : t; break;
        default: break;
    }
    return fminf(8.0f, fmaxf(-8.0f, v));
}

// A program in shared memory: the interpreter's loop reads one word per
// instruction, ahead of its use (opcode | operand << 8).
struct StagedProgram {
    std::uint32_t length;
    std::uint16_t code[64];
    float constants[63];
};

__device__ __forceinline__ void stage_program(const Program& p, StagedProgram& to, std::uint32_t lane) {
    for (std::uint32_t i = lane; i < 63; i += 32) {
        to.code[i] = (std::uint16_t)(p.opcode[i] | p.operand[i] << 8);
        to.constants[i] = p.constants[i];
    }
    if (lane == 0) {
        to.length = p.length;
        to.code[63] = 0;
    }
}

// Postfix interpreter (cuda/gp_score.cuh:64-102); feature(i) supplies terminal
// i.  The top of the stack stays in a register; the rest is one shared column
// per lane (stack[d][lane], 15 deep).  A chain of one latency after the other:
// from global memory with the stack in local memory a 63-node program took
// 11-14 thousand cycles.
template <class Feature>
__device__ __forceinline__ float eval_program(const StagedProgram& p, float (*stack)[32], std::uint32_t lane,
                                              Feature feature) {
    float top = 0.0f;
    int depth = 0;                 // entries below `top`, which is the first push's when depth < 0
    --depth;
    std::uint32_t next = p.code[0];
#pragma unroll 1
    for (std::uint32_t i = 0; i < p.length; ++i) {
        const std::uint32_t op = next & 255u, operand = next >> 8;
        next = p.code[i + 1];
        if (op < 2) {
            if (depth >= 0) stack[depth][lane] = top;
            ++depth;
            top = op == 0 ? feature((int)operand) : p.constants[operand];
        } else if (op == 7) {
            top = apply_operation(7, top, 0.0f, 0.0f);
        } else {
            const float t = op == 10 ? top : 0.0f;
            const float r = op == 10 ? stack[--depth][lane] : top;
            const float l = stack[--depth][lane];
            top = apply_operation((int)op, l, r, t);
        }
    }
    return top;
}

// First maximum within 1e-6 among legal lanes (score_cpu rule); 32 if none.
__device__ __forceinline__ std::uint32_t choose_action(float value, bool legal, std::uint32_t lane) {
    float maximum = legal ? value : -INFINITY;
    for (int o = 16; o; o >>= 1) maximum = fmaxf(maximum, __shfl_xor_sync(kFull, maximum, o));
    return __reduce_min_sync(kFull, legal && maximum - value <= 1e-6f ? lane : 32u);
}

// conditional_three controllers (python/gp_faco/controller.py:60-84,
// cuda/gp_score.cuh role loop): role 0 picks the restart half (2 options,
// stride 16), role 1 the start region (4, stride 4), role 2 the MNE level
// (4, stride 1), each from the prefix the earlier roles fixed.  Lane i <
// width scores the role's tree on the features of action prefix + i*stride
// (feature_of(index, action)); a lane is legal when any action of its
// stride-wide window is; the first maximum within 1e-6 wins.  Role scores
// go to slots 0-1, 2-5 and 6-9 of `role_scores` (may be null).
template <class FeatureOf>
__device__ __forceinline__ std::uint32_t choose_conditional(const StagedProgram* trees, float (*stack)[32],
                                                            FeatureOf feature_of, std::uint32_t mask,
                                                            std::uint32_t lane, float* role_scores) {
    std::uint32_t prefix = 0;
#pragma unroll 1
    for (int role = 0; role < 3; ++role) {
        const std::uint32_t width = role == 0 ? 2u : 4u, stride = role == 0 ? 16u : role == 1 ? 4u : 1u;
        const std::uint32_t action = prefix + (lane < width ? lane : 0u) * stride;
        const bool legal = lane < width && ((mask >> action) & ((1u << stride) - 1u)) != 0u;
        const float value = eval_program(trees[role], stack, lane, [&](int i) { return feature_of(i, action); });
        if (role_scores && lane < width) role_scores[(role == 0 ? 0 : role == 1 ? 2 : 6) + lane] = value;
        const std::uint32_t pick = choose_action(value, legal, lane);
        prefix += stride * (pick < 32u ? pick : 0u);
    }
    return prefix;
}

__device__ __forceinline__ float clamp01(double v) { return (float)(v < 0.0 ? 0.0 : v > 1.0 ? 1.0 : v); }

// ---------------------------------------------------------------------------
// The reference's 12-feature controller (feature spec 2): per batch, after
// the trail update, the ants' fingerprints, the archive of distinct
// near-best tours and the feedback (update_control, control_state.cuh:
// 124-245), then the decision for the next batch -- alternative reference,
// 8 start regions, 12 x 32 features, scoring, and the action (MNE target,
// start list, restart from the alternative; build_control_features and
// apply_control_action, :247-364).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double unit_clip(double v) { return v < 0.0 ? 0.0 : v > 1.0 ? 1.0 : v; }

// A tour in device memory: its order, its positions (may be null) and the
// position of node 0.
struct TourRef {
    const node_t* tour;
    const node_t* pos;
    std::uint32_t p0;
};

__device__ __forceinline__ node_t* archive_tour(const ColonyView& cv, std::uint32_t side, std::uint32_t slot) {
    return cv.archive + (size_t)((side * kArchive + slot) * 2u) * cv.n_pad;
}

// canonical_compare (control_ops.hpp:61-74) by one warp: both tours read
// from node 0 towards its smaller neighbour; -1, 0 or 1.  Each lane loads 16
// elements of both tours before the first vote, so the loads overlap.
__device__ __forceinline__ std::uint32_t canonical_index(std::uint32_t p0, bool forward, std::uint32_t i,
                                                         std::uint32_t n) {
    std::uint32_t x = forward ? p0 + i : p0 + n - i;   // < 2n
    return x >= n ? x - n : x;
}
__device__ int warp_canonical_compare(TourRef a, TourRef b, std::uint32_t n, std::uint32_t lane) {
    constexpr std::uint32_t kUnroll = 16;
    const bool fa = a.tour[a.p0 + 1 == n ? 0 : a.p0 + 1] < a.tour[a.p0 == 0 ? n - 1 : a.p0 - 1];
    const bool fb = b.tour[b.p0 + 1 == n ? 0 : b.p0 + 1] < b.tour[b.p0 == 0 ? n - 1 : b.p0 - 1];
    for (std::uint32_t base = 1; base < n; base += 32 * kUnroll) {
        std::uint32_t va[kUnroll], vb[kUnroll];
#pragma unroll
        for (std::uint32_t u = 0; u < kUnroll; ++u) {
            const std::uint32_t i = base + u * 32 + lane;
            va[u] = i < n ? a.tour[canonical_index(a.p0, fa, i, n)] : 0u;
            vb[u] = i < n ? b.tour[canonical_index(b.p0, fb, i, n)] : 0u;
        }
#pragma unroll
        for (std::uint32_t u = 0; u < kUnroll; ++u) {
            const unsigned m = __ballot_sync(kFull, va[u] != vb[u]);
            if (m) return __shfl_sync(kFull, va[u] < vb[u] ? -1 : 1, __ffs(m) - 1);
        }
    }
    return 0;
}

// XOR of the n edge fingerprints (fingerprint_ants, control_state.cuh:45-64)
// and the position of node 0, by one warp.
__device__ Fingerprint warp_fingerprint(const node_t* tour, std::uint32_t n, std::uint32_t lane, std::uint32_t& p0) {
    unsigned long long f1 = 0, f2 = 0;
    std::uint32_t z = 0xffffffffu;
    for (std::uint32_t base = 0; base < n; base += 128) {
        std::uint32_t a[4], b[4];
#pragma unroll
        for (std::uint32_t u = 0; u < 4; ++u) {
            const std::uint32_t i = base + u * 32 + lane;
            a[u] = i < n ? tour[i] : 0u;
            b[u] = i < n ? tour[i + 1 == n ? 0 : i + 1] : 0u;
        }
#pragma unroll
        for (std::uint32_t u = 0; u < 4; ++u) {
            const std::uint32_t i = base + u * 32 + lane;
            if (i >= n) continue;
            const Fingerprint e = fingerprint_edge(a[u], b[u]);
            f1 ^= e.first;
            f2 ^= e.second;
            if (a[u] == 0) z = i;
        }
    }
    for (int o = 16; o; o >>= 1) {
        f1 ^= __shfl_xor_sync(kFull, f1, o);
        f2 ^= __shfl_xor_sync(kFull, f2, o);
        z = min(z, __shfl_xor_sync(kFull, z, o));
    }
    p0 = z;
    return {f1, f2};
}

// Candidates of the archive selection: 0-3 the archive slots, 4 + a ant a.
// Archive fields come from the shared copy of the controller state; the
// ants' costs, fingerprints and node-0 positions from shared memory when the
// colony has at most kStageAnts ants, else from global memory.
constexpr std::uint32_t kStageAnts = 128;
struct CandidateView {
    const ColonyView& cv;
    const RefControl& ctl;
    const long long* costs;
    const Fingerprint* ids;
    const std::uint32_t* p0s;
    __device__ long long cost(std::uint32_t c) const { return c < kArchive ? ctl.archive_cost[c] : costs[c - kArchive]; }
    __device__ Fingerprint id(std::uint32_t c) const { return c < kArchive ? ctl.archive_id[c] : ids[c - kArchive]; }
    __device__ TourRef ref(std::uint32_t c) const {
        if (c < kArchive) {
            const node_t* t = archive_tour(cv, ctl.side, c);
            return {t, t + cv.n_pad, ctl.archive_p0[c]};
        }
        return {cv.ant_tours + (size_t)(c - kArchive) * cv.n_pad, nullptr, p0s[c - kArchive]};
    }
};

constexpr std::uint32_t kCtlWords = (kArchive + kCtlMaxAnts + 31) / 32;

// The archive band as an integer: an integer cost c exceeds the double
// global_cost * (1 + band) exactly when c exceeds its floor.
__device__ __forceinline__ long long band_limit(long long global_cost) {
    return (long long)floor((double)global_cost * (1 + kArchiveBand));
}

// The least candidate of the warp by (cost, fingerprint, index), in every
// lane; lanes without one hold (LLONG_MAX, all ones, 0xffffffff).
__device__ __forceinline__ void warp_least(std::uint32_t& best, long long& cost, Fingerprint& id) {
#pragma unroll 1
    for (int o = 16; o; o >>= 1) {
        const std::uint32_t ob = __shfl_xor_sync(kFull, best, o);
        const long long oc = __shfl_xor_sync(kFull, cost, o);
        const Fingerprint oi{__shfl_xor_sync(kFull, id.first, o), __shfl_xor_sync(kFull, id.second, o)};
        const bool less = (oi.first < id.first) | ((oi.first == id.first) & (oi.second < id.second));
        const bool same = (oi.first == id.first) & (oi.second == id.second);
        const bool take = (oc < cost) | ((oc == cost) & (less | (same & (ob < best))));
        best = take ? ob : best;
        cost = take ? oc : cost;
        id.first = take ? oi.first : id.first;
        id.second = take ? oi.second : id.second;
    }
}

// Archive selection by warp 0 (update_control's slot loop): the global best
// first, then up to 3 distinct tours of the old archive and the batch within
// 2 % of the global cost, each the least by (cost, fingerprint, canonical
// order, candidate index).
__device__ std::uint32_t ref_archive_select(const CandidateView& v, const ColonyState& st, std::uint32_t A,
                                            bool improved, std::uint32_t n, std::uint32_t lane, long long limit,
                                            std::uint32_t* excluded, std::uint32_t* chosen) {
    const std::uint32_t total = kArchive + A;
    for (std::uint32_t w = lane; w < (total + 31) / 32; w += 32) excluded[w] = 0;
    __syncwarp();
    auto is_excluded = [&](std::uint32_t c) { return (excluded[c >> 5] >> (c & 31u)) & 1u; };
    auto eligible = [&](std::uint32_t c) {
        if (c < kArchive && c >= v.ctl.archive_size) return false;
        return v.cost(c) <= limit && !is_excluded(c);
    };
    std::uint32_t count = 0;
    auto add = [&](std::uint32_t w) {
        if (lane == 0) {
            chosen[count] = w;
            excluded[w >> 5] |= 1u << (w & 31u);
        }
        ++count;
        __syncwarp();
        const Fingerprint idw = v.id(w);
        const TourRef rw = v.ref(w);
        for (std::uint32_t base = 0; base < total; base += 32) {
            const std::uint32_t c = base + lane;
            unsigned m = __ballot_sync(kFull, c < total && !is_excluded(c) && fp_equal(v.id(c), idw));
            while (m) {
                const std::uint32_t j = base + __ffs(m) - 1;
                m &= m - 1;
                if (warp_canonical_compare(v.ref(j), rw, n, lane) == 0 && lane == 0)
                    excluded[j >> 5] |= 1u << (j & 31u);
                __syncwarp();
            }
        }
        __syncwarp();
    };
    add(improved ? kArchive + st.iteration_best : 0u);
#pragma unroll 1
    for (std::uint32_t slot = 1; slot < kArchive; ++slot) {
        std::uint32_t best = 0xffffffffu;
        long long bc = LLONG_MAX;
        Fingerprint bi{~0ull, ~0ull};
#pragma unroll 1
        for (std::uint32_t c = lane; c < total; c += 32) {
            if (!eligible(c)) continue;
            const long long cc = v.cost(c);
            const Fingerprint ci = v.id(c);
            if (best == 0xffffffffu || cc < bc || (cc == bc && fp_less(ci, bi))) { best = c; bc = cc; bi = ci; }
        }
        warp_least(best, bc, bi);
        if (best == 0xffffffffu) break;
        // equal cost and fingerprint with another tour: canonical order decides
        for (std::uint32_t base = 0; base < total; base += 32) {
            const std::uint32_t c = base + lane;
            unsigned m = __ballot_sync(kFull, c < total && c != best && eligible(c) && v.cost(c) == bc &&
                                                  fp_equal(v.id(c), bi));
            while (m) {
                const std::uint32_t j = base + __ffs(m) - 1;
                m &= m - 1;
                if (warp_canonical_compare(v.ref(j), v.ref(best), n, lane) < 0) best = j;
            }
        }
        add(best);
    }
    return count;
}

// The same selection when every pair of candidates with equal fingerprints
// holds the same tour (rep[c]: the first valid candidate with c's cost and
// fingerprint): a group of identical tours acts as its first member, and the
// least by (cost, fingerprint, index) needs no tour comparison.
__device__ std::uint32_t ref_archive_select_groups(const CandidateView& v, const ColonyState& st, std::uint32_t A,
                                                   bool improved, std::uint32_t lane, long long limit,
                                                   const std::uint16_t* rep, std::uint32_t* excluded,
                                                   std::uint32_t* chosen) {
    const std::uint32_t total = kArchive + A;
    for (std::uint32_t w = lane; w < (total + 31) / 32; w += 32) excluded[w] = 0;
    __syncwarp();
    const std::uint32_t first = improved ? kArchive + st.iteration_best : 0u;
    if (lane == 0) {
        chosen[0] = first;
        excluded[rep[first] >> 5] |= 1u << (rep[first] & 31u);
    }
    __syncwarp();
    std::uint32_t count = 1;
#pragma unroll 1
    for (std::uint32_t slot = 1; slot < kArchive; ++slot) {
        std::uint32_t best = 0xffffffffu;
        long long bc = LLONG_MAX;
        Fingerprint bi{~0ull, ~0ull};
#pragma unroll 1
        for (std::uint32_t c = lane; c < total; c += 32) {
            if (rep[c] != c || ((excluded[c >> 5] >> (c & 31u)) & 1u)) continue;
            // (volatile keeps the loop's loads in the loop: moved out of it
            // and over the slots they took 33 thousand cycles instead of 8)
            const long long cc = c < kArchive ? v.ctl.archive_cost[c]
                                              : static_cast<const volatile long long*>(v.costs)[c - kArchive];
            if (cc > limit) continue;
            const Fingerprint ci = v.id(c);
            if (best == 0xffffffffu || cc < bc || (cc == bc && fp_less(ci, bi))) { best = c; bc = cc; bi = ci; }
        }
        warp_least(best, bc, bi);
        if (best == 0xffffffffu) break;
        if (lane == 0) {
            chosen[count] = best;
            excluded[best >> 5] |= 1u << (best & 31u);
        }
        ++count;
        __syncwarp();
    }
    return count;
}

struct RefShared {
    RefControl ctl;                       // the colony's controller state while the kernel runs
    float feat[12][32];
    float scores[32];
    node_t regions[8][kRegionNodes];
    long long ant_cost[kStageAnts];
    Fingerprint ant_id[kStageAnts];
    std::uint32_t ant_p0[kStageAnts];
    std::uint16_t rep[kArchive + kCtlMaxAnts];
    std::uint32_t collision;
    std::uint32_t excluded[kCtlWords];
    std::uint32_t chosen[kArchive], next_p0[kArchive];
    long long chosen_cost[kArchive];
    Fingerprint chosen_id[kArchive];
    std::uint32_t count, alternative, mask, action, largest;
    StagedProgram trees[3];
    float stack[15][32];
    float gap[2], difference, elapsed, stagnation;
    long long limit;                      // archive band of the global best
};

__device__ __forceinline__ CandidateView candidates(const ColonyView& cv, const RefShared& sh, std::uint32_t A) {
    const bool staged = A <= kStageAnts;
    return {cv, sh.ctl, staged ? sh.ant_cost : cv.ant_costs,
            staged ? sh.ant_id : reinterpret_cast<const Fingerprint*>(cv.ant_ids), staged ? sh.ant_p0 : cv.ant_p0};
}

// update_control for one colony (after reduce/select and the trail update);
// sh.ctl holds the controller state.
__device__ void ref_update(const ColonyView& cv, const InstanceView& in, const ColonyState& st,
                           const ColonyParams& P, RefShared& sh) {
    RefControl& ctl = sh.ctl;
    const std::uint32_t n = in.n, A = P.ants;
    const std::uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const bool staged = A <= kStageAnts;
    // the ants' fingerprints come from fingerprint_kernel
    if (staged)
        for (std::uint32_t a = threadIdx.x; a < A; a += blockDim.x) {
            sh.ant_cost[a] = cv.ant_costs[a];
            sh.ant_id[a] = {cv.ant_ids[2 * a], cv.ant_ids[2 * a + 1]};
            sh.ant_p0[a] = cv.ant_p0[a];
        }
    if (threadIdx.x == 0) sh.collision = 0;
    if (threadIdx.x == 64) sh.limit = band_limit(st.global_cost);
    __syncthreads();
    const bool improved = st.global_cost < ctl.tracked_global;
    const CandidateView v = candidates(cv, sh, A);
    const std::uint32_t total = kArchive + A;
    // groups of equal (cost, fingerprint); a fingerprint shared across costs,
    // or by two different tours, sends the selection to the general path
    for (std::uint32_t c = threadIdx.x; c < total; c += blockDim.x) {
        std::uint16_t r = 0xffffu;
        if (c >= kArchive || c < ctl.archive_size) {
            r = (std::uint16_t)c;
            const Fingerprint fc = v.id(c);
            const long long cc = v.cost(c);
#pragma unroll 1
            for (std::uint32_t q = 0; q < c; ++q) {
                if (q < kArchive && q >= ctl.archive_size) continue;
                if (!fp_equal(v.id(q), fc)) continue;
                if (v.cost(q) == cc) { r = (std::uint16_t)q; break; }
                sh.collision = 1;
            }
        }
        sh.rep[c] = r;
    }
    __syncthreads();
    for (std::uint32_t c = warp; c < total; c += warps) {
        const std::uint32_t r = sh.rep[c];
        if (r != 0xffffu && r != c && warp_canonical_compare(v.ref(c), v.ref(r), n, lane) != 0 && lane == 0)
            sh.collision = 1;
    }
    __syncthreads();
    if (warp == 0) {
        const std::uint32_t count =
            sh.collision ? ref_archive_select(v, st, A, improved, n, lane, sh.limit, sh.excluded, sh.chosen)
                         : ref_archive_select_groups(v, st, A, improved, lane, sh.limit, sh.rep, sh.excluded, sh.chosen);
        if (lane == 0) {
            sh.count = count;
#pragma unroll 1
            for (std::uint32_t i = 0; i < count; ++i) {
                sh.chosen_cost[i] = v.cost(sh.chosen[i]);
                sh.chosen_id[i] = v.id(sh.chosen[i]);
            }
        }
    } else if (warp == 1) {
        // feedback (update_feedback, control_ops.hpp:177-188), beside the
        // selection: the LS work fractions summed in ant order
        std::uint32_t returned = 0;
        double work = 0;
        for (std::uint32_t base = 0; base < A; base += 32) {
            const std::uint32_t a = base + lane;
            bool back = false;
            double wa = 0.0;
            if (a < A) {
                back = fp_equal(v.id(kArchive + a), ctl.active_id);
                if (P.ls_limit) wa = (double)cv.ant_counts[3 * a + 1] / (double)P.ls_limit;
            }
            returned += __popc(__ballot_sync(kFull, back));
#pragma unroll 1
            for (std::uint32_t j = 0; j < 32 && base + j < A; ++j) work += __shfl_sync(kFull, wa, j);
        }
        if (lane == 0) {
            const float rf = (float)unit_clip((double)returned / (double)A), wf = (float)unit_clip(work / (double)A);
            ctl.return_rate += (rf - ctl.return_rate) * 0.0625f;
            ctl.ls_work += (wf - ctl.ls_work) * 0.0625f;
            if (improved) ctl.stagnant_batches = 0;
            else if (ctl.stagnant_batches != ~0ull) ++ctl.stagnant_batches;
            if (ctl.epoch_batches != ~0ull) ++ctl.epoch_batches;
            const Fingerprint best = v.id(kArchive + st.iteration_best);
            if (st.epoch_cost < ctl.tracked_epoch) ctl.epoch_id = best;
            ctl.active_id = st.source_is_epoch ? ctl.epoch_id : best;
            ctl.tracked_global = st.global_cost;
            ctl.tracked_epoch = st.epoch_cost;
        }
    }
    __syncthreads();
    // chosen tours into the other half of the archive buffer: the slots side
    // by side, eight nodes per thread (tour rows are 16-byte aligned, n_pad nodes)
    const std::uint32_t next = ctl.side ^ 1u, count = sh.count, share = blockDim.x / kArchive;
    const std::uint32_t slot = threadIdx.x / share;
    if (slot < count) {
        const node_t* tour = v.ref(sh.chosen[slot]).tour;
        node_t* dst = archive_tour(cv, next, slot);
        for (std::uint32_t g = threadIdx.x - slot * share; g * 8 < n; g += share) {
            const uint4 x = reinterpret_cast<const uint4*>(tour)[g];
            reinterpret_cast<uint4*>(dst)[g] = x;
            const std::uint32_t words[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const std::uint32_t at = g * 8 + u, node = (words[u >> 1] >> (16 * (u & 1))) & 0xffffu;
                if (at >= n) continue;
                dst[cv.n_pad + node] = (node_t)at;
                if (node == 0) sh.next_p0[slot] = at;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (std::uint32_t i = 0; i < kArchive; ++i) {
            ctl.archive_cost[i] = i < count ? sh.chosen_cost[i] : 0;
            ctl.archive_id[i] = i < count ? sh.chosen_id[i] : Fingerprint{0, 0};
            ctl.archive_p0[i] = i < count ? sh.next_p0[i] : 0u;
        }
        ctl.archive_size = count;
        ctl.side = next;
    }
    __syncthreads();
}

// The decision before batch `batch` (build_control_features, score and
// apply_control_action).  Called by the whole block; st and sh.ctl shared.
__device__ void ref_decide(const ColonyView& cv, const InstanceView& in, ColonyState& st, const ColonyParams& P,
                           std::uint32_t colony, std::uint32_t colony_count, std::uint32_t batch,
                           std::uint32_t parent_p0, RefShared& sh) {
    RefControl& ctl = sh.ctl;
    const std::uint32_t n = in.n, k = in.k;
    const std::uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const std::uint32_t side = ctl.side, size = ctl.archive_size;
    if (warp >= 2 && warp < 5 && (warp == 2 || cv.controller_kind == 1))
        stage_program(cv.program[warp - 2], sh.trees[warp - 2], lane);
    if (warp == 0) {
        // alternative reference: the archive tour other than the active one
        // that differs most from it on the sampled nodes (control_cpu.cpp:46-63);
        // each lane takes samples lane and lane + 32 of every archive tour
        const TourRef parent{cv.parent, nullptr, parent_p0};
        std::uint32_t x[2], ps[2], pp[2], missing[kArchive] = {0, 0, 0, 0};
        bool have[2];
        for (std::uint32_t h = 0; h < 2; ++h) {
            have[h] = lane + 32 * h < in.sample_count;
            x[h] = have[h] ? in.samples[lane + 32 * h] : 0u;
        }
        std::uint32_t pos[kArchive][2];
        for (std::uint32_t h = 0; h < 2; ++h) {
            const std::uint32_t nb = have[h] ? cv.parent_nbr[x[h]] : 0u;
            ps[h] = nb & 0xffffu;
            pp[h] = nb >> 16;
#pragma unroll
            for (std::uint32_t i = 0; i < kArchive; ++i)
                pos[i][h] = have[h] && i < size ? archive_tour(cv, side, i)[cv.n_pad + x[h]] : 0u;
        }
#pragma unroll
        for (std::uint32_t i = 0; i < kArchive; ++i) {
            if (i >= size) continue;
            const node_t* t = archive_tour(cv, side, i);
            for (std::uint32_t h = 0; h < 2; ++h) {
                if (!have[h]) continue;
                const std::uint32_t px = pos[i][h];
                const std::uint32_t cs = t[px + 1 == n ? 0 : px + 1], cp = t[px == 0 ? n - 1 : px - 1];
                missing[i] += (cs != ps[h] && cs != pp[h]) + (cp != ps[h] && cp != pp[h]);
            }
        }
#pragma unroll 1
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (std::uint32_t i = 0; i < kArchive; ++i) missing[i] += __shfl_xor_sync(kFull, missing[i], o);
        std::uint32_t alt = kArchive, largest = 0;
#pragma unroll 1
        for (std::uint32_t i = 0; i < size; ++i) {
            const TourRef ri{archive_tour(cv, side, i), archive_tour(cv, side, i) + cv.n_pad, ctl.archive_p0[i]};
            if (fp_equal(ctl.archive_id[i], ctl.active_id) && warp_canonical_compare(ri, parent, n, lane) == 0)
                continue;
            bool better_tie = false;
            if (alt != kArchive && missing[i] == largest) {
                const long long ci = ctl.archive_cost[i], ca = ctl.archive_cost[alt];
                const Fingerprint fi = ctl.archive_id[i], fa = ctl.archive_id[alt];
                const TourRef ra{archive_tour(cv, side, alt), archive_tour(cv, side, alt) + cv.n_pad,
                                 ctl.archive_p0[alt]};
                better_tie = ci < ca || (ci == ca && (fp_less(fi, fa) ||
                                                      (fp_equal(fi, fa) && warp_canonical_compare(ri, ra, n, lane) < 0)));
            }
            if (alt == kArchive || missing[i] > largest || better_tie) { alt = i; largest = missing[i]; }
        }
        if (lane == 0) {
            sh.alternative = alt;
            sh.largest = largest;
            sh.gap[1] = alt < kArchive ? (float)unit_clip(((double)ctl.archive_cost[alt] / (double)st.global_cost - 1) /
                                                          kArchiveBand)
                                       : 0.0f;
            sh.difference = alt < kArchive ? (float)largest / (float)(2 * in.sample_count) : 0.0f;
            sh.mask = cv.action_mask & (alt < kArchive ? 0xFFFFFFFFu : 0xFFFFu);
        }
    } else if (threadIdx.x == 32) {
        // what does not depend on the alternative, in a warp of its own (FP64 divisions)
        sh.gap[0] = (float)unit_clip(((double)st.parent_cost / (double)st.global_cost - 1) / kArchiveBand);
        sh.elapsed = (float)unit_clip((double)((unsigned long long)batch * P.ants) /
                                      (double)((unsigned long long)P.total_iterations * P.ants));
        const unsigned long long stag = ctl.stagnant_batches;
        sh.stagnation = (float)(stag < 32 ? (double)stag / 32.0 : 1.0);
    }
    __syncthreads();
    const std::uint32_t alt = sh.alternative, count = n < kRegionNodes ? n : kRegionNodes;
    for (std::uint32_t w = warp; w < 8; w += warps) {
        // start region (mode, region) and its 4 features (region_features,
        // control_ops.hpp:192-214); lane 2i + s takes node i and its
        // predecessor (s = 0) or successor (s = 1); sums in node order
        const std::uint32_t mode = w >> 2, region = w & 3u;
        const bool valid = mode == 0 || alt < kArchive;
        node_t* nodes = sh.regions[w];
        const node_t* rtour = mode == 0 ? cv.parent : archive_tour(cv, side, alt < kArchive ? alt : 0);
        if (valid) {
            warp_build_region(rtour, n, in.primary, k, cv.key, batch, mode, region, nodes, lane);
        } else {
            if (lane < kRegionNodes) nodes[lane] = 0;
            __syncwarp();
        }
        float regional[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (valid) {
            const std::uint32_t i = lane >> 1, s = lane & 1u;
            const bool active = i < count;
            double half = 0.0, strength_v = 0.0;
            std::uint32_t dis = 0, disp = 0;
            std::uint32_t xn = 0, y = 0;
            if (active) {
                xn = nodes[i];
                if (mode == 0) {
                    const std::uint32_t nb = cv.parent_nbr[xn];
                    y = s ? nb & 0xffffu : nb >> 16;
                } else {
                    const std::uint32_t px = rtour[cv.n_pad + xn];
                    y = s ? rtour[px + 1 == n ? 0 : px + 1] : rtour[px == 0 ? n - 1 : px - 1];
                }
                std::uint32_t pj[kArchive];
#pragma unroll
                for (std::uint32_t j = 0; j < kArchive; ++j) pj[j] = j < size ? archive_tour(cv, side, j)[cv.n_pad + xn] : 0u;
                const int2 a = in.xy[xn], b = in.xy[y];
                half = 0.5 * (double)euc2d(a, b);
                float tau = st.default_trail;
#pragma unroll 1
                for (std::uint32_t t = 0; t < k; ++t)
                    if (in.primary[(size_t)xn * k + t] == y) { tau = cv.trails[(size_t)xn * k + t]; break; }
#pragma unroll
                for (std::uint32_t j = 0; j < kArchive; ++j) {
                    if (j >= size) continue;
                    const node_t* t = archive_tour(cv, side, j);
                    const std::uint32_t sj = t[pj[j] + 1 == n ? 0 : pj[j] + 1], qj = t[pj[j] == 0 ? n - 1 : pj[j] - 1];
                    dis += sj != y && qj != y;
                }
                const double lo = (double)st.tau_min, hi = (double)st.tau_max;
                strength_v = lo == hi ? 1.0 : unit_clip(((double)tau - lo) / (hi - lo));
                disp = !has_node(nodes, count, y);
            }
            const double other = __shfl_down_sync(kFull, half, 1);
            double ex = 0.0;
            if (active && s == 0) {
                const double scale = in.local_scale[xn] < in.scale_epsilon ? in.scale_epsilon : in.local_scale[xn];
                ex = unit_clip(((half + other) / scale - 1) / 3);
            }
            double excess = 0, strength = 0;
#pragma unroll 1
            for (std::uint32_t q = 0; q < count; ++q) {
                excess += __shfl_sync(kFull, ex, 2 * q);
                strength += __shfl_sync(kFull, strength_v, 2 * q);
                strength += __shfl_sync(kFull, strength_v, 2 * q + 1);
            }
#pragma unroll 1
            for (int o = 16; o; o >>= 1) {
                dis += __shfl_xor_sync(kFull, dis, o);
                disp += __shfl_xor_sync(kFull, disp, o);
            }
            // a ratio of small integers rounds to the same float directly as
            // through double; division by 16 or 32 is an exact scaling
            if (count == kRegionNodes) {
                regional[0] = (float)(excess * (1.0 / kRegionNodes));
                regional[2] = (float)(strength * (0.5 / kRegionNodes));
            } else {
                regional[0] = (float)(excess / count);
                regional[2] = (float)(strength / (double)(2 * count));
            }
            regional[1] = __fdiv_rn((float)dis, (float)(2 * count * size));
            regional[3] = __fdiv_rn((float)disp, (float)(2 * count));
        }
        if (lane < 4) {
            const std::uint32_t level = lane, a = mode * 16 + region * 4 + level;
            sh.feat[0][a] = sh.elapsed;
            sh.feat[1][a] = sh.stagnation;
            sh.feat[2][a] = ctl.return_rate;
            sh.feat[3][a] = ctl.ls_work;
            sh.feat[4][a] = (float)mode;
            sh.feat[5][a] = (float)(level + 1) * 0.25f;
            sh.feat[6][a] = sh.gap[mode];
            sh.feat[7][a] = mode ? sh.difference : 0.0f;
            for (int f = 0; f < 4; ++f) sh.feat[8 + f][a] = regional[f];
        }
    }
    __syncthreads();
    if (warp == 0) {
        const std::uint32_t mask = sh.mask;
        std::uint32_t a;
        if (cv.controller_kind == 1) {
            sh.scores[lane] = 0.0f;
            __syncwarp();
            a = choose_conditional(sh.trees, sh.stack, [&](int i, std::uint32_t act) { return sh.feat[i][act]; }, mask,
                                   lane, sh.scores);
        } else {
            const float value = eval_program(sh.trees[0], sh.stack, lane, [&](int i) { return sh.feat[i][lane]; });
            sh.scores[lane] = value;
            a = choose_action(value, (mask >> lane) & 1u, lane);
        }
        __syncwarp();
        const std::uint32_t chosen = a < 32 ? a : 0;
        const DecisionCapture& cap = P.capture;
        for (std::uint32_t i = 0; i < cap.count; ++i) {
            if (cap.points[i] != batch + 1) continue;
            const size_t slot = (size_t)i * colony_count + colony;
            for (std::uint32_t f = 0; f < 12; ++f) cap.features[(slot * 12 + f) * 32 + lane] = sh.feat[f][lane];
            cap.scores[slot * 32 + lane] = sh.scores[lane];
            if (lane == 0) {
                cap.masks[slot] = mask;
                cap.actions[slot] = (std::int32_t)chosen;
            }
        }
        if (lane == 0) {
            sh.action = chosen;
            st.action = (std::int32_t)chosen;
            st.mne_target = 2u << (chosen & 3u);
            st.region = 5;
            ctl.alternative = alt;
            ctl.legal_mask = mask;
            ctl.start_count = count;
            if (chosen >= 16) {
                // restart from the alternative reference (control_state.cuh:302-336)
                st.epoch_cost = st.parent_cost = ctl.archive_cost[alt];
                trail_limits(st.epoch_cost, P.retention, P.p_root, k, st.tau_min, st.tau_max);
                st.default_trail = st.tau_max;
                st.source_is_epoch = 0;
                st.iteration_best = 0;
                ctl.tracked_epoch = st.epoch_cost;
                ctl.active_id = ctl.epoch_id = ctl.archive_id[alt];
                ctl.return_rate = ctl.ls_work = 0.0f;
                ctl.epoch_batches = 0;
                if (ctl.restarts != ~0ull) ++ctl.restarts;
            }
        }
        if (lane < kRegionNodes)
            ctl.start_nodes[lane] = sh.regions[(chosen >> 4) * 4 + ((chosen >> 2) & 3u)][lane];
    }
    __syncthreads();
    if (sh.action >= 16) {
        const node_t* tour = archive_tour(cv, side, alt);
        for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) cv.parent[i] = cv.epoch[i] = tour[i];
        __syncthreads();
        for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            cv.parent_nbr[cv.parent[i]] = (std::uint32_t)cv.parent[i + 1 == n ? 0 : i + 1] |
                                          ((std::uint32_t)cv.parent[i == 0 ? n - 1 : i - 1] << 16);
            if (cv.parent_pos) cv.parent_pos[cv.parent[i]] = (node_t)i;
        }
        const float tmax = st.tau_max;
        for (std::uint32_t i = threadIdx.x; i < n * k; i += blockDim.x) {
            cv.trails[i] = tmax;
            cv.products[i] = tmax * cv.eta[i];
        }
    }
    __syncthreads();
}

// Departure-only prior products (departure_rows) of the colonies whose mode
// is 1, one block per colony: run after the prior's heuristic is applied.
__global__ void __launch_bounds__(256) prior_rows_kernel(const InstanceView* instances, const ColonyView* colonies,
                                                         const std::uint32_t* modes) {
    const std::uint32_t c = blockIdx.x;
    if (!modes[c]) return;
    const ColonyView cv = colonies[c];
    const InstanceView in = instances[cv.instance];
    departure_rows(in, cv, threadIdx.x, blockDim.x, in.n);
}

// Fingerprints (and node-0 positions) of every ant's tour of a batch, one
// warp per ant over the colonies of `list` (all colonies when null)
// (fingerprint_ants, control_state.cuh:45-64); `zero` forces every
// fingerprint to 0 (the collision diagnostic).
__global__ void __launch_bounds__(256) fingerprint_kernel(const ColonyView* colonies, const std::uint32_t* list,
                                                          std::uint32_t ants, std::uint32_t colony_count,
                                                          std::uint32_t zero) {
    const std::uint32_t job = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (job >= ants * colony_count) return;
    const std::uint32_t slot = job / ants, ant = job % ants;
    const std::uint32_t colony = list ? list[slot] : slot;
    const ColonyView& cv = colonies[colony];
    std::uint32_t p0;
    const Fingerprint f = warp_fingerprint(cv.ant_tours + (size_t)ant * cv.n_pad, cv.n, lane, p0);
    if (lane == 0) {
        cv.ant_ids[2 * ant] = zero ? 0ull : f.first;
        cv.ant_ids[2 * ant + 1] = zero ? 0ull : f.second;
        cv.ant_p0[ant] = p0;
    }
}

__global__ void colony_init_kernel(const InstanceView* instances, const ColonyView* colonies, ColonyState* states,
                                   ColonyParams P, std::uint32_t colony_count) {
    const std::uint32_t c = blockIdx.x;
    const ColonyView cv = colonies[c];
    const InstanceView in = instances[cv.instance];
    const std::uint32_t n = in.n, k = in.k;
    __shared__ float s_tmax;
    __shared__ ColonyState s_st;
    if (threadIdx.x == 0) {
        ColonyState st{};
        st.epoch_cost = st.global_cost = st.parent_cost = st.iteration_best_cost = in.initial_cost;
        trail_limits(in.initial_cost, P.retention, P.p_root, k, st.tau_min, st.tau_max);
        st.default_trail = st.tau_max;
        *cv.walk = 0;
        st.mne_target = P.mne_target;
        st.action = -1;
        st.region = 4;
        states[c] = st;
        s_st = st;
        s_tmax = st.tau_max;
    }
    for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const node_t v = in.initial[i];
        cv.parent[i] = cv.epoch[i] = cv.global[i] = v;
        if (cv.parent_pos) cv.parent_pos[v] = (node_t)i;
        cv.parent_nbr[v] = (std::uint32_t)in.initial[i + 1 == n ? 0 : i + 1] |
                           ((std::uint32_t)in.initial[i == 0 ? n - 1 : i - 1] << 16);
    }
    __syncthreads();
    const float tmax = s_tmax;
    for (std::uint32_t i = threadIdx.x; i < n * k; i += blockDim.x) {
        cv.trails[i] = tmax;
        cv.eta[i] = in.eta[i];
        cv.products[i] = tmax * in.eta[i];
    }
    if (P.ref_control && cv.control) {
        // the archive holds the initial tour (initialize_control,
        // control_state.cuh:21-43); then the decision before batch 0
        __shared__ RefShared s_ref;
        node_t* a0 = archive_tour(cv, 0, 0);
        for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            a0[i] = in.initial[i];
            a0[cv.n_pad + in.initial[i]] = (node_t)i;
        }
        __shared__ std::uint32_t s_p0;
        if (threadIdx.x < 32) {
            std::uint32_t p0;
            Fingerprint f = warp_fingerprint(in.initial, n, threadIdx.x, p0);
            if (P.zero_fingerprints) f = Fingerprint{0, 0};
            if (threadIdx.x == 0) {
                s_p0 = p0;
                RefControl ctl{};
                ctl.archive_size = 1;
                ctl.archive_cost[0] = in.initial_cost;
                ctl.archive_id[0] = f;
                ctl.archive_p0[0] = p0;
                ctl.active_id = ctl.epoch_id = f;
                ctl.tracked_global = ctl.tracked_epoch = in.initial_cost;
                ctl.alternative = kArchive;
                s_ref.ctl = ctl;
            }
        }
        __syncthreads();
        ref_decide(cv, in, s_st, P, c, colony_count, 0, s_p0, s_ref);
        if (threadIdx.x == 0) {
            states[c] = s_st;
            *cv.control = s_ref.ctl;
        }
    }
}

__device__ __forceinline__ void write_trace(TraceRow& row, const ColonyState& st, std::uint32_t mne,
                                            std::int32_t action, unsigned long long steps, unsigned long long evals) {
    row.iteration_best_cost = st.iteration_best_cost;
    row.global_cost = st.global_cost;
    row.parent_cost = st.parent_cost;
    row.iteration_best = st.iteration_best;
    row.source_is_epoch = st.source_is_epoch;
    row.tau_min = st.tau_min;
    row.tau_max = st.tau_max;
    row.mne_target = mne;
    row.action = action;
    row.construction_steps = steps;
    row.ls_evaluations = evals;
}

// Fused reduce_and_select + update_pheromone for one colony, then (GP-controlled
// evaluations) the controller decision for the next iteration.  Block b
// updates colony list[b] (colony b when `list` is null); `colony_count` is
// the evaluation's colony count.
//
// CONTROL 0: plain FACO, 1: the engine's own controllers (feature spec 3), 2:
// the reference's (spec 2).  A kernel each: the spec-2 decision takes 128
// registers, with which the block of a plain colony, 256 threads then, waited
// for half an SM to fall idle.  An update is the serial link between a
// colony's iterations and bound by latency: one read of the best tour writes
// the parent, its neighbours and the incumbents, the two FP64 chains (trail
// limits; parent source and deposit) run in two warps, and 512 threads hold
// two groups of trail entries each.  One GB300, in thousand cycles of one
// colony's update, before -> after: N=1000-2000 (trails apart) 15.6 -> 12.2,
// spec 3 at N=500 52 -> 37, spec 2 at N=500 146 -> 88; whole runs: 128 x 32
// ants at N=1000-2000 146.2 -> 141.8 ms, the uneven batch 84.2 -> 82.2.
__host__ __device__ constexpr std::uint32_t update_threads(int control) { return control == 2 ? 256u : 512u; }

template <int CONTROL>
__global__ void __launch_bounds__(update_threads(CONTROL), CONTROL == 2 ? 2 : 3)
colony_update_kernel(const InstanceView* instances, const ColonyView* colonies, ColonyState* states, ColonyParams P,
                     TraceRow* trace, const std::uint32_t* list, std::uint32_t colony_count, std::uint32_t trace_cap) {
    constexpr std::uint32_t kWarps = update_threads(CONTROL) / 32;
    const std::uint32_t c = list ? list[blockIdx.x] : blockIdx.x;
    const ColonyView cv = colonies[c];
    const InstanceView in = instances[cv.instance];
    const std::uint32_t n = in.n, k = in.k, A = P.ants;
    const std::uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ unsigned long long s_red[6][kWarps];
    __shared__ ColonyState s_st;
    __shared__ std::uint32_t s_from_epoch, s_restart;
    __shared__ float s_tmin, s_tmax, s_inc, s_feat[7];
    __shared__ long long s_sum_final, s_sum_cons;
    __shared__ unsigned long long s_steps, s_evals;
    __shared__ std::uint32_t s_used_mne, s_parent_p0;

    start_next_kernel();
    wait_previous_kernel();
    for (std::uint32_t w = threadIdx.x; w < sizeof(ColonyState) / 4; w += blockDim.x)
        reinterpret_cast<std::uint32_t*>(&s_st)[w] = reinterpret_cast<const std::uint32_t*>(states + c)[w];
    // iteration best: first strict minimum over ants (costs are >= 0); work counters
    unsigned long long best = ~0ull, steps = 0, evals = 0, moved = 0, sum_final = 0, sum_cons = 0;
    for (std::uint32_t a = threadIdx.x; a < A; a += blockDim.x) {
        const unsigned long long key = ((unsigned long long)cv.ant_costs[a] << 16) | a;
        best = key < best ? key : best;
        steps += cv.ant_counts[3 * a];
        evals += cv.ant_counts[3 * a + 1];
        moved += cv.ant_counts[3 * a + 2];
        sum_final += (unsigned long long)cv.ant_costs[a];
        sum_cons += (unsigned long long)cv.ant_ccosts[a];
    }
    const std::uint32_t used = A < 32 * kWarps ? (A + 31) / 32 : kWarps;   // warps that hold ants
    if (warp < used) {
        for (int o = 16; o; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(kFull, best, o);
            best = other < best ? other : best;
            steps += __shfl_xor_sync(kFull, steps, o);
            evals += __shfl_xor_sync(kFull, evals, o);
            moved += __shfl_xor_sync(kFull, moved, o);
            sum_final += __shfl_xor_sync(kFull, sum_final, o);
            sum_cons += __shfl_xor_sync(kFull, sum_cons, o);
        }
        if (lane == 0) {
            s_red[0][warp] = best; s_red[1][warp] = steps; s_red[2][warp] = evals;
            s_red[3][warp] = moved; s_red[4][warp] = sum_final; s_red[5][warp] = sum_cons;
        }
    }
    __syncthreads();
    best = s_red[0][0];
    for (std::uint32_t w = 1; w < used; ++w) best = s_red[0][w] < best ? s_red[0][w] : best;
    const std::uint32_t ib = (std::uint32_t)(best & 0xffffu);
    const long long cost = (long long)(best >> 16);
    const bool ie = cost < s_st.epoch_cost, ig = cost < s_st.global_cost;
    const long long epoch_cost = ie ? cost : s_st.epoch_cost;
    if (threadIdx.x == 0) {
        float tmin, tmax;
        trail_limits(epoch_cost, P.retention, P.p_root, k, tmin, tmax);
        s_tmin = tmin;
        s_tmax = tmax;
    }
    if (threadIdx.x == 32) {
        const bool from_epoch = source_uniform(cv.key, s_st.iteration) < P.epoch_source_probability;
        s_from_epoch = from_epoch;
        s_inc = (float)(1.0 / (double)(from_epoch ? epoch_cost : cost));
    }
    const std::uint32_t vectors = (n + 7) / 8;   // 8 nodes; rows are padded to whole ones
    const node_t* best_tour = cv.ant_tours + (size_t)ib * cv.n_pad;
    for (std::uint32_t g = threadIdx.x; (ie || ig) && g < vectors; g += blockDim.x) {
        const uint4 x = reinterpret_cast<const uint4*>(best_tour)[g];
        if (ie) reinterpret_cast<uint4*>(cv.epoch)[g] = x;
        if (ig) reinterpret_cast<uint4*>(cv.global)[g] = x;
    }
    __syncthreads();
    // the parent (the epoch's best, which may be this iteration's) and its packed neighbours
    const bool fe = s_from_epoch;
    const node_t* source = fe && !ie ? cv.epoch : best_tour;
    for (std::uint32_t g = threadIdx.x; g < vectors; g += blockDim.x) {
        const uint4 x = reinterpret_cast<const uint4*>(source)[g];
        std::uint32_t before = source[g == 0 ? n - 1 : 8 * g - 1];
        const std::uint32_t after = source[8 * g + 8 < n ? 8 * g + 8 : 0];
        reinterpret_cast<uint4*>(cv.parent)[g] = x;
        const std::uint32_t words[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (std::uint32_t u = 0; u < 8; ++u) {
            const std::uint32_t i = 8 * g + u, node = (words[u >> 1] >> (16 * (u & 1))) & 0xffffu;
            if (i >= n) continue;
            const std::uint32_t next = i + 1 == n || u == 7 ? after : (words[(u + 1) >> 1 & 3] >> (16 * ((u + 1) & 1))) & 0xffffu;
            cv.parent_nbr[node] = next | before << 16;
            if (cv.parent_pos) cv.parent_pos[node] = (node_t)i;
            before = node;
            if (CONTROL == 2 && node == 0) s_parent_p0 = i;
        }
    }
    if (threadIdx.x == 0) {
        for (std::uint32_t w = 0; w < used; ++w) {
            if (w == 0) steps = evals = moved = sum_final = sum_cons = 0;
            steps += s_red[1][w]; evals += s_red[2][w]; moved += s_red[3][w];
            sum_final += s_red[4][w]; sum_cons += s_red[5][w];
        }
        ColonyState& st = s_st;
        st.epoch_cost = epoch_cost;
        if (ig) { st.global_cost = cost; st.last_improvement = st.iteration + 1; }
        st.tau_min = s_tmin;
        st.tau_max = s_tmax;
        st.parent_cost = fe ? epoch_cost : cost;
        st.iteration_best = ib;
        st.iteration_best_cost = cost;
        st.source_is_epoch = fe;
        st.construction_steps += steps;
        st.ls_evaluations += evals;
        st.reversed_elements += moved;
        *cv.walk = (std::uint32_t)(steps / A);
        st.default_trail = fmaxf(st.tau_min, st.default_trail * P.retention_f);
        s_sum_final = (long long)sum_final; s_sum_cons = (long long)sum_cons;
        s_steps = steps; s_evals = evals; s_used_mne = st.mne_target;
        s_restart = 0;
    }
    __syncthreads();
    if (P.trail_blocks <= 1) {
        trail_update(n, k, in.primary, cv.parent_nbr, P.retention_f, s_tmin, s_tmax, s_inc, cv.eta, cv.trails,
                     cv.products, threadIdx.x, blockDim.x);
        if (P.prior_rows && P.prior_rows[c]) {
            __syncthreads();
            departure_rows(in, cv, threadIdx.x, blockDim.x, n);
        }
    }
    std::int32_t action = -1;
    if constexpr (CONTROL == 2) {
        // the 12-feature controller: the trace row holds the action this
        // batch ran with; archive and feedback; the next batch's decision
        __shared__ RefShared s_ref;
        if (threadIdx.x == 0) {
            s_ref.ctl = *cv.control;
            if (trace && s_st.iteration < trace_cap)
                write_trace(trace[(size_t)s_st.iteration * colony_count + c], s_st, s_used_mne, s_st.action, s_steps,
                            s_evals);
        }
        __syncthreads();
        ref_update(cv, in, s_st, P, s_ref);
        if (s_st.iteration + 1 < P.total_iterations)
            ref_decide(cv, in, s_st, P, c, colony_count, s_st.iteration + 1, s_parent_p0, s_ref);
        if (threadIdx.x == 0) *cv.control = s_ref.ctl;
    } else if (CONTROL == 1 && cv.program) {
        // mean normalised entropy of the trail rows (exact integer sum)
        __shared__ StagedProgram s_trees[3];
        __shared__ float s_stack[15][32], s_action[3][32];
        if (warp == 5) {
            // the descriptors of action `lane`: MNE level, start region, restart flag
            s_action[0][lane] = (float)(lane & 3u) / 3.0f;
            s_action[1][lane] = (float)((lane >> 2) & 3u) / 3.0f;
            s_action[2][lane] = lane >= 16u ? 1.0f : 0.0f;
        }
        if (warp >= 2 && warp < 5 && (warp == 2 || cv.controller_kind == 1))
            stage_program(cv.program[warp - 2], s_trees[warp - 2], lane);
        __syncthreads();
        unsigned long long q = 0;
        for (std::uint32_t row = threadIdx.x; row < n; row += blockDim.x)
            q += row_entropy_q(cv.trails + (size_t)row * k, k, P.log2k);
        for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(kFull, q, o);
        if (lane == 0) s_red[0][warp] = q;
        __syncthreads();
        if (lane == 0 && warp < 7) {
            // one feature per warp: their FP64 and FP32 divisions side by side
            const ColonyState& st = s_st;
            const std::uint32_t t1 = st.iteration + 1, stag = t1 - st.last_improvement, age = t1 - st.last_restart;
            const long long b = st.iteration_best_cost;
            float f = 0.0f;
            if (warp == 0) f = (float)t1 / (float)P.total_iterations;
            else if (warp == 1) f = (float)stag / (float)(stag + 16);
            else if (warp == 2) f = clamp01((double)(s_sum_final - (long long)A * b) / ((double)A * (double)b));
            else if (warp == 3) {
                q = 0;
                for (std::uint32_t w = 0; w < kWarps; ++w) q += s_red[0][w];
                f = clamp01((double)q * (1.0 / 1048576.0) / (double)n);
            } else if (warp == 4) f = (float)st.restarts / (float)(st.restarts + 1);
            else if (warp == 5) f = clamp01((double)(s_sum_cons - s_sum_final) / (double)s_sum_cons * 10.0);
            else f = (float)age / (float)(age + 16);
            s_feat[warp] = f;
        }
        __syncthreads();
        if (warp == 0) {
            // features of action a: the 7 colony features, then its descriptors
            auto feature_of = [&](int i, std::uint32_t a) {
                return i < 7 ? s_feat[i] : i < 10 ? s_action[i - 7][a] : 0.0f;
            };
            std::uint32_t a;
            if (cv.controller_kind == 1) {
                a = choose_conditional(s_trees, s_stack, feature_of, cv.action_mask, lane, nullptr);
            } else {
                const float value = eval_program(s_trees[0], s_stack, lane, [&](int i) { return feature_of(i, lane); });
                a = choose_action(value, (cv.action_mask >> lane) & 1u, lane);
            }
            if (lane == 0) {
                const std::uint32_t chosen = a < 32 ? a : 0;
                s_st.action = (std::int32_t)chosen;
                s_st.mne_target = 2u << (chosen & 3u);
                s_st.region = (chosen >> 2) & 3u;
                if (chosen >= 16) {
                    s_restart = 1;
                    ++s_st.restarts;
                    s_st.last_restart = s_st.iteration + 1;
                    s_st.epoch_cost = s_st.global_cost;
                    s_st.parent_cost = s_st.global_cost;
                    trail_limits(s_st.epoch_cost, P.retention, P.p_root, k, s_st.tau_min, s_st.tau_max);
                    s_st.default_trail = s_st.tau_max;
                }
            }
        }
        __syncthreads();
        action = s_st.action;
        if (s_restart) {
            // restart: parent and epoch <- global best, trails <- tau_max
            for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) cv.parent[i] = cv.epoch[i] = cv.global[i];
            __syncthreads();
            for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
                cv.parent_nbr[cv.parent[i]] = (std::uint32_t)cv.parent[i + 1 == n ? 0 : i + 1] |
                                              ((std::uint32_t)cv.parent[i == 0 ? n - 1 : i - 1] << 16);
                if (cv.parent_pos) cv.parent_pos[cv.parent[i]] = (node_t)i;
            }
            const float tmax = s_st.tau_max;
            for (std::uint32_t i = threadIdx.x; i < n * k; i += blockDim.x) {
                cv.trails[i] = tmax;
                cv.products[i] = tmax * cv.eta[i];
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        ColonyState st = s_st;
        if (trace && st.iteration < trace_cap && CONTROL != 2)
            write_trace(trace[(size_t)st.iteration * colony_count + c], st, s_used_mne, action, s_steps, s_evals);
        ++st.iteration;
        states[c] = st;
    }
}

cudaError_t launch_colony_update(const InstanceView* instances, const ColonyView* colonies, ColonyState* states,
                                 const ColonyParams& P, TraceRow* trace, const std::uint32_t* list,
                                 std::uint32_t blocks, std::uint32_t colony_count, std::uint32_t trace_cap,
                                 cudaStream_t stream, bool overlapped) {
    const auto launch = [&](auto control) {
        constexpr int kControl = decltype(control)::value;
        return launch_overlapped(overlapped, colony_update_kernel<kControl>, blocks, update_threads(kControl), 0, stream,
                                 instances, colonies, states, P, trace, list, colony_count, trace_cap);
    };
    if (P.ref_control) return launch(std::integral_constant<int, 2>{});
    return P.controlled ? launch(std::integral_constant<int, 1>{}) : launch(std::integral_constant<int, 0>{});
}

// The trail update of large candidate matrices, after the colony update has
// chosen the parent and the trail limits (it leaves the trails alone when
// P.trail_blocks > 1): block (x, y) updates rows [n x / X, n (x+1) / X) of
// colony y of the launch (of `list`, or all when null) -- evaporation,
// deposit on the parent's edges, bounds and products exactly as the colony
// update would -- then, for a colony whose prior re-ranks departures, those
// rows' products.  One block per colony streams a large matrix at a small
// fraction of the memory bandwidth; X blocks per colony fill the GPU.
__global__ void __launch_bounds__(256) colony_trails_kernel(const InstanceView* instances,
                                                            const ColonyView* colonies, const ColonyState* states,
                                                            ColonyParams P, const std::uint32_t* list) {
    const std::uint32_t c = list ? list[blockIdx.y] : blockIdx.y;
    const ColonyView cv = colonies[c];
    const InstanceView in = instances[cv.instance];
    const std::uint32_t n = in.n, k = in.k;
    const std::uint32_t r0 = (std::uint32_t)((unsigned long long)n * blockIdx.x / gridDim.x);
    const std::uint32_t r1 = (std::uint32_t)((unsigned long long)n * (blockIdx.x + 1) / gridDim.x);
    if (r0 >= r1) return;
    const ColonyState& st = states[c];
    const float tmin = st.tau_min, tmax = st.tau_max, inc = (float)(1.0 / (double)st.parent_cost);
    const std::size_t off = (std::size_t)r0 * k;
    trail_update(r1 - r0, k, in.primary + off, cv.parent_nbr + r0, P.retention_f, tmin, tmax, inc, cv.eta + off,
                 cv.trails + off, cv.products + off, threadIdx.x, blockDim.x);
    if (P.prior_rows && P.prior_rows[c]) {
        __syncthreads();
        departure_rows(in, cv, r0 + threadIdx.x, blockDim.x, r1);
    }
}

__global__ void pheromone_step_kernel(std::uint32_t n, std::uint32_t k, const node_t* primary,
                                      const std::uint32_t* parent_nbr, float ret, float tmin, float tmax, float inc,
                                      const float* eta, float* trails, float* products) {
    trail_update(n, k, primary, parent_nbr, ret, tmin, tmax, inc, eta, trails, products,
                 blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ---------------------------------------------------------------------------
// GP scoring: one warp per colony, lane = action (cuda/gp_score.cuh:64-102).
// A warp takes its colony's 12 x 32 features once, checks that they are in
// [0, 1] (kErrFeature otherwise: the host then hands out no scores) and keeps
// them in shared memory for the interpreter.  The check on the device costs
// nothing beside the reads (4,096 colonies: 6.3 MB); as a host loop it was 17
// of the call's 18.8 ms.
// ---------------------------------------------------------------------------
constexpr std::uint32_t kScoreWarps = 4;

__device__ __forceinline__ void stage_features(const float* features, std::uint32_t colony, std::uint32_t colonies,
                                               std::uint32_t lane, float (&staged)[12][32], unsigned* error) {
    bool inside = true;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        const float v = features[((size_t)i * colonies + colony) * 32 + lane];
        inside = inside && v >= 0.0f && v <= 1.0f;
        staged[i][lane] = v;
    }
    if (!inside) atomicOr(error, kErrFeature);
    __syncwarp();
}

// Controllers (3 tree slots each, kinds[i]): joint ones score all 32 lanes,
// conditional ones write their role scores to slots 0-9 of the colony's row.
__global__ void __launch_bounds__(kScoreWarps * 32)
score_controllers_kernel(const Program* trees, const std::uint32_t* kinds, std::uint32_t replicas,
                         const float* features, const std::uint32_t* masks, float* scores, std::int32_t* actions,
                         std::uint32_t colonies, unsigned* error) {
    __shared__ float staged[kScoreWarps][12][32], stacks[kScoreWarps][15][32];
    __shared__ StagedProgram trees_of[kScoreWarps][3];
    const std::uint32_t colony = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (colony >= colonies) return;
    float(&mine)[12][32] = staged[threadIdx.x >> 5];
    stage_features(features, colony, colonies, lane, mine, error);
    const std::uint32_t controller = colony / replicas;
    const Program* slots = trees + 3 * (size_t)controller;
    StagedProgram* own = trees_of[threadIdx.x >> 5];
    float(*stack)[32] = stacks[threadIdx.x >> 5];
    for (int t = 0; t < (kinds[controller] == 1 ? 3 : 1); ++t) stage_program(slots[t], own[t], lane);
    __syncwarp();
    std::uint32_t chosen;
    if (kinds[controller] == 1) {
        chosen = choose_conditional(own, stack, [&](int i, std::uint32_t a) { return mine[i][a]; }, masks[colony], lane,
                                    scores + (size_t)colony * 32);
    } else {
        const float value = eval_program(own[0], stack, lane, [&](int i) { return mine[i][lane]; });
        scores[(size_t)colony * 32 + lane] = value;
        chosen = choose_action(value, (masks[colony] >> lane) & 1u, lane);
    }
    if (lane == 0) actions[colony] = (std::int32_t)chosen;
}

__global__ void __launch_bounds__(kScoreWarps * 32)
score_kernel(const Program* programs, std::uint32_t replicas, const float* features, const std::uint32_t* masks,
             float* scores, std::int32_t* actions, std::uint32_t colonies, unsigned* error) {
    __shared__ float staged[kScoreWarps][12][32], stacks[kScoreWarps][15][32];
    __shared__ StagedProgram program_of[kScoreWarps];
    const std::uint32_t colony = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (colony >= colonies) return;
    float(&mine)[12][32] = staged[threadIdx.x >> 5];
    stage_features(features, colony, colonies, lane, mine, error);
    StagedProgram& own = program_of[threadIdx.x >> 5];
    stage_program(programs[colony / replicas], own, lane);
    __syncwarp();
    const float value = eval_program(own, stacks[threadIdx.x >> 5], lane, [&](int i) { return mine[i][lane]; });
    scores[(size_t)colony * 32 + lane] = value;
    const std::uint32_t chosen = choose_action(value, (masks[colony] >> lane) & 1u, lane);
    if (lane == 0) actions[colony] = (std::int32_t)chosen;
}

}  // namespace faco

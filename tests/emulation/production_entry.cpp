
// One engine-mode ant on the host, in the variants the engine launches: an
// engine mode or'ed with its local search (kTwoOptOnly, kOrOptOnly), the
// per-colony choice between single and batched steps (walk against
// batch_from), and in the global-memory workspace the parent's inverse copied
// from the colony, its row ending where the next colony's starts.  Otherwise
// as emulator_entry.cpp; *batches counts the batches tried.
extern "C" int emu_production_ant(std::uint32_t mode, std::uint32_t batch_from, std::uint32_t walk, std::uint32_t n,
                                  std::uint32_t k, std::uint32_t b, std::uint32_t w, const int* xy,
                                  const std::uint16_t* primary, const std::uint16_t* backup, const std::uint16_t* ls,
                                  const int* ls_dist, const std::uint16_t* parent, const std::uint32_t* parent_nbr,
                                  const float* products, unsigned long long key, std::uint32_t batch,
                                  std::uint32_t ant, std::uint32_t target, long long parent_cost,
                                  std::uint32_t ls_mode, std::uint16_t* out_tour, long long* out_costs,
                                  unsigned* out_counts, unsigned* error, unsigned* batches) {
    using namespace faco;
    const std::uint32_t n_pad = pad8(n);
    struct alignas(16) Vector { node_t v[8]; };   // device rows start on 16 bytes
    const auto rows = [&](std::size_t count, node_t fill) {
        std::vector<Vector> r(count * n_pad / 8);
        std::fill(&r.data()->v[0], &r.data()->v[0] + count * n_pad, fill);
        return r;
    };
    InstanceView in{};
    in.n = n; in.k = k; in.b = b; in.w = w;
    in.xy = reinterpret_cast<const int2*>(xy);
    in.primary = primary; in.backup = backup; in.ls = ls; in.ls_dist = ls_dist;
    ColonyView cv{};
    cv.n = n; cv.n_pad = n_pad; cv.key = key;
    cv.products = const_cast<float*>(products);
    cv.parent_nbr = const_cast<std::uint32_t*>(parent_nbr);
    cv.walk = &walk;
    // padding holds garbage, as after another evaluation on the device
    auto own = rows(2, 0xABAB), tours = rows(ant + 1, 0xABAB), ws = rows(2 * (ant + 1), 0xABAB);
    cv.parent = own.data()->v;
    for (std::uint32_t i = 0; i < n; ++i) {
        cv.parent[i] = parent[i];
        cv.parent[n_pad + parent[i]] = static_cast<node_t>(i);
    }
    if (global_mode(static_cast<int>(mode))) cv.parent_pos = cv.parent + n_pad;
    cv.ant_tours = tours.data()->v;
    std::vector<long long> costs(ant + 1), ccosts(ant + 1);
    std::vector<unsigned> counts(3 * (ant + 1));
    cv.ant_costs = costs.data(); cv.ant_ccosts = ccosts.data(); cv.ant_counts = counts.data();
    ColonyState st{};
    st.parent_cost = parent_cost; st.mne_target = target; st.iteration = batch; st.region = 4;
    uint2 job{0, ant};
    AntLaunch L{};
    L.instances = &in; L.colonies = &cv; L.states = &st; L.work = &job; L.ants = ant + 1; L.warps = 1;
    L.n_max = n; L.ls_limit = 100000; L.ls_mode = ls_mode; L.batch_from = batch_from; L.error = error;
    L.workspace = ws.data()->v;
    L.ant_tours_base = cv.ant_tours;
    // shared memory starts with garbage, as on the device
    std::vector<Vector> smem(block_smem_bytes(n, 1) / 16 + 1);
    std::memset(smem.data(), 0xAB, smem.size() * sizeof(Vector));
    unsigned char* sm = reinterpret_cast<unsigned char*>(smem.data());
    emu_batches = 0;
    void (*run)(const AntLaunch, unsigned char*) = nullptr;
    switch (mode) {
#define VARIANT(m)                                                                  \
    case m | kTwoOptOnly: run = ant_kernel_emu<m | kTwoOptOnly>; break;             \
    case m | kOrOptOnly: run = ant_kernel_emu<m | kOrOptOnly>; break;
        VARIANT(kModeEngine)
        VARIANT(kModeEngineGlobal)
        VARIANT(kModeEngineFollow)
        VARIANT(kModeEngineGlobalFollow)
        VARIANT(kModeEngineFollowDense)
#undef VARIANT
        default: return -1;
    }
    Warp warp;
    std::vector<std::thread> th;
    for (unsigned l = 0; l < 32; ++l)
        th.emplace_back([&, l] {
            tl_warp = &warp;
            tl_lane = l;
            run(L, sm);
        });
    for (auto& t : th) t.join();
    std::memcpy(out_tour, cv.ant_tours + static_cast<std::size_t>(ant) * n_pad, n * sizeof(node_t));
    out_costs[0] = ccosts[ant];
    out_costs[1] = costs[ant];
    for (int i = 0; i < 3; ++i) out_counts[i] = counts[3 * ant + i];
    *batches = emu_batches;
    return 0;
}

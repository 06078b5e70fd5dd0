// Checks of the engine's host code on the fake runtime (fake_cudart.h): ./runtime_checks NAME runs one.
#include "fake_cudart.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>

#include <algorithm>
#include <cmath>

#include "amr_kernels.h"
#include "jp.h"
#include "kernels.h"
#include "solver.h"

using jp::amr::AdaptCounts;

static int failures = 0;
#define CHECK(x)                                                            \
    do {                                                                    \
        if (!(x)) {                                                         \
            std::printf("%s:%d: %s (%s)\n", __FILE__, __LINE__, #x, jp_last_error()); \
            ++failures;                                                     \
        }                                                                   \
    } while (0)

static bool is(const fake::Op& o, const char* kernel) {
    return o.kind == fake::Op::KERNEL && o.name.find(kernel) != std::string::npos;
}
template <class T>
static T arg(const fake::Op& o, int i) {
    return *static_cast<T*>(o.args[i]);
}

// ---- an AMR solver of 64 coarse blocks whose adaptation kernels "find" the grid in `grid` ----
static AdaptCounts grid;
static jp_solver* amr(double max_gb, int flags = 0) {
    jp_config c;
    jp_config_default(&c, JP_AMR);
    c.n = 32;
    c.l1_mode = c.l2_mode = JP_REFINE_SENSOR;
    c.frac1 = 0.25;
    c.develop_steps = 1;
    c.max_gb = max_gb;
    c.flags = flags;
    jp_solver* s = nullptr;
    CHECK(jp_create(&c, &s) == JP_OK);
    return s;
}
static void set_grid(int nref0, int nref1) {
    grid = AdaptCounts{};
    grid.nref0 = nref0;
    grid.nf1 = 8 * nref0;
    grid.nref1 = nref1;
    grid.nf2 = 8 * nref1;
    grid.n_skin0 = nref0;
    grid.n_skin1 = nref1;
}
static jp_solver* watched = nullptr;  // its level-1 capacity decides whether the grid overflows
static void supply_grid() {
    fake::on_d2h = [](void* dst, size_t bytes) {
        if (bytes != sizeof(AdaptCounts)) return;
        jp_amr_counts c;
        const bool over = watched && jp_amr_get_counts(watched, &c) == JP_OK && grid.nf1 > c.cap1;
        grid.err = over ? jp::amr::ADAPT_ERR_CAP1 : 0;
        std::memcpy(dst, &grid, bytes);
    };
}
// k_leaf_macro writes the values of every unit of its grid
static void check_leaf_macro(fake::Op& o) {
    if (is(o, "k_leaf_macro") && fake::room(arg<const void*>(o, 4)) < (size_t)o.grid.x * 512 * 16)
        fake::fault("k_leaf_macro past its buffer");
}

// Every list of the coarse step grows from a count that a fill has set to zero: on every route through an
// adaptation the fill is ordered after the last use of the count and before the kernel that adds to it.
static void regrid_orders_list_counts() {
    struct Use {
        size_t op;
        const char* count;
    };
    std::vector<Use> uses;
    fake::on_kernel = [&](fake::Op& o) {
        const int i = is(o, "k_fill_list") ? 2 : is(o, "k_prep_list") ? 7 : is(o, "k_prep_cells") ? 4 : -1;
        if (i >= 0) uses.push_back({fake::ops.size() - 1, arg<const char*>(o, i)});
    };
    supply_grid();
    set_grid(16, 10);
    jp_solver* s = amr(64.0);
    for (int k = 0; k < 3; ++k) {
        CHECK(jp_step(s, 2) == JP_OK);
        set_grid(15 + k, 12 - k);
        CHECK(jp_regrid(s) == JP_OK);
    }
    CHECK(uses.size() == 4 * 6);  // one initial build, three regrids
    std::map<const char*, size_t> last;
    for (const Use& u : uses) {
        long long fill = -1;
        for (size_t i = 0; i < u.op; ++i) {
            const fake::Op& o = fake::ops[i];
            if (o.kind == fake::Op::MEMSET && u.count >= o.dst && u.count < o.dst + o.bytes) fill = (long long)i;
        }
        CHECK(fill >= 0);
        if (fill < 0) continue;
        CHECK(fake::before(fake::ops[fill], fake::ops[u.op]));
        if (last.count(u.count)) CHECK(fake::before(fake::ops[last[u.count]], fake::ops[fill]));
        last[u.count] = u.op;
    }
    jp_destroy(s);
}

// Whichever allocation of a pool's growth fails, a later diagnostic writes within its buffer: also once
// there is memory again and a grid is built that the grown capacities hold.
static void growth_out_of_memory_then_diag() {
    supply_grid();
    fake::on_kernel = check_leaf_macro;
    double d[3];
    for (const bool level1 : {false, true}) {
        for (int k = 0; k < 80; ++k) {
            set_grid(16, 10);
            jp_solver* s = watched = amr(64.0);
            CHECK(jp_diag(s, d) == JP_OK);
            if (level1) set_grid(40, 10);   // 320 blocks, 184 held
            else set_grid(16, 40);          // 320 blocks, 200 held
            fake::fail_from = fake::fail_to = fake::allocations + k;
            const jp_status grown = jp_regrid(s);
            const bool reached = fake::allocations > fake::fail_from;
            fake::fail_to = -1;
            CHECK(grown == (reached ? JP_ERR_NOMEM : JP_OK));
            if (level1) set_grid(45, 20);
            else set_grid(22, 48);
            jp_status st = jp_regrid(s);
            if (st == JP_ERR_STATE) st = jp_init_tgv(s);
            CHECK(st == JP_OK);
            CHECK(jp_diag(s, d) == JP_OK);
            jp_destroy(s);
            watched = nullptr;
            if (!reached) break;
        }
    }
}

// Out of memory for a buffer of the pools' size, a diagnostic takes one of the grid's own.
static void diag_buffer_of_the_grid() {
    supply_grid();
    fake::on_kernel = check_leaf_macro;
    double d[3];
    set_grid(16, 10);
    jp_solver* s = amr(64.0);
    fake::fail_from = fake::fail_to = fake::allocations;
    CHECK(jp_diag(s, d) == JP_OK);
    fake::fail_to = -1;
    set_grid(22, 20);
    CHECK(jp_regrid(s) == JP_OK);
    CHECK(jp_diag(s, d) == JP_OK);
    const long long held = fake::allocations;
    set_grid(16, 24);
    CHECK(jp_regrid(s) == JP_OK);
    CHECK(jp_diag(s, d) == JP_OK);
    CHECK(fake::allocations == held);  // a regrid within the pools keeps the buffer
    jp_destroy(s);
}

// A regrid whose level-2 blocks neither fit nor may grow leaves no count that the pools do not hold: the calls that
// need a grid refuse, every other stays within its arrays, and a new initial state or a state file brings the
// solver back.
static void refused_level2_growth_leaves_no_grid() {
    supply_grid();
    fake::on_kernel = check_leaf_macro;
    double d[3];
    set_grid(16, 10);
    const std::string path = "refused.jps";
    jp_solver* s = watched = amr(0.075);  // 384 blocks of 184,589 bytes, not 584
    CHECK(jp_diag(s, d) == JP_OK);
    CHECK(jp_save_state(s, path.c_str()) == JP_OK);
    jp_ensemble* e = nullptr;
    CHECK(jp_ensemble_create(0, &e) == JP_OK && jp_ensemble_add(e, s) == JP_OK);
    for (int k = 0; k < 2; ++k) {
        set_grid(20, 40);  // 320 blocks, 200 held
        CHECK(jp_regrid(s) == JP_ERR_CAPACITY);
        CHECK(jp_diag(s, d) == JP_ERR_STATE);
        CHECK(jp_step(s, 1) == JP_ERR_STATE);
        CHECK(jp_regrid(s) == JP_ERR_STATE);
        CHECK(jp_ensemble_step(e, 1) == JP_ERR_STATE);
        jp_amr_counts c;
        CHECK(jp_amr_get_counts(s, &c) == JP_OK && c.nf1 <= c.cap1 && c.nf2 <= c.cap2);
        std::vector<int> table(4096);
        for (int t = JP_TABLE_REF0; t <= JP_TABLE_DEEP; ++t) {
            int64_t n = 0;
            CHECK(jp_get_table(s, t, table.data(), (int64_t)table.size(), &n) == JP_OK);
        }
        for (int level = 0; level < 3; ++level) {
            int64_t n = 0;
            CHECK(jp_population_count(s, level, &n) == JP_OK);
            std::vector<double> p(n + 1);
            CHECK(jp_get_populations(s, level, JP_LAYOUT_BLOCKED, JP_F32, p.data(), n) == JP_OK);
            CHECK(jp_get_populations(s, level, JP_LAYOUT_BLOCKED, JP_F64, p.data(), n) == JP_OK);
        }
        CHECK(jp_save_state(s, "dropped.jps") == JP_OK);
        set_grid(16, 10);
        CHECK((k == 0 ? jp_init_tgv(s) : jp_load_state(s, path.c_str())) == JP_OK);
        CHECK(jp_step(s, 1) == JP_OK && jp_diag(s, d) == JP_OK && jp_ensemble_step(e, 1) == JP_OK);
        CHECK(jp_amr_get_counts(s, &c) == JP_OK && c.nf2 == 80);
    }
    set_grid(30, 10);  // level 1 refused: the grid at hand stays
    CHECK(jp_regrid(s) == JP_ERR_CAPACITY);
    jp_amr_counts c;
    CHECK(jp_amr_get_counts(s, &c) == JP_OK && c.nf1 == 128 && c.nf2 == 80);
    CHECK(jp_step(s, 1) == JP_OK && jp_diag(s, d) == JP_OK);
    set_grid(16, 40);  // an initial build that does not fit
    CHECK(jp_init_tgv(s) == JP_ERR_CAPACITY);
    CHECK(jp_diag(s, d) == JP_ERR_STATE);
    CHECK(jp_amr_get_counts(s, &c) == JP_OK && c.nf2 <= c.cap2);
    set_grid(16, 10);
    CHECK(jp_init_tgv(s) == JP_OK && jp_diag(s, d) == JP_OK);
    jp_ensemble_destroy(e);
    jp_destroy(s);
}

static int count_of(const char* kernel, size_t from) {
    int n = 0;
    for (size_t i = from; i < fake::ops.size(); ++i) n += is(fake::ops[i], kernel);
    return n;
}
static jp_solver* cube(int n, int vec, int tpb, int flags = 0) {
    jp_config c;
    jp_config_default(&c, JP_UNIFORM);
    c.n = n;
    c.vec = vec;
    c.threads_per_block = tpb;
    c.flags = flags;
    jp_solver* s = nullptr;
    CHECK(jp_create(&c, &s) == JP_OK);
    return s;
}

// A thread mapping that the caller chose is that of every step, alone and in an ensemble; with none, FP32 cubes of
// these sizes step two at a time.  The autotuner answers with the mapping whose rate it reports.
static void chosen_mapping_takes_every_step() {
    const int maps[4][2] = {{0, 0}, {4, 0}, {0, 256}, {2, 128}};
    for (const auto& m : maps) {
        const bool chosen = m[0] || m[1];
        jp_solver* s = cube(32, m[0], m[1]);
        size_t from = fake::ops.size();
        CHECK(jp_step(s, 5) == JP_OK);
        CHECK(count_of("k_stream_collide_pair", from) == (chosen ? 0 : 2));
        CHECK(count_of("k_stream_collide", from) == (chosen ? 5 : 3));
        jp_destroy(s);
        jp_ensemble* e = nullptr;
        CHECK(jp_ensemble_create(0, &e) == JP_OK);
        std::vector<jp_solver*> v;
        for (int n : {32, 48, 64, 96, 128, 32, 48, 64, 96, 128}) {
            v.push_back(cube(n, m[0], m[1]));
            CHECK(jp_ensemble_add(e, v.back()) == JP_OK);
        }
        from = fake::ops.size();
        CHECK(jp_ensemble_step(e, 5) == JP_OK);
        CHECK(count_of("k_stream_collide_pair", from) == (chosen ? 0 : 2));
        CHECK(count_of("k_stream_collide", from) == (chosen ? 5 : 3));
        jp_ensemble_destroy(e);
        for (jp_solver* x : v) jp_destroy(x);
    }
    for (const bool two_faster : {true, false}) {
        // a single step takes 1 ms, a two-step pass 1.5 or 2.5
        size_t from = fake::ops.size();
        fake::elapsed = [&] {  // of four steps
            return !is(fake::ops.back(), "k_stream_collide_pair") ? 4.f : two_faster ? 3.f : 5.f;
        };
        jp_config c;
        jp_config_default(&c, JP_UNIFORM);
        c.n = 32;
        double best = 0;
        CHECK(jp_autotune(&c, 4, &best) == JP_OK);
        CHECK(count_of("k_stream_collide_pair", from) > 0);
        CHECK((c.vec == 0) == two_faster && (c.threads_per_block == 0) == two_faster);
        CHECK(best == 32.0 * 32 * 32 * 4 / ((two_faster ? 3.0 : 4.0) * 1e-3));
    }
}

// The relaxation's coefficients are the combination of each value's nearest float and its two neighbours that
// keeps mass best, at every viscosity (1 / (omega w) is above 64 for omega below 0.28).
static void coefficients_search_both_neighbours() {
    for (float omega : {1.99f, 1.6f, 1.0f, 0.5f, 0.29f, 0.27f, 0.2f, 0.1357f, 0.08f, 0.031f, 0.0021f, 3.3e-5f}) {
        const jp::BgkCoef c = jp::bgk_coefficients(omega);
        const double om = omega;
        const auto off = [&](double b0, double b1, double b2, double k1, double k2) {
            const double c0 = b0 + 6 * b1 + 12 * b2;
            const double k = k1 * (double(c.a1) * c.a1) + 4 * k2 * (double(c.a2) * c.a2);
            return std::fabs(2 * k - 1.5 * c0) + 0.1 * std::fabs(c0 - om);
        };
        std::vector<float> v[5];
        const double exact[5] = {om / 3, om / 18, om / 36, 9 / om, 18 / om};
        for (int i = 0; i < 5; ++i)
            for (float to : {-INFINITY, float(exact[i]), INFINITY}) v[i].push_back(std::nextafter(float(exact[i]), to));
        double least = INFINITY;
        for (float b0 : v[0])
            for (float b1 : v[1])
                for (float b2 : v[2])
                    for (float k1 : v[3])
                        for (float k2 : v[4]) least = std::min(least, off(b0, b1, b2, k1, k2));
        CHECK(off(c.b0, c.b1, c.b2, c.k1, c.k2) == least);
    }
}

// An in-place cube holds one population array: the memory that a conversion takes goes back with it.
static void in_place_conversions_keep_no_memory() {
    for (const int n : {8, 32, 64}) {
        jp_solver* s = cube(n, 0, 0, JP_FLAG_INPLACE);
        const int64_t count = 19LL * n * n * n;
        std::vector<double> p(count);
        jp_info before, after;
        CHECK(jp_get_info(s, &before) == JP_OK);
        const size_t held = fake::allocated();
        for (int k = 0; k < 2; ++k) {
            CHECK(jp_get_populations(s, 0, JP_LAYOUT_FLAT, JP_F64, p.data(), count) == JP_OK);
            CHECK(fake::allocated() == held);
            CHECK(jp_set_populations(s, 0, JP_LAYOUT_BLOCKED, JP_F32, p.data(), count) == JP_OK);
            CHECK(fake::allocated() == held);
        }
        CHECK(jp_get_info(s, &after) == JP_OK && after.bytes_state == before.bytes_state);
        jp_destroy(s);
    }
}

// With no device memory left, populations still convert: through the other array, or in place through the scratch
// that the cube was created with.
static void conversions_without_memory() {
    for (const int flags : {0, (int)JP_FLAG_INPLACE}) {
        jp_solver* s = cube(32, 0, 0, flags);
        const int64_t count = 19LL * 32 * 32 * 32;
        std::vector<double> p(count);
        fake::fail_from = fake::allocations;
        fake::fail_to = 1LL << 60;
        for (const int layout : {(int)JP_LAYOUT_FLAT, (int)JP_LAYOUT_BLOCKED})
            for (const int dtype : {(int)JP_F32, (int)JP_F64}) {
                CHECK(jp_get_populations(s, 0, layout, dtype, p.data(), count) == JP_OK);
                CHECK(jp_set_populations(s, 0, layout, dtype, p.data(), count) == JP_OK);
            }
        fake::fail_to = -1;
        const size_t from = fake::ops.size();
        CHECK(jp_get_populations(s, 0, JP_LAYOUT_FLAT, JP_F64, p.data(), count) == JP_OK);
        CHECK(count_of("k_convert", from) == 2);
        jp_destroy(s);
    }
}

// A conversion that fails half-way returns with none of its copies still reading or writing the caller's memory.
static void failed_conversion_waits_for_its_copies() {
    for (const int chunk : {1, 2, 3}) {
        jp_solver* s = cube(32, 0, 0, JP_FLAG_INPLACE);
        const int64_t count = 19LL * 32 * 32 * 32;
        std::vector<double> p(count);
        int launches = 0;
        fake::fail_from = fake::allocations;  // many chunks
        fake::fail_to = 1LL << 60;
        fake::launch_error = [&](const std::string& k) {
            if (k.find("k_convert") == std::string::npos || ++launches < chunk) return cudaSuccess;
            return cudaErrorLaunchOutOfResources;
        };
        CHECK(jp_get_populations(s, 0, JP_LAYOUT_FLAT, JP_F64, p.data(), count) == JP_ERR_CUDA);
        CHECK(fake::copies_in_flight() == 0);
        launches = 0;
        CHECK(jp_set_populations(s, 0, JP_LAYOUT_FLAT, JP_F64, p.data(), count) == JP_ERR_CUDA);
        CHECK(fake::copies_in_flight() == 0);
        fake::launch_error = nullptr;
        fake::fail_to = -1;
        jp_destroy(s);
    }
}

// Coarse steps without JP_FLAG_GRAPH count their kernels alike, launched directly or replayed.
static void replayed_steps_count_their_kernels() {
    supply_grid();
    for (const int nref1 : {10, 0}) {
        set_grid(16, nref1);
        jp_solver* s = amr(64.0);
        int64_t each = 0;
        for (int k = 0; k < 16; ++k) {
            const int64_t c0 = jp_launch_count();
            CHECK(jp_step(s, 1) == JP_OK);
            const int64_t n = jp_launch_count() - c0;
            if (k == 0) each = n;
            CHECK(n == each && n > 0);
        }
        size_t replays = 0;
        for (const fake::Op& o : fake::ops) replays += o.kind == fake::Op::GRAPH_LAUNCH;
        CHECK(replays > 0);
        jp_destroy(s);
    }
}

// A captured step replayed on another stream than the solver's: its upload is ordered before it.
static void upload_precedes_replay_on_its_stream() {
    supply_grid();
    set_grid(16, 10);
    jp_solver* s = amr(64.0, JP_FLAG_GRAPH);
    cudaStream_t lane;
    CHECK(cudaStreamCreateWithFlags(&lane, cudaStreamNonBlocking) == cudaSuccess);
    const size_t from = fake::ops.size();
    for (int k = 0; k < 4; ++k) CHECK(jp::amr_graph_step_on(s, lane) == JP_OK);
    const fake::Op* upload = nullptr;
    int replays = 0;
    for (size_t i = from; i < fake::ops.size(); ++i) {
        const fake::Op& o = fake::ops[i];
        if (o.kind == fake::Op::GRAPH_UPLOAD) upload = &o;
        if (o.kind != fake::Op::GRAPH_LAUNCH) continue;
        ++replays;
        CHECK(o.stream == lane && upload && fake::before(*upload, o));
    }
    CHECK(replays == 4);
    jp_destroy(s);
}

// Steps become graphs without a stream capture, which would make other threads' calls that wait for the device
// fail meanwhile, and a graph's kernels are ordered exactly as the launches of the step are.
static void graphs_order_kernels_as_streams_do() {
    supply_grid();
    for (const int flags : {0, (int)JP_FLAG_GRAPH, (int)JP_FLAG_SKIP_PREP, (int)JP_FLAG_SKIP_RESTRICT})
        for (const int nref1 : {10, 0}) {
            set_grid(16, nref1);
            jp_solver* s = amr(64.0, flags & JP_FLAG_GRAPH ? 0 : flags);  // one step by launches
            size_t from = fake::ops.size();
            CHECK(jp_step(s, 1) == JP_OK);
            const std::vector<fake::Op> direct(fake::ops.begin() + (long)from, fake::ops.end());
            jp_solver* g = flags & JP_FLAG_GRAPH ? amr(64.0, flags) : s;
            from = fake::ops.size();
            CHECK(jp_step(g, 8) == JP_OK);
            for (size_t i = from; i < fake::ops.size(); ++i) CHECK(fake::ops[i].kind != fake::Op::CAPTURE);
            CHECK(!fake::graphs.empty());
            if (fake::graphs.empty()) return;
            const std::vector<fake::Node>& nodes = fake::graphs.back();
            CHECK(nodes.size() == direct.size());
            // the same kernels in the order of issue
            for (size_t i = 0; i < nodes.size() && i < direct.size(); ++i) CHECK(nodes[i].name == direct[i].name);
            for (size_t i = 0; i < nodes.size() && i < direct.size(); ++i)
                for (size_t j = 0; j < i; ++j)
                    CHECK(std::count(nodes[i].after.begin(), nodes[i].after.end(), j) == (fake::before(direct[j], direct[i]) ? 1 : 0));
            if (g != s) jp_destroy(g);
            jp_destroy(s);
        }
}

// A state file that ends early, or memory that does, half-way through a load leaves no mixture of two grids (and no
// recorded steps of arrays that have moved): the solver has no grid until a load or a new initial state succeeds.
static void failed_load_leaves_no_grid() {
    supply_grid();
    fake::on_kernel = check_leaf_macro;
    double d[3];
    set_grid(20, 18);
    jp_solver* big = amr(64.0);
    set_grid(16, 10);
    CHECK(jp_save_state(big, "big.jps") == JP_OK);
    jp_destroy(big);
    std::FILE* f = std::fopen("big.jps", "rb");
    std::vector<char> bytes(64 << 20);
    bytes.resize(std::fread(bytes.data(), 1, bytes.size(), f));
    std::fclose(f);
    jp_solver* s = amr(64.0);
    const auto refused = [&](jp_status want) {
        CHECK(jp_load_state(s, "cut.jps") == want);
        CHECK(jp_step(s, 1) == JP_ERR_STATE && jp_diag(s, d) == JP_ERR_STATE);
        set_grid(16, 10);
        CHECK(jp_init_tgv(s) == JP_OK && jp_step(s, 12) == JP_OK && jp_diag(s, d) == JP_OK);
    };
    const auto cut = [&](size_t n) {
        std::FILE* out = std::fopen("cut.jps", "wb");
        std::fwrite(bytes.data(), 1, n, out);
        std::fclose(out);
    };
    CHECK(jp_step(s, 12) == JP_OK);  // recorded
    cut(100);
    CHECK(jp_load_state(s, "cut.jps") == JP_ERR_INVALID);  // within the headers: nothing touched
    CHECK(jp_step(s, 1) == JP_OK);
    for (const size_t n : {(size_t)300, (size_t)5000, bytes.size() / 2, bytes.size() - 4}) {
        cut(n);
        refused(JP_ERR_INVALID);
    }
    cut(bytes.size());
    for (int k = 0; k < 7; ++k) {  // the level-2 pool's arrays
        fake::fail_from = fake::fail_to = fake::allocations + k;
        refused(JP_ERR_NOMEM);
    }
    fake::fail_to = -1;
    CHECK(jp_load_state(s, "cut.jps") == JP_OK && jp_step(s, 12) == JP_OK && jp_diag(s, d) == JP_OK);
    jp_destroy(s);
    // into pools larger than the file's, whose arrays shrink one by one
    for (int k = 0; k < 60; ++k) {
        set_grid(16, 10);
        s = watched = amr(64.0);
        set_grid(40, 40);
        CHECK(jp_regrid(s) == JP_OK);
        fake::fail_from = fake::fail_to = fake::allocations + k;
        const jp_status st = jp_load_state(s, "big.jps");
        fake::fail_to = -1;
        set_grid(40, 40);
        CHECK(st == JP_ERR_NOMEM ? jp_init_tgv(s) == JP_OK : st == JP_OK);
        jp_amr_counts c;
        CHECK(jp_step(s, 2) == JP_OK && jp_diag(s, d) == JP_OK && jp_amr_get_counts(s, &c) == JP_OK);
        std::vector<float> p(19 * 512 * 2000);
        for (int level = 0; level < 3; ++level) {
            int64_t n = 0;
            CHECK(jp_population_count(s, level, &n) == JP_OK);
            CHECK(jp_get_populations(s, level, JP_LAYOUT_BLOCKED, JP_F32, p.data(), n) == JP_OK);
        }
        CHECK(c.nf1 <= c.cap1 && c.nf2 <= c.cap2);
        watched = nullptr;
        jp_destroy(s);
        if (st == JP_OK) break;
        CHECK(k < 59);
    }
}

int main(int argc, char** argv) {
    const std::map<std::string, void (*)()> checks = {
        {"regrid_orders_list_counts", regrid_orders_list_counts},
        {"growth_out_of_memory_then_diag", growth_out_of_memory_then_diag},
        {"diag_buffer_of_the_grid", diag_buffer_of_the_grid},
        {"refused_level2_growth_leaves_no_grid", refused_level2_growth_leaves_no_grid},
        {"chosen_mapping_takes_every_step", chosen_mapping_takes_every_step},
        {"coefficients_search_both_neighbours", coefficients_search_both_neighbours},
        {"in_place_conversions_keep_no_memory", in_place_conversions_keep_no_memory},
        {"conversions_without_memory", conversions_without_memory},
        {"failed_conversion_waits_for_its_copies", failed_conversion_waits_for_its_copies},
        {"replayed_steps_count_their_kernels", replayed_steps_count_their_kernels},
        {"upload_precedes_replay_on_its_stream", upload_precedes_replay_on_its_stream},
        {"graphs_order_kernels_as_streams_do", graphs_order_kernels_as_streams_do},
        {"failed_load_leaves_no_grid", failed_load_leaves_no_grid},
    };
    const auto it = argc == 2 ? checks.find(argv[1]) : checks.end();
    if (it == checks.end()) return 2;
    it->second();
    for (const std::string& f : fake::faults) std::printf("%s\n", f.c_str());
    std::printf("%d failed checks, %zu faults\n", failures, fake::faults.size());
    return failures || !fake::faults.empty() ? 1 : 0;
}

// host_engine_check.cpp -- the host side of the library over a fake CUDA runtime
// (fake_cudart.h).  argv: the scenario, then a continuous-energy problem's
// folder, its cross-section folder, a one-group problem's folder, that of one
// with many bins and a folder to write to.  Prints "ok", or what is wrong.
#include <cstdio>
#include <cstring>
#include <functional>
#include <string>
#include <thread>
#include <vector>

#include "fake_cudart.h"
#include "mc_device.h"
#include "mcgpu.h"

static std::string ce, xs, mg, tmp, wide;
constexpr size_t kWideBins = 20003;   // of the wide problem (4 layers, one group)
static int bad = 0;
#define WANT(x)                                                          \
    do {                                                                 \
        if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } \
    } while (0)

static mc_problem *load(const std::string &d)
{
    mc_problem *p = nullptr;
    if (mc_problem_load_xml(d.c_str(), xs.c_str(), &p) != MC_OK) {
        std::printf("load: %s\n", mc_last_error(p));
        std::exit(2);
    }
    return p;
}

// Two threads read different estimators of one handle at the same time, as a
// const handle allows.
static void concurrent_reads()
{
    mc_problem *p = load(ce);
    uint32_t ne = 0;
    mc_tally_count(p, &ne);
    WANT(ne >= 2);
    // distinct sums in every bin, by way of a saved state
    const std::string f = tmp + "/state";
    WANT(mc_state_save(p, f.c_str()) == MC_OK);
    std::vector<char> raw;
    if (FILE *h = std::fopen(f.c_str(), "rb")) {
        for (int c; (c = std::fgetc(h)) != EOF;) raw.push_back((char)c);
        std::fclose(h);
    }
    const size_t head = 8 + 4 * 8, bins = (raw.size() - head) / 16;
    for (size_t j = 0; j < 2 * bins; ++j) {
        const double v = 1.0 + (double)j;
        std::memcpy(&raw[head + 8 * j], &v, 8);
    }
    if (FILE *h = std::fopen(f.c_str(), "wb")) {
        std::fwrite(raw.data(), 1, raw.size(), h);
        std::fclose(h);
    }
    WANT(mc_state_load(p, f.c_str()) == MC_OK);
    fake::meet(2, 300);
    std::vector<double> sum[2], sq[2];
    std::vector<std::thread> ts;
    for (uint32_t e = 0; e < 2; ++e)
        ts.emplace_back([&, e] {
            uint64_t nb = 0;
            mc_tally_size(p, e, &nb);
            sum[e].assign(nb, 0.0);
            sq[e].assign(nb, 0.0);
            WANT(mc_tally_read(p, e, nullptr, nullptr, sum[e].data(), sq[e].data(), nb) == MC_OK);
        });
    for (auto &t : ts) t.join();
    fake::meet(0, 0);
    double want = 1.0;
    for (int e = 0; e < 2; ++e)
        for (size_t j = 0; j < sum[e].size(); ++j, want += 1.0) WANT(sum[e][j] == want && sq[e][j] == want + (double)bins);
    mc_problem_free(p);
}

// A handle whose problem was not loaded has no tallies to clear or to read.
static void not_loaded()
{
    mc_problem *p = nullptr;
    WANT(mc_problem_load_xml((tmp + "/nowhere").c_str(), xs.c_str(), &p) == MC_ERR_INPUT);
    WANT(p != nullptr);
    WANT(mc_reset_tallies(p) != MC_OK);
    WANT(mc_state_save(p, (tmp + "/none").c_str()) != MC_OK);
    WANT(mc_run(p, 0, 10, 1, MC_MIXED_EVENT, nullptr) != MC_OK);
    mc_problem_free(p);
}

// A batch's graph holds the scratch buffers' addresses: a run that makes one of
// them grow needs another graph.
static void deeper_stack()
{
    mc_problem *ps[2] = {load(mg), load(mg)};
    const uint64_t n[2] = {5000, 70};
    mc_batch *b = nullptr;
    WANT(mc_batch_create(ps, 2, n, &b) == MC_OK);
    mc_tune t;
    std::memset(&t, 0, sizeof(t));
    t.kernel = 2;
    fake::reset();
    WANT(mc_batch_run(b, 1, &t) == MC_OK && fake::captures() == 1);
    WANT(mc_batch_run(b, 2, &t) == MC_OK && fake::captures() == 1);   // the same graph again
    t.stack_depth = 100;
    WANT(mc_batch_run(b, 3, &t) == MC_OK && fake::captures() == 2);
    WANT(mc_batch_run(b, 4, &t) == MC_OK && fake::captures() == 2);
    t.stack_depth = 3;
    WANT(mc_batch_run(b, 5, &t) == MC_OK && fake::captures() == 3);   // and another overflow limit
    mc_batch_free(b);
    for (mc_problem *p : ps) mc_problem_free(p);
}

static mc_tune tuned(uint32_t kernel, uint32_t chunk = 0, uint32_t digests = 0)
{
    mc_tune t;
    std::memset(&t, 0, sizeof(t));
    t.kernel = kernel;
    t.chunk = chunk;
    t.record_digests = digests;
    return t;
}

// A failed query of a kernel's residency is not kept: the next run asks again.
static void failed_query()
{
    int refused = 0;
    for (long k = 0;; ++k) {
        mc_problem *p = load(ce);
        const mc_tune t = tuned(2);
        fake::reset();
        fake::fail_call(k);
        const mc_status st = mc_run(p, 0, 1000, 1, MC_MIXED_EVENT, &t);
        const bool hit = fake::failed();
        fake::reset();
        if (st == MC_ERR_ARG) {
            ++refused;
            WANT(mc_run(p, 0, 1000, 1, MC_MIXED_EVENT, &t) == MC_OK);
        }
        mc_problem_free(p);
        if (!hit) break;
    }
    WANT(refused > 0);
}

// A run whose second kernel, the one that adds the replicated sums, could not be
// launched fails, and its replicas are cleared before the next run folds into
// them, whatever runs in between.
static void failed_reduce()
{
    mc_problem *p = load(ce);
    uint32_t ne = 0;
    size_t bins = 0;
    mc_tally_count(p, &ne);
    for (uint32_t e = 0; e < ne; ++e) {
        uint64_t n = 0;
        mc_tally_size(p, e, &n);
        bins += n;
    }
    const mc_tune t = tuned(2);
    auto run = [&](uint64_t n) { return mc_run(p, 0, n, 1, MC_MIXED_EVENT, &t); };
    auto cleared = [&] {
        for (const fake::Fill &f : fake::fills())
            if (f.bytes == 64 * 2 * sizeof(double) * ((bins + 15) & ~(size_t)15)) return true;   // in whole lines
        return false;
    };
    WANT(run(70000) == MC_OK && cleared());
    fake::reset();
    WANT(run(70000) == MC_OK && !cleared());    // the second kernel leaves them clear
    for (int between = 0; between < 2; ++between) {
        fake::reset();
        fake::fail_launch("k_batch_reduce");
        WANT(run(70000) != MC_OK && fake::failed());
        if (between) {
            fake::reset();
            fake::fail_launch("k_track");
            WANT(run(1000) != MC_OK && fake::failed());
        }
        fake::reset();
        WANT(run(70000) == MC_OK && cleared());
    }
    mc_problem_free(p);
}

// A handle and what belongs to it, for one attempt.
struct Attempt {
    mc_problem *p = nullptr, *q = nullptr;
    mc_batch *b = nullptr;
    std::vector<double> out;
    explicit Attempt(const std::string &d) : p(load(d)), out(4096) {}
    ~Attempt()
    {
        if (b) mc_batch_free(b);
        if (q) mc_problem_free(q);
        mc_problem_free(p);
    }
};

// Every runtime call of `act` fails once: the status tells, and the same call
// on the same handle works afterwards.
static void every_call(const char *name, const std::string &d, const std::function<void(Attempt &)> &setup,
                       const std::function<mc_status(Attempt &)> &act)
{
    for (long k = 0;; ++k) {
        Attempt a(d);
        setup(a);
        fake::reset();
        fake::fail_call(k);
        const mc_status st = act(a);
        if (!fake::failed()) {
            if (st != MC_OK || k == 0) { std::printf("%s: %d calls, status %d\n", name, (int)k, (int)st); ++bad; }
            fake::reset();
            return;
        }
        fake::fail_call(-1);
        if (st == MC_OK) { std::printf("%s: call %d failed and nobody noticed\n", name, (int)k); ++bad; }
        const mc_status again = act(a);
        if (again != MC_OK) {
            std::printf("%s: after call %d failed: status %d, %s\n", name, (int)k, (int)again, mc_last_error(a.p));
            ++bad;
        }
        fake::reset();
    }
}

static void failed_calls()
{
    auto none = [](Attempt &) {};
    auto run = [](uint64_t n, mc_mode m, mc_tune t) { return [=](Attempt &a) { return mc_run(a.p, 0, n, 1, m, &t); }; };
    every_call("mixed, sums in shared memory", ce, none, run(1000, MC_MIXED_EVENT, tuned(2)));
    every_call("mixed, replicas", ce, none, run(70000, MC_MIXED_EVENT, tuned(2)));
    every_call("mixed, replicas, second run", ce, [&](Attempt &a) { run(70000, MC_MIXED_EVENT, tuned(2))(a); },
               run(70000, MC_MIXED_EVENT, tuned(2)));
    every_call("mixed, multigroup", mg, none, run(300000, MC_MIXED_EVENT, tuned(2)));
    every_call("mixed, tile kernel", mg, none, run(1000, MC_MIXED_EVENT, tuned(1)));
    every_call("replay", ce, none, run(1000, MC_FP64_REPLAY, tuned(0)));
    every_call("replay in chunks, with digests", mg, none, run(1000, MC_FP64_REPLAY, tuned(0, 300, 1)));
    every_call("plain", mg, none, run(1000, MC_FP64_PLAIN, tuned(0)));
    every_call("reset", ce, none, [](Attempt &a) { return mc_reset_tallies(a.p); });
    every_call("read", ce, none, [](Attempt &a) { return mc_tally_read(a.p, 1, a.out.data(), nullptr, nullptr, nullptr, a.out.size()); });
    every_call("upload", ce, [&](Attempt &a) { run(10, MC_MIXED_EVENT, tuned(2))(a); }, [](Attempt &a) { return mc_problem_upload(a.p); });
    auto params = [](Attempt &a) { mc_lr_params(a.p, a.out.data(), 128); };
    every_call("forward", mg, params, [](Attempt &a) { return mc_forward(a.p, a.out.data(), 1000, 1, a.out.data() + 128, a.out.data() + 1024); });
    every_call("backward", mg, params, [](Attempt &a) { return mc_backward(a.p, a.out.data(), 1000, 1, a.out.data() + 128, a.out.data() + 1024); });
    every_call("replay without allocation", mg, none,
               [](Attempt &a) { return mc_run_replay_noalloc(a.p, 0, 1000, 1, a.out.data(), a.out.data() + 1024); });
    auto batch = [](Attempt &a) {
        a.q = load(mg);
        mc_problem *ps[2] = {a.p, a.q};
        const uint64_t n[2] = {5000, 70};
        WANT(mc_batch_create(ps, 2, n, &a.b) == MC_OK);
    };
    const mc_tune two = tuned(2), one = tuned(1);
    every_call("batch", mg, batch, [&](Attempt &a) { return mc_batch_run(a.b, 1, &two); });
    every_call("batch, another shape", mg, [&](Attempt &a) { batch(a); mc_batch_run(a.b, 1, &two); },
               [&](Attempt &a) { const mc_status st = mc_batch_run(a.b, 1, &one); return st != MC_OK ? st : mc_batch_run(a.b, 1, &two); });
    every_call("batch reset", mg, batch, [](Attempt &a) { return mc_batch_reset(a.b); });
    every_call("batch read", mg, batch, [](Attempt &a) {
        return mc_batch_tally_read(a.b, a.out.data(), nullptr, nullptr, nullptr, a.out.size());
    });
}

// The replay without allocation clears the rows that it uses, not its scratch.
static void noalloc_clears()
{
    Attempt a(mg);
    size_t bins = 0;
    uint32_t ne = 0;
    mc_tally_count(a.p, &ne);
    for (uint32_t e = 0; e < ne; ++e) {
        uint64_t n = 0;
        mc_tally_size(a.p, e, &n);
        bins += n;
    }
    for (uint64_t n : {1, 8, 9, 1000}) {
        fake::reset();
        WANT(mc_run_replay_noalloc(a.p, 0, n, 1, a.out.data(), a.out.data() + 1024) == MC_OK);
        size_t most = 0;
        for (const fake::Fill &f : fake::fills()) most = f.bytes > most ? f.bytes : most;
        WANT(most <= 4096 || most == (n + 7) / 8 * 8 * bins * sizeof(double));
    }
}

// The FP64 kernels' launch shape is that of the histories of one launch, not of
// the whole run: few of them are spread over all schedulers.
static void launch_shape()
{
    Attempt a(ce);
    auto grid = [&](uint32_t chunk, uint64_t n, mc_mode m) {
        const mc_tune t = tuned(0, chunk);
        fake::reset();
        WANT(mc_run(a.p, 0, n, 1, m, &t) == MC_OK);
        unsigned g = 0;
        for (const fake::Launch &l : fake::launches())
            if (l.kernel.find("k_history_fp64") != std::string::npos) { WANT(g == 0 || g == l.grid); g = l.grid; }
        return g;
    };
    for (mc_mode m : {MC_FP64_REPLAY, MC_FP64_PLAIN})
        for (uint32_t chunk : {1u, 61u, 600u, 5000u}) WANT(grid(chunk, 100000, m) == grid(chunk, chunk, m));
    WANT(grid(61, 100000, MC_FP64_REPLAY) == 16);      // four warps to a CTA, a history to a warp
    // derivatives of a problem of so many columns that 1 GiB holds few histories
    Attempt b(wide);
    std::vector<double> par(128), out((size_t)2 * 4 * kWideBins), sg(out.size());
    WANT(mc_lr_params(b.p, par.data(), 128) == MC_OK);
    auto lr_grid = [&](uint64_t n) {
        fake::reset();
        WANT(mc_backward(b.p, par.data(), n, 1, out.data(), sg.data()) == MC_OK);
        for (const fake::Launch &l : fake::launches())
            if (l.kernel.find("k_history_fp64") != std::string::npos) return l.grid;
        return 0u;
    };
    WANT(lr_grid(3000) == lr_grid((1u << 30) / 8 / 13 / kWideBins));
}

// The columns of one launch keep within 1 GiB, or two histories.
static void row_bound()
{
    const double GiB = (double)(1u << 30);
    for (double c = 1.0; c < 4e8; c *= 1.013)
        for (uint64_t n : {(uint64_t)1, (uint64_t)5, (uint64_t)1000, (uint64_t)1 << 40}) {
            const uint64_t cols = (uint64_t)c, chunk = mc::hist_chunk(cols, n, 0), rows = mc::hist_rows(chunk);
            const double bytes = 8.0 * (double)cols * (double)rows;
            WANT(chunk >= 1 && chunk <= n && rows >= chunk && rows % 2 == 0 && rows < chunk + 8);
            WANT(bytes <= GiB || rows == 2);
            // no launch is more than a vector shorter than the bound allows
            if (chunk < n && chunk < 1u << 22) WANT((double)(chunk + 8) * 8.0 * (double)cols > GiB);
        }
    WANT(mc::hist_chunk(10, 1000, 61) == 61 && mc::hist_chunk(10, 50, 61) == 50 && mc::hist_chunk(10, (uint64_t)1 << 40, (uint64_t)1 << 30) == 1u << 22);
}

// Saved states are found again by later builds: their problems' keys, as the
// first builds that saved states wrote them.
static void state_keys()
{
    const struct { const std::string &d; uint64_t key; } known[] = {{ce, 0x1FD0E85AACFAC887ull}, {mg, 0xA429E906F037B4E1ull}};
    for (const auto &k : known) {
        Attempt a(k.d);
        const std::string f = tmp + "/keyed";
        WANT(mc_state_save(a.p, f.c_str()) == MC_OK && mc_state_load(a.p, f.c_str()) == MC_OK);
        uint64_t head[5] = {};
        if (FILE *h = std::fopen(f.c_str(), "rb")) {
            WANT(std::fread(head, 8, 5, h) == 5);
            std::fclose(h);
        }
        WANT(head[4] == k.key);
    }
}

int main(int argc, char **argv)
{
    if (argc < 7) return 2;
    ce = argv[2]; xs = argv[3]; mg = argv[4]; wide = argv[5]; tmp = argv[6];
    const struct { const char *name; void (*run)(); } all[] = {
        {"concurrent reads", concurrent_reads}, {"not loaded", not_loaded}, {"deeper stack", deeper_stack}, {"failed query", failed_query},
        {"failed reduce", failed_reduce}, {"failed calls", failed_calls},
        {"noalloc clears", noalloc_clears}, {"launch shape", launch_shape},
        {"row bound", row_bound}, {"state keys", state_keys}};
    for (const auto &s : all)
        if (std::strcmp(s.name, argv[1]) == 0) {
            s.run();
            if (!bad) std::printf("ok\n");
            return bad != 0;
        }
    std::printf("no such scenario\n");
    return 2;
}

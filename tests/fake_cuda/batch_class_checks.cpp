// TEST INFRASTRUCTURE ONLY: the host logic behind batches and the mirror-group
// kernel on the class-by-class stand-ins (batch_class_kernels.cpp).  One check
// per run, named by the first argument; prints "ok <check>".
#include "batch_class_control.h"
#include "cuda_runtime.h"
#include "fake_control.h"
#include "fake_expect.h"
#include "occastft_gb300.h"
#include "ocs_kernels.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace {

void check(bool ok, const std::string& what)
{
    if (ok) return;
    std::printf("FAIL %s (last error: %s)\n", what.c_str(), ocs_last_error());
    std::exit(1);
}

struct Batch {
    struct Item {
        std::vector<float> x, out;
        int exp;
        float ov;
        std::string opts;
    };
    std::vector<Item> items;
    std::vector<ocs_request> reqs;

    void add(uint64_t n, int exp, float ov, const std::string& opts)
    {
        Item it{std::vector<float>(n), {}, exp, ov, opts};
        std::mt19937 rng((unsigned)(n + exp));
        for (float& v : it.x) v = (float)(int)(rng() % 2001 - 1000) / 1000.0f;
        ocs_geometry g;
        check(ocs_geometry_get(n, exp, ov, opts.c_str(), &g) == OCS_OK, "geometry");
        it.out.assign(g.out_floats, -7.0f);
        items.push_back(it);
    }
    void seal()
    {
        reqs.clear();
        for (Item& it : items)
            reqs.push_back(ocs_request{it.x.data(), it.x.size(), it.exp, it.ov, it.opts.c_str(), it.out.data(),
                                       it.out.size(), -1, 0});
    }
    int run(cudaStream_t st) { return ocs_batch_device(reqs.data(), (int)reqs.size(), st); }
    bool right() const
    {
        for (const Item& it : items) {
            const std::vector<float> want = fake::expected_out(it.x.data(), it.x.size(), it.exp, it.ov, it.opts);
            if (std::memcmp(it.out.data(), want.data(), want.size() * 4) != 0) return false;
        }
        return true;
    }
};

const char* kOpts[] = {"", "--half_complex_return", "--hanning_window --serial_power", "--layout=dense",
                       "--half_complex_return --layout=dense --remove_dc"};

// Every class is one run of the tile list, in window order, with the kernel
// table of its form; the outputs are right.
void classes(cudaStream_t st)
{
    for (int round = 0; round < 4; ++round) {
        Batch b;
        for (int i = 0; i < 60; ++i) b.add(3000 + 977 * i, 6 + (i * 5 + round) % 8, 0.5f, kOpts[i % 5]);
        b.seal();
        check(b.run(st) == OCS_OK, "launch");
        cudaStreamSynchronize(st);
        check(b.right(), "outputs");
        uint32_t next = 0;
        int last = 0;
        for (const fake::ClassLaunch& c : fake::take_class_launches()) {
            check(c.begin == next, "class start");
            next += (uint32_t)c.tiles.size();
            const int exp = ocs::batch_class_exp(c.id);
            check(exp >= last, "class order");
            last = exp;
            for (const auto& t : c.tiles) {
                check(ocs::batch_class(t.exp, t.outk) == c.id, "tile's class");
                // whole rounds of the tile's body, but for a request's last tile
                const uint64_t least = ocs::batch_min_frames(t.exp, t.outk);
                check(t.f0 % least == 0 && (t.nframes % least == 0 || t.f0 + t.nframes == t.frames), "tile's frames");
                if (exp >= 12)
                    check(t.plan == ocs::mirror_plan_id(exp, ocs::batch_mirror_paired(exp, t.outk)), "table");
                else if (exp != 7 && exp != 11)
                    check(t.plan == exp, "pair plan's table");
            }
            check(next <= c.all_tiles, "tile count");
        }
    }
}

// One request at a time at 2^12 .. 2^15: the stand-in checks the table of the form.
void one_request(cudaStream_t st)
{
    for (int exp = 12; exp <= 15; ++exp)
        for (const char* o : kOpts) {
            Batch b;
            b.add(40000, exp, 0.5f, o);
            Batch::Item& it = b.items[0];
            check(ocs_activate_device(it.x.data(), it.x.size(), exp, 0.5f, o, it.out.data(), it.out.size(), st) == OCS_OK,
                  "request");
            cudaStreamSynchronize(st);
            check(b.right(), "output");
        }
}

// A class whose launch fails after another's has begun: the next batch, on
// another stream, must not touch the descriptors and counters at work.
void failed_launch(cudaStream_t st)
{
    cudaStream_t other;
    check(cudaStreamCreateWithFlags(&other, cudaStreamNonBlocking) == cudaSuccess, "stream");
    for (int round = 0; round < 3; ++round) {
        Batch a, b;
        for (int i = 0; i < 12; ++i) {
            a.add(5000 + 100 * i, 8 + 2 * (i % 2), 0.5f, "");
            b.add(9000 + 300 * i, 9 + 2 * (i % 2), 0.25f, "--half_complex_return");
        }
        a.seal();
        b.seal();
        fake::class_us = 50000;
        fake::fail_class = 1;
        check(a.run(st) != OCS_OK, "a failing launch");
        fake::fail_class = -1;
        fake::class_us = 0;
        check(b.run(other) == OCS_OK, "the next batch");
        cudaStreamSynchronize(st);
        cudaStreamSynchronize(other);
        check(fake::changed_under_work.load() == 0, "descriptors changed under a running class");
        check(b.right(), "outputs of the next batch");
    }
    cudaStreamDestroy(other);
}

// Two batches of the same windows and size whose frames lie in different
// windows: the tile length kept for the first must not stretch the second's.
void tune_key(cudaStream_t st)
{
    setenv("OCS_AUTOTUNE", "1", 1);
    fake::tile_us = 500;  // fewer, longer tiles are much faster: the tuner takes a long one
    const uint64_t many = 2100, few = 20;
    auto longest8 = [&](uint64_t at8, uint64_t at12) {
        Batch b;
        b.add(at8 * 128, 8, 0.5f, "");
        b.add(at12 * 2048, 12, 0.5f, "");
        b.seal();
        check(b.run(st) == OCS_OK, "launch");
        cudaStreamSynchronize(st);
        check(b.right(), "outputs");
        // the classes of the last launch: 2^8, 2^12
        const std::vector<fake::ClassLaunch> l = fake::take_class_launches();
        uint64_t most = 0;
        for (const auto& t : l[l.size() - 2].tiles) most = std::max(most, t.nframes);
        return most;
    };
    // mostly at 2^12, 8 groups make enough tiles: lengths of 8 .. 64 are timed
    longest8(few, many);
    // mostly at 2^8, they do not, and the lengths are 1 .. 8, whatever the first batch kept
    check(longest8(many, few) <= (uint64_t)ocs::batch_tile_frames(8, 8), "the second batch's tiles");
    fake::tile_us = 0;
}

}  // namespace

int main(int argc, char** argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    setenv("OCS_AUTOTUNE", "0", 1);
    check(ocs_init(0) == OCS_OK, "init");
    cudaStream_t st;
    check(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess, "stream");
    if (what == "classes") classes(st);
    else if (what == "one_request") one_request(st);
    else if (what == "failed_launch") failed_launch(st);
    else if (what == "tune_key") tune_key(st);
    else check(false, "unknown check");
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    std::printf("ok %s\n", what.c_str());
    return 0;
}

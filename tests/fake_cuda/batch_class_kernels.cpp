// TEST INFRASTRUCTURE ONLY: the stand-in kernels of fake_kernels.cpp with the
// real kernels' present answers (which kernel takes which window) and with a
// batch launch that works class by class from batch_classes(), as the real one
// does: one unit of stream work per class, with that class's queue counter.  The
// launch of a class can be made to fail, and each class can take some time.
#include "cuda_runtime.h"
#include "fake_control.h"
#include "ocs_kernels.h"

#include "batch_class_control.h"

#include <chrono>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>

// the other stand-ins, with the ones replaced below under other names
#define launch_batch launch_batch_one
#define pair_has pair_has_any
#define pair_twiddle_count pair_twiddle_count_any
#define build_pair_twiddles build_pair_twiddles_any
#define pairx2_has pairx2_has_any
#define pairx2_per_cta pairx2_per_cta_any
#define launch_pairx2 launch_pairx2_any
#define tpf_has tpf_has_any
#define batch_tile_frames batch_tile_frames_any
#include "fake_kernels.cpp"
#undef launch_batch
#undef pair_has
#undef pair_twiddle_count
#undef build_pair_twiddles
#undef pairx2_has
#undef pairx2_per_cta
#undef launch_pairx2
#undef tpf_has
#undef batch_tile_frames

namespace fake {
std::atomic<int> fail_class{-1};
std::atomic<int> class_us{0};
std::atomic<int> tile_us{0};
std::atomic<long> changed_under_work{0};
namespace {
std::mutex g_mu;
std::map<const void*, int> g_plans;
std::vector<ClassLaunch> g_launches;
}  // namespace
int plan_of(const void* table)
{
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_plans.find(table);
    return it == g_plans.end() ? -1 : it->second;
}
std::vector<ClassLaunch> take_class_launches()
{
    std::lock_guard<std::mutex> lk(g_mu);
    std::vector<ClassLaunch> r;
    r.swap(g_launches);
    return r;
}
}  // namespace fake

namespace ocs {

bool pair_has(int exp) { return exp == 6 || (exp >= 8 && exp <= 10); }
bool tpf_has(int exp, int outk) { return outk == OUT_HALF ? exp == 6 : (exp >= 6 && exp <= 8); }
bool pairx2_has(int exp, int outk) { return exp >= 12 && exp <= 15 && outk != OUT_PLANES; }
int pairx2_per_cta(int exp) { return exp == 12 ? 2 : 1; }
int pair_twiddle_count(int pid) { return pid & kMirrorPlan ? 64 : 1 << (pid & 31); }
cudaError_t build_pair_twiddles(float2* tw, int pid, cudaStream_t)
{
    std::lock_guard<std::mutex> lk(fake::g_mu);
    fake::g_plans[tw] = pid;
    return cudaSuccess;
}
cudaError_t launch_pairx2(int exp, int outk, const FusedArgs& a, int grid, cudaStream_t st)
{
    if (grid < 1 || fake::plan_of(a.tw) != mirror_plan_id(exp, mirror_paired(exp, outk))) return cudaErrorInvalidValue;
    return fused_like(exp, outk, a, st);
}
int batch_tile_frames(int exp, int groups) { return (exp <= 8 ? 4096 >> exp : exp <= 12 ? 8192 >> exp : 2) * groups; }

cudaError_t launch_batch(const FusedArgs* d_reqs, const BatchTile* d_tiles, const uint32_t* d_ntiles,
                         uint32_t* d_counter, int, cudaStream_t st)
{
    const BatchClasses k = batch_classes();
    ++fake::launches;
    for (int i = 0; i < k.count; ++i) {
        if (i == fake::fail_class.load()) return cudaErrorInvalidValue;
        const BatchClasses::Class c = k.cls[i];
        ++fake::kernel_launches;
        fake::enqueue(st, [=] {
            fake::ClassLaunch rec;
            rec.id = c.id;
            rec.begin = c.begin;
            rec.all_tiles = *d_ntiles;
            const std::vector<BatchTile> tiles(d_tiles + c.begin, d_tiles + c.begin + c.tiles);
            std::vector<FusedArgs> reqs;
            for (const BatchTile& t : tiles) reqs.push_back(d_reqs[t.req]);
            const uint32_t first = d_counter[i];
            std::this_thread::sleep_for(
                std::chrono::microseconds(fake::class_us.load() + fake::tile_us.load() * (long)c.tiles));
            for (uint32_t t = first; t < c.tiles; ++t) {
                if (std::memcmp(&tiles[t], &d_tiles[c.begin + t], sizeof(BatchTile)) != 0 ||
                    std::memcmp(&reqs[t], &d_reqs[tiles[t].req], sizeof(FusedArgs)) != 0) {
                    ++fake::changed_under_work;
                    return;
                }
                const FusedArgs& a = reqs[t];
                rec.tiles.push_back({a.exp, a.outk, tiles[t].f0, tiles[t].nframes, a.frames, fake::plan_of(a.tw_pair)});
                for (uint64_t f = tiles[t].f0; f < tiles[t].f0 + tiles[t].nframes; ++f)
                    frame_out(a.x, a.n, a.hop, a.out, a.ohalf, a.dense, a.exp, a.outk, f);
            }
            d_counter[i] = c.tiles;
            std::lock_guard<std::mutex> lk(fake::g_mu);
            fake::g_launches.push_back(rec);
        });
    }
    return cudaSuccess;
}

}  // namespace ocs

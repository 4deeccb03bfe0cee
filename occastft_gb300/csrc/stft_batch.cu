// Uneven batches: the launches of one batch, and the kernels of windows 2^6 .. 2^9.
#include "stft_batch_kernel.cuh"

#include <algorithm>

namespace ocs {

size_t batch_smem_bytes() { return batch_smem(0); }
bool batch_supports(int exp) { return exp >= kBatchMinExp && exp <= kBatchMaxExp; }
// `groups` groups of frames, a group being what a CTA of the one-frame kernel
// holds (two frames at 2^13, as the mirror-group body).  The host's autotuner
// picks the count per batch mix, a power of two, and makes a tile no shorter than
// batch_min_frames, so that tiles are whole rounds of every body and start on
// whole pairs of frames.
int batch_tile_frames(int exp, int groups) { return (exp == 13 ? 2 : fused_fpc(exp)) * groups; }

static_assert(batch_min_frames(7, OUT_POWER) == 8 * TplCfg<7>::F && batch_min_frames(8, OUT_POWER) == 8 * TplCfg<8>::F,
              "a round of the lanes-per-frame bodies");
static_assert(batch_min_frames(9, OUT_POWER) == 2 * pair_ppc(9) && batch_min_frames(10, OUT_POWER) == 2 * pair_ppc(10),
              "a round of the paired bodies");
static_assert(batch_min_frames(12, OUT_POWER) == 2 * mirror_gpc(mirror_lp(12, true)) &&
                  batch_min_frames(12, OUT_HALF) == mirror_gpc(mirror_lp(12, false)) &&
                  batch_min_frames(13, OUT_HALF) == mirror_gpc(mirror_lp(13, false)),
              "a round of the mirror-group bodies");
static_assert(batch_min_frames(6, OUT_HALF) % fused_fpc(6) == 0 && batch_min_frames(7, OUT_HALF) % fused_fpc(7) == 0 &&
                  batch_min_frames(8, OUT_HALF) % fused_fpc(8) == 0 && batch_min_frames(9, OUT_HALF) % fused_fpc(9) == 0 &&
                  batch_min_frames(10, OUT_HALF) % fused_fpc(10) == 0 &&
                  fused_fpc(11) % batch_min_frames(11, OUT_POWER) == 0,
              "whole rounds of the one-frame bodies");

int batch_occupancy()
{
    const int lo = std::min(std::min(batch_occupancy_t<6>(), batch_occupancy_t<7>()),
                            std::min(batch_occupancy_t<8>(), batch_occupancy_t<9>()));
    return std::min(std::min(lo, batch_occupancy_hi()), batch_occupancy_all());
}

static cudaError_t launch_one(int cls, const FusedArgs* reqs, const BatchTile* tiles, uint32_t nt, uint32_t* counter,
                              int grid, bool first, cudaStream_t st)
{
    switch (cls) {
    case 6: return launch_batch_t<6>(reqs, tiles, nt, counter, grid, first, st);
    case 7: return launch_batch_t<7>(reqs, tiles, nt, counter, grid, first, st);
    case 8: return launch_batch_t<8>(reqs, tiles, nt, counter, grid, first, st);
    case 9: return launch_batch_t<9>(reqs, tiles, nt, counter, grid, first, st);
    default: return launch_batch_hi(cls, reqs, tiles, nt, counter, grid, first, st);
    }
}

cudaError_t launch_batch(const FusedArgs* d_reqs, const BatchTile* d_tiles, const uint32_t*, uint32_t* d_counter,
                         int grid, cudaStream_t st)
{
    const BatchClasses& k = batch_classes();
    uint32_t tiles = 0;
    for (int i = 0; i < k.count; ++i) tiles += k.cls[i].tiles;
    // up to four tiles per CTA: one launch for all window sizes
    if (k.count > 1 && tiles <= 4 * (uint32_t)grid)
        return launch_batch_all(d_reqs, d_tiles, tiles, d_counter, grid, st);
    for (int i = 0; i < k.count; ++i) {
        const BatchClasses::Class& c = k.cls[i];
        const cudaError_t e = launch_one(c.id, d_reqs, d_tiles + c.begin, c.tiles, d_counter + i,
                                         (int)std::min<uint32_t>((uint32_t)grid, c.tiles), i == 0, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ocs

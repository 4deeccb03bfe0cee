// Batch kernels of windows 2^10 .. 2^13 (2^12 in two forms).
#include "stft_batch_kernel.cuh"

#include <algorithm>

namespace ocs {

int batch_occupancy_hi()
{
    return std::min(std::min(batch_occupancy_t<10>(), batch_occupancy_t<11>()),
                    std::min(std::min(batch_occupancy_t<12>(), batch_occupancy_t<kBatchSingle12>()),
                             batch_occupancy_t<13>()));
}

cudaError_t launch_batch_hi(int cls, const FusedArgs* reqs, const BatchTile* tiles, uint32_t nt, uint32_t* counter,
                            int grid, bool first, cudaStream_t st)
{
    switch (cls) {
    case 10: return launch_batch_t<10>(reqs, tiles, nt, counter, grid, first, st);
    case 11: return launch_batch_t<11>(reqs, tiles, nt, counter, grid, first, st);
    case 12: return launch_batch_t<12>(reqs, tiles, nt, counter, grid, first, st);
    case kBatchSingle12: return launch_batch_t<kBatchSingle12>(reqs, tiles, nt, counter, grid, first, st);
    case 13: return launch_batch_t<13>(reqs, tiles, nt, counter, grid, first, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace ocs

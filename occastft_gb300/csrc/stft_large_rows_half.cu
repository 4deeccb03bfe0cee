// The half-complex row pass of 1024 points (windows 2^21, 2^22 and 2^24 up) on
// scalar complex arithmetic: packed, it is slower, the other passes faster.
// 3e7 samples, overlap 0.5 / 0.75, packed -> scalar: 2^21 214.7 / 365 -> 209.6 /
// 348 us, 2^22 232.7 / 406 -> 229.7 / 397 (all passes scalar: 2^21 217.6 / 371).
#define OCS_SCALAR_COMPLEX
#include "stft_large_rows.cuh"

namespace ocs {

cudaError_t launch_rows_half_11(const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    return launch_rows_t<11, OUT_HALF>(a, frames, st);
}

}  // namespace ocs

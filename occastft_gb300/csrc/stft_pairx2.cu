// The mirror-group STFT kernel's dispatch over window exponents; the
// instantiations are in stft_mirror_lo.cu and stft_mirror_hi.cu.
#include "stft_mirror_kernel.cuh"

namespace ocs {

bool pairx2_has(int exp, int outk) { return mirror_supported(exp) && outk != OUT_PLANES; }
static_assert(mirror_gpc(mirror_lp(12, false)) == 2 * mirror_gpc(mirror_lp(12, true)) &&
                  mirror_gpc(mirror_lp(13, false)) == 2 * mirror_gpc(mirror_lp(13, true)),
              "a CTA holds as many frames in either form");
int pairx2_per_cta(int exp) { return mirror_gpc(mirror_lp(exp, exp <= 13)); }

cudaError_t launch_pairx2(int exp, int outk, const FusedArgs& a, int grid, cudaStream_t st)
{
    if (!pairx2_has(exp, outk)) return cudaErrorInvalidValue;
    return exp <= 13 ? launch_mirror_lo(exp, outk, a, grid, st) : launch_mirror_hi(exp, outk, a, grid, st);
}

int pairx2_occupancy(int exp, int outk)
{
    if (!pairx2_has(exp, outk)) return 0;
    return exp <= 13 ? occupancy_mirror_lo(exp, outk) : occupancy_mirror_hi(exp, outk);
}

}  // namespace ocs

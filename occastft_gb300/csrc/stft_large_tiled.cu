// Instantiations and launch of the tiled two-launch kernels (windows 2^16 .. 2^19).
#include "stft_large_tiled.cuh"

namespace ocs {
namespace {

// Requests of a few frames, whose two grids and the next request's find an SM for
// each CTA (half of 152 for one request), overlap each pass's launch with the pass
// before (launch_pdl): one frame, power / half-complex, 2^16 12.4 / 14.4 -> 9.1 /
// 10.8 us, 2^18 18.1 / 20.2 -> 12.5 / 14.4 (the untiled passes: 18.9 / 18.8).
// Beyond that CTAs share SMs while others are free (2^17, 7 frames and 88 CTAs 18.8
// -> 19.8 us), and long requests lose the room (2^18, 1e8 samples, 532 -> 540 us).
constexpr uint64_t kOverlapCtas = 76;
template <typename... P>
cudaError_t launch_pass(bool overlap, void (*kernel)(P...), uint64_t grid, int threads, size_t smem, cudaStream_t st,
                        const LargeArgs& a)
{
    if (overlap) return launch_pdl(kernel, (int)grid, threads, smem, st, a);
    kernel<<<(unsigned)grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}
template <int L1>
uint64_t cols_grid(const LargeArgs& a, uint64_t frames)
{
    using C = LtCol<L1>;
    return (frames + C::FPC - 1) / C::FPC * (a.m2 / C::TC);
}
uint64_t rows_grid(const LargeArgs& a, uint64_t frames) { return frames * (a.m1 / (2 * kLtTile)); }

template <int L1>
cudaError_t launch_cols_t(const LargeArgs& a, uint64_t frames, cudaStream_t st, bool* overlap)
{
    using C = LtCol<L1>;
    const cudaError_t e = ensure_smem_attr<large_tiled_columns_kernel<L1>>(C::SMEM);
    if (e != cudaSuccess) return e;
    LargeArgs b = a;
    b.frames_launch = frames;
    const uint64_t grid = cols_grid<L1>(a, frames);
    *overlap = grid + rows_grid(a, frames) <= kOverlapCtas;
    return launch_pass(*overlap, large_tiled_columns_kernel<L1>, grid, 256, C::SMEM, st, b);
}

template <int L2, int OUTK>
cudaError_t launch_rows_t(const LargeArgs& a, uint64_t frames, cudaStream_t st, bool overlap)
{
    using R = LtRow<L2>;
    const cudaError_t e = ensure_smem_attr<large_tiled_rows_kernel<L2, OUTK>>(R::SMEM);
    if (e != cudaSuccess) return e;
    return launch_pass(overlap, large_tiled_rows_kernel<L2, OUTK>, rows_grid(a, frames), R::THREADS, R::SMEM, st, a);
}

template <int L2>
cudaError_t launch_rows_e(int outk, const LargeArgs& a, uint64_t frames, cudaStream_t st, bool overlap)
{
    switch (outk) {
    case OUT_POWER: return launch_rows_t<L2, OUT_POWER>(a, frames, st, overlap);
    case OUT_POWER_SERIAL: return launch_rows_t<L2, OUT_POWER_SERIAL>(a, frames, st, overlap);
    case OUT_HALF: return launch_rows_t<L2, OUT_HALF>(a, frames, st, overlap);
    case OUT_PLANES: return launch_rows_t<L2, OUT_PLANES>(a, frames, st, overlap);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// M1 = 2^l1, M2 = 2^l2
cudaError_t launch_large_tiled(int l1, int l2, int outk, const LargeArgs& args, uint64_t frames, cudaStream_t st)
{
    LargeArgs a = args;
    a.m1 = 1ull << l1;
    a.m2 = 1ull << l2;
    bool overlap = false;
    cudaError_t e = cudaErrorInvalidValue;
    switch (l1) {
    case 8: e = launch_cols_t<8>(a, frames, st, &overlap); break;
    case 9: e = launch_cols_t<9>(a, frames, st, &overlap); break;
    case 10: e = launch_cols_t<10>(a, frames, st, &overlap); break;
    default: break;
    }
    if (e != cudaSuccess) return e;
    switch (l2) {
    case 7: return launch_rows_e<7>(outk, a, frames, st, overlap);
    case 8: return launch_rows_e<8>(outk, a, frames, st, overlap);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace ocs

// Row pass of the untiled four-step FFT (stft_large.cu): the kernel and its
// launch, for the two translation units that hold its instantiations.
#pragma once
#include "stft_fused_kernel.cuh"

namespace ocs {
namespace {

constexpr int kTileR = 8;  // rows (and as many mirror rows) per row-pass CTA

// Row-pass buffers: row r starts at r * large_row_stride + large_row_shift(r),
// the stride a multiple of 16 float2 and the shift 0, 8, 4, 12, 2, 10, 6, 14
// for r mod 8, so that the output loop's reads of 8 rows at 4 consecutive
// columns tile the 16 bank pairs twice.
__host__ __device__ constexpr int large_row_stride(int exp2) { return (fused_buf_stride(exp2) + 14 + 15) / 16 * 16; }
__device__ __forceinline__ int large_row_shift(int r) { return 8 * (r & 1) + 4 * ((r >> 1) & 1) + 2 * ((r >> 2) & 1); }

// exp(-2 pi i j / L) from a two-level table: lo[j & 1023] * hi[j >> 10]
__device__ __forceinline__ float2 tw2l(const float2* lo, const float2* hi, uint64_t j)
{
    return cmul(lo[j & 1023u], hi[j >> 10]);
}

// ---------------------------------------------------------------- row pass
template <int EXP2, int OUTK>
__global__ void __launch_bounds__(2 * kTileR * (fused_M(EXP2) / fused_cfg(EXP2).R))
    large_rows_kernel(const LargeArgs a)
{
    using K = Core<EXP2>;
    constexpr int M2 = K::M, R = K::R, T = K::T;
    constexpr int BS = large_row_stride(EXP2);
    extern __shared__ float2 sbuf[];  // 2*kTileR row buffers (large_row_stride / large_row_shift)
    const int tid = threadIdx.x;
    const uint64_t M1 = a.m1;
    const uint64_t M = M1 * M2;
    const uint64_t N = 2 * M;
    const uint64_t blocks = M1 / (2 * kTileR);
    const uint64_t fl = blockIdx.x / blocks;
    const uint64_t b = blockIdx.x % blocks;
    const uint64_t f = a.f0 + fl;

    // slot s < kTileR: row b*8 + s; slot kTileR + s: its mirror M1 - row,
    // except that row 0's mirror slot holds row M1/2
    auto row_of = [&](int s) -> uint64_t {
        const uint64_t d = b * kTileR + (uint64_t)(s % kTileR);
        if (s < kTileR) return d;
        return d == 0 ? M1 / 2 : M1 - d;
    };
    const int rs = tid / T, t = tid % T;
    const float2* y = a.scratch + fl * M;
    float2* buf = sbuf + rs * BS + large_row_shift(rs);
    {
        const float2* yr = y + row_of(rs) * M2;
        float2 v[R];
#pragma unroll
        for (int u = 0; u < R; ++u) v[u] = yr[t + u * T];
        K::fft(v, buf, a.tw2, t);  // slot u: Z[k1 + M1 (t + u T)]
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R; ++u) buf[K::pd(t + u * T)] = v[u];
    }
    __syncthreads();
    if (f >= a.frames_total) return;

    // outputs: lanes over the 8 rows of a slot group, then over k2.  Thread
    // tid keeps slot (tid & 7) of each group (first the rows, then their
    // mirrors) and steps k2 by 16, so everything that depends on the slot is
    // formed once per group.
    const bool dc = a.remove_dc != 0;
    const uint32_t m1 = (uint32_t)M1, m2 = (uint32_t)M2;
    if constexpr (OUTK == OUT_POWER || OUTK == OUT_POWER_SERIAL) {
        // Power: one untangle at k gives X[k] and X[M + k], and for a real
        // frame |X[N - k]| = |X[k]|, |X[M - k]| = |X[M + k]|, so only the 8
        // rows are untangled and their mirrors (which hold the partners)
        // come for free.  Row 0 pairs with itself (k2 with M2 - k2) and so
        // does row M1/2 (k2 with M2 - 1 - k2): the first CTA's slot 0 takes
        // row 0 for k2 < M2/2, row M1/2 for the other half, and k = M/2 last.
        const int s = tid & (kTileR - 1);
        const bool special = b == 0 && s == 0;
        const uint32_t k1 = (uint32_t)row_of(s);
        const float2* zs = sbuf + s * BS + large_row_shift(s);
        const float2* zp = sbuf + (s + kTileR) * BS + large_row_shift(s + kTileR);
        const float2 wk1 = special ? tw2l(a.twn_lo, a.twn_hi, m1 / 2) : tw2l(a.twn_lo, a.twn_hi, k1);
        float* ro = a.out + f * (a.dense ? M + 1 : N);
        auto emit = [&](uint32_t k, float2 A, float2 B, float2 w) {
            float2 ev, wo;
            K::untangle(A, B, w, ev, wo);
            float2 X0 = make_float2(ev.x + wo.x, ev.y + wo.y);        // X[k]
            const float2 X1 = make_float2(ev.x - wo.x, ev.y - wo.y);  // X[k + M]
            if (dc && k == 0) X0 = make_float2(0.0f, 0.0f);
            const float p0 = power_of<OUTK>(X0), p1 = power_of<OUTK>(X1);
            const bool mirror = k != 0 && k != (uint32_t)(M / 2);
            if (!a.dense) {
                __stcs(ro + k, p0);
                __stcs(ro + (k + M), p1);
                if (mirror) {
                    __stcs(ro + (N - k), p0);
                    __stcs(ro + (M - k), p1);
                }
            } else {
                __stcs(ro + k, p0);
                if (mirror) __stcs(ro + (M - k), p1);
                if (k == 0) __stcs(ro + M, p1);
            }
        };
        if (!special) {
#pragma unroll 2
            for (uint32_t k2 = (uint32_t)tid / kTileR; k2 < m2; k2 += blockDim.x / kTileR)
                emit(k1 + m1 * k2, zs[K::pd((int)k2)], zp[K::pd((int)(m2 - 1 - k2))], cmul(wk1, a.tw2[k2]));
        } else {
            for (uint32_t k2 = (uint32_t)tid / kTileR; k2 < m2; k2 += blockDim.x / kTileR) {
                if (k2 < m2 / 2) {
                    emit(m1 * k2, zs[K::pd((int)k2)], zs[K::pd((int)((m2 - k2) & (m2 - 1)))], a.tw2[k2]);
                } else {
                    const uint32_t hk = k2 - m2 / 2;  // row M1/2 sits in slot kTileR
                    emit(m1 / 2 + m1 * hk, zp[K::pd((int)hk)], zp[K::pd((int)(m2 - 1 - hk))], cmul(wk1, a.tw2[hk]));
                }
            }
            if (tid == 0) {
                const float2 A = zs[K::pd((int)(m2 / 2))];
                emit((uint32_t)(M / 2), A, A, a.tw2[m2 / 2]);
            }
        }
    } else {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int s = (tid & (kTileR - 1)) + kTileR * h;
        const uint32_t k1 = (uint32_t)row_of(s);
        // partner Z[M - k]: row (M1 - k1) mod M1; column M2-1-k2, or (M2-k2) mod M2 for row 0
        const int ps = (k1 == 0 || k1 == m1 / 2) ? s : (s < kTileR ? s + kTileR : s - kTileR);
        const bool row0 = k1 == 0;
        const float2* zs = sbuf + s * BS + large_row_shift(s);
        const float2* zp = sbuf + ps * BS + large_row_shift(ps);
        // W_N^k for k = k1 + M1 k2: W_N^{k1} W_{2 M2}^{k2}; the second factor
        // is the untangle table of the M2-point plan (its first M2 entries)
        const float2 wk1 = tw2l(a.twn_lo, a.twn_hi, k1);
        float* ro = a.out + f * N;
        float* rod = a.out + f * (M + 1);
        float2* o2 = reinterpret_cast<float2*>(a.out);
#pragma unroll 2
        for (uint32_t k2 = (uint32_t)tid / kTileR; k2 < m2; k2 += blockDim.x / kTileR) {
            const uint32_t pk2 = row0 ? ((m2 - k2) & (m2 - 1)) : (m2 - 1 - k2);
            const float2 A = zs[K::pd((int)k2)];
            const float2 B = zp[K::pd((int)pk2)];
            const uint32_t k = k1 + m1 * k2;
            float2 ev, wo;
            K::untangle(A, B, cmul(wk1, a.tw2[k2]), ev, wo);
            float2 X0 = make_float2(ev.x + wo.x, ev.y + wo.y);        // X[k]
            const float2 X1 = make_float2(ev.x - wo.x, ev.y - wo.y);  // X[k + M]
            if (dc && k == 0) X0 = make_float2(0.0f, 0.0f);
            if constexpr (OUTK == OUT_PLANES) {
                a.out[f * N + k] = X0.x;
                a.out_im[f * N + k] = X0.y;
                a.out[f * N + k + M] = X1.x;
                a.out_im[f * N + k + M] = X1.y;
            } else if constexpr (OUTK == OUT_HALF) {
                if (!a.dense) {
                    const uint64_t flat = f * N + k;
                    if (flat < a.ohalf) __stcs(o2 + flat, X0);
                    if (flat + M < a.ohalf) __stcs(o2 + flat + M, X1);
                } else {
                    float2* rc = o2 + f * (M + 1);
                    __stcs(rc + k, X0);
                    if (k == 0) __stcs(rc + M, X1);
                }
            } else {
                const float p0 = power_of<OUTK>(X0), p1 = power_of<OUTK>(X1);
                if (!a.dense) {
                    __stcs(ro + k, p0);
                    __stcs(ro + k + M, p1);
                } else {
                    __stcs(rod + k, p0);
                    if (k == 0) __stcs(rod + M, p1);
                }
            }
        }
    }
    }
}

template <int EXP2, int OUTK>
cudaError_t launch_rows_t(const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    constexpr int T = fused_M(EXP2) / fused_cfg(EXP2).R;
    constexpr size_t smem = (size_t)2 * kTileR * large_row_stride(EXP2) * sizeof(float2);
    auto k = large_rows_kernel<EXP2, OUTK>;
    const cudaError_t e = ensure_smem_attr<large_rows_kernel<EXP2, OUTK>>(smem);
    if (e != cudaSuccess) return e;
    const uint64_t grid = frames * (a.m1 / (2 * kTileR));
    k<<<(unsigned)grid, 2 * kTileR * T, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace
}  // namespace ocs

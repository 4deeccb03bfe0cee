// STFT for windows 2^16 .. 2^30 (sm_103a): a four-step FFT in two launches
// up to 2^22, three above.  Windows 2^16 .. 2^19 run the tiled passes of
// stft_large_tiled.cuh; the ones here take 2^20 and up.  The scratch of all of
// them, and the chunks a request is cut into, are at the end of this file.
//
// One frame of N real samples is the M = N/2 point complex FFT of
// z[m] = y[2m] + i y[2m+1] plus the real-input untangle, as in the fused
// kernels; here M = M1 * M2 does not fit one CTA, so with m = c + M2 m1 and
// k = k1 + M1 k2:
//   column pass  Y[k1][c]  = W_M^{c k1} * sum_{m1} z[c + M2 m1] W_{M1}^{m1 k1}
//   row pass     Z[k1 + M1 k2] = sum_c Y[k1][c] W_{M2}^{c k2}
// followed by X[k] = (Z[k] + conj Z[M-k]) + W_N^k (Z[k] - conj Z[M-k]) / i and
// X[k + M] = (Z[k] + conj Z[M-k]) - W_N^k (...) (the window table carries the
// untangle's factor 1/2).
//
// Column pass: a CTA owns 16 (columns of 256 points) or 8 consecutive columns
// of one frame.  It reads the frame's samples row by row (128 or 64
// contiguous bytes per row), applies the
// window, runs 8 M1-point FFTs with the fused kernels' Stockham core, applies
// W_M^{c k1} and writes Y row-major to a scratch area (again 64-byte rows).
// Row pass: a CTA owns 8 rows k1 and their 8 mirror rows M1 - k1 (row M1/2
// stands in for the mirror of row 0), so every Z[M-k] it needs is its own.
// It runs 16 M2-point FFTs, then writes outputs with lanes over k1, i.e. 8
// consecutive bins per (k2) run.
//
// Above 2^22 the column FFT would exceed a CTA, so M = P1 * P2 * Q and the
// column length P = P1 * P2 splits once more (m = c + Q (a + P2 m1),
// k1 = k1a + P1 k1b):
//   column pass  U[k1a][c + Q a] = W_P^{a k1a} sum_{m1} z[c + Q a + Q P2 m1] W_{P1}^{m1 k1a}
//   middle pass  Y[k1a + P1 k1b][c] = W_M^{c k1} sum_a U[k1a][c + Q a] W_{P2}^{a k1b}
//   row pass     as above, over P rows of Q points.
// The column pass is the two-launch column pass with Q P2 columns and the
// twiddle exponent taken from the column's block (c + Q a) & ~(Q - 1) = Q a,
// since W_P^{a k1a} = W_M^{Q a k1a}.
//
// DC removal subtracts the mean of the windowed frame; in the transform that
// changes bin 0 only (to zero), which is what the row pass writes.  The
// reference's EXPC runs any exponent >= 12 through a radix-2 Stockham
// (RunnerCommon.cpp:278-289, Serial/src/functionImpl.cpp:186-270).
#include "stft_large_rows.cuh"

#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>

namespace ocs {
cudaError_t launch_rows_half_11(const LargeArgs& a, uint64_t frames, cudaStream_t st);  // stft_large_rows_half.cu

namespace {

constexpr int kTileC = 8;  // columns per middle-pass CTA (column pass: large_col_tile)
// Column-pass buffer stride: = 2 (mod 8) float2.  An 8-byte shared access is
// served per half-warp; in the staging loops a half-warp is 4 rows x 4 lanes,
// lane q on columns 2q and 2q+1, so the columns must start 4 bank pairs
// apart for the 16 lanes to hit 16 distinct ones (with = 4 (mod 8) lanes q
// and q + 2 collided: 2.9 wavefronts per load where 2 are needed).
__host__ __device__ constexpr int large_col_stride(int exp1)
{
    return fused_buf_stride(exp1) + ((2 - fused_buf_stride(exp1) % 8) + 8) % 8;
}
__host__ __device__ constexpr int large_l1(int exp) { return exp / 2; }         // log2 M1
__host__ __device__ constexpr int large_l2(int exp) { return exp - 1 - exp / 2; }  // log2 M2

// ---------------------------------------------------------------- column pass
// Column FFTs of up to 512 points (windows 2^23 .. 2^29) keep the CTA's
// window coefficients in registers and take 4 consecutive frames of the same
// columns per CTA; the larger ones (more chunks per thread, or 1024 threads
// at 64 registers) take one frame per CTA and read the window each time.
//
// A CTA owns 16 columns (rows of 128 bytes, 8 lanes per row) where that keeps
// it at 256 threads (column FFTs of 256 points, windows 2^23 .. 2^27), else
// 8: each warp-wide row load then touches half as many cache lines.
__host__ __device__ constexpr int large_col_tile(int exp1)
{
    return 16 * (fused_M(exp1) / fused_cfg(exp1).R) <= 256 ? 16 : 8;
}
// Its buffer stride: with 16 columns an odd number of float2, so that a
// half-warp's 8-byte staging accesses (2 rows x 8 lanes, lane q on columns 2q
// and 2q + 1) land on 16 distinct bank pairs; with 8 columns the stride of
// the middle pass.
__host__ __device__ constexpr int large_col_stride_t(int exp1, int tc)
{
    return tc == 16 ? (fused_buf_stride(exp1) | 1) : large_col_stride(exp1);
}
__host__ __device__ constexpr bool large_col_cache_win(int exp1)
{
    return fused_M(exp1) / (2 * (fused_M(exp1) / fused_cfg(exp1).R)) <= 8 &&
           large_col_tile(exp1) * (fused_M(exp1) / fused_cfg(exp1).R) <= 256;
}
__host__ __device__ constexpr int large_col_frames(int exp1) { return large_col_cache_win(exp1) ? 4 : 1; }

// four window coefficients at real index i (a multiple of 4); no table: 1/2
__device__ __forceinline__ float4 large_win4(const float* win, uint32_t i)
{
    return win ? *reinterpret_cast<const float4*>(win + i) : make_float4(0.5f, 0.5f, 0.5f, 0.5f);
}

template <int EXP1>
__global__ void __launch_bounds__(large_col_tile(EXP1) * (fused_M(EXP1) / fused_cfg(EXP1).R))
    large_columns_kernel(const LargeArgs a)
{
    using K = Core<EXP1>;
    constexpr int M1 = K::M, R = K::R, T = K::T;
    constexpr int TC = large_col_tile(EXP1);  // columns
    constexpr int QR = TC / 2;                // float4 chunks per row
    constexpr int NT = TC * T;                // threads
    constexpr int NE = M1 * QR / NT;          // float4 row chunks per thread (= R / 2)
    constexpr int BS = large_col_stride_t(EXP1, TC);
    extern __shared__ float2 sbuf[];  // TC column buffers of BS slots
    const int tid = threadIdx.x;
    const uint64_t M2 = a.m2;
    const uint64_t tiles = M2 / TC;
    const uint64_t fg = blockIdx.x / tiles;  // group of FPC frames within this launch
    const uint64_t c0 = (blockIdx.x % tiles) * TC;
    const uint64_t N = 2 * (uint64_t)M1 * M2;
    const bool aligned = (a.hop & 3) == 0 && (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;
    // this CTA's window coefficients: chunk j is row m1 = e / QR, columns 2q,
    // 2q+1 (q = e % QR) with e = tid + j NT; row m1 starts at real index
    // 2 (c0 + M2 m1), a multiple of 16
    constexpr bool CACHE_WIN = large_col_cache_win(EXP1);
    constexpr int FPC = large_col_frames(EXP1);
    float4 wv[CACHE_WIN ? NE : 1];
    if constexpr (CACHE_WIN) {
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const int e = tid + j * NT, m1 = e / QR, q = e % QR;
            wv[j] = large_win4(a.win, 2u * ((uint32_t)c0 + (uint32_t)M2 * (uint32_t)m1) + 4u * (uint32_t)q);
        }
    }
    const int col = tid / T, t = tid % T;
    float2* buf = sbuf + col * BS;
    const uint64_t c = c0 + col;

#pragma unroll 1
    for (int ff = 0; ff < FPC; ++ff) {
        const uint64_t fl = fg * FPC + ff;  // frame within this launch
        if (fl >= a.frames_launch) break;
        const uint64_t f = a.f0 + fl;
        const uint64_t s0 = f * a.hop;
        if (ff > 0) __syncthreads();  // the previous frame's reads of the buffers are over
        // rows of TC complex samples (64 or 128 bytes)
        if (aligned && f < a.frames_total && s0 + N <= a.n) {
            // frame inside the signal and 16-byte aligned: QR threads per
            // row, a float4 (two complex samples) each
            const float* xf = a.x + s0;
            auto chunk = [&](int e, const float4& w) {
                const int m1 = e / QR, q = e % QR;
                const uint32_t i = 2u * ((uint32_t)c0 + (uint32_t)M2 * (uint32_t)m1) + 4u * (uint32_t)q;
                const float4 xv = *reinterpret_cast<const float4*>(xf + i);
                sbuf[(2 * q) * BS + K::pd(m1)] = make_float2(xv.x * w.x, xv.y * w.y);
                sbuf[(2 * q + 1) * BS + K::pd(m1)] = make_float2(xv.z * w.z, xv.w * w.w);
            };
            if constexpr (CACHE_WIN) {
#pragma unroll
                for (int j = 0; j < NE; ++j) chunk(tid + j * NT, wv[j]);
            } else {
                for (int e = tid; e < M1 * QR; e += NT) {
                    const uint32_t i = 2u * ((uint32_t)c0 + (uint32_t)M2 * (uint32_t)(e / QR)) + 4u * (uint32_t)(e % QR);
                    chunk(e, large_win4(a.win, i));
                }
            }
        } else {
            // lane pairs take one row, samples past the signal end read as zero
            for (int e = tid; e < M1 * TC; e += NT) {
                const int cc = e % TC, m1 = e / TC;
                const uint64_t m = c0 + cc + M2 * (uint64_t)m1;  // complex index in the frame
                const uint64_t i = 2 * m;                         // real sample index in the frame
                const uint64_t g = s0 + i;
                float xr = 0.0f, xi = 0.0f;
                if (f < a.frames_total) {
                    if (g < a.n) xr = a.x[g];
                    if (g + 1 < a.n) xi = a.x[g + 1];
                }
                const float2 w = a.win ? *reinterpret_cast<const float2*>(a.win + i) : make_float2(0.5f, 0.5f);
                sbuf[cc * BS + K::pd(m1)] = make_float2(xr * w.x, xi * w.y);
            }
        }
        __syncthreads();
        float2 v[R];
#pragma unroll
        for (int u = 0; u < R; ++u) v[u] = buf[K::pd(t + u * T)];
        K::fft(v, buf, a.tw1, t);  // slot u holds column FFT bin k1 = t + u*T
        __syncthreads();
        // W_M^{c k1}, k1 = t + u T: a two-level lookup at u = 0 and 8, then
        // products with W_M^{c T} (at most 7 rounding steps)
        const uint64_t ce = c & a.col_mask;  // c, or the block Q a of the three-pass form
        const float2 step = tw2l(a.twm_lo, a.twm_hi, ce * (uint64_t)T);
        float2 w = make_float2(1.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int k1 = t + u * T;
            w = (u % 8 == 0) ? tw2l(a.twm_lo, a.twm_hi, ce * (uint64_t)k1) : cmul(w, step);
            buf[K::pd(k1)] = cmul(v[u], w);
        }
        __syncthreads();
        // Y row-major: row k1 holds this CTA's TC columns at c0 (64 or 128
        // bytes), written as QR float4 (two complex values) per row
        float2* y = a.scratch + fl * (uint64_t)M1 * M2;
        for (int e = tid; e < M1 * QR; e += NT) {
            const int k1 = e / QR, q = e % QR;
            const float2 lo = sbuf[(2 * q) * BS + K::pd(k1)], hi = sbuf[(2 * q + 1) * BS + K::pd(k1)];
            *reinterpret_cast<float4*>(y + (uint64_t)k1 * M2 + c0 + 2 * q) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    }
}

// ---------------------------------------------------------------- middle pass
// Three-pass form: a CTA owns 8 consecutive columns c of block k1a of one
// frame.  It reads rows a (P2 of them, 8 complex values = 64 bytes each, at
// U + k1a Q P2 + Q a + c0), runs 8 P2-point FFTs on the Stockham core,
// multiplies W_M^{c (k1a + P1 k1b)} and writes rows k1a + P1 k1b of Y.
// Per launch: m1 = P1, m2 = Q, scratch = U, scratch2 = Y.
template <int EXPM>
__global__ void __launch_bounds__(kTileC * (fused_M(EXPM) / fused_cfg(EXPM).R))
    large_middle_kernel(const LargeArgs a)
{
    using K = Core<EXPM>;
    constexpr int P2 = K::M, R = K::R, T = K::T;
    constexpr int NT = kTileC * T;
    constexpr int BS = large_col_stride(EXPM);
    extern __shared__ float2 sbuf[];
    const int tid = threadIdx.x;
    const uint64_t P1 = a.m1, Q = a.m2;
    const uint64_t M = P1 * (uint64_t)P2 * Q;
    const uint64_t ctiles = Q / kTileC;
    const uint64_t c0 = (blockIdx.x % ctiles) * kTileC;
    const uint64_t k1a = (blockIdx.x / ctiles) % P1;
    const uint64_t fl = blockIdx.x / (ctiles * P1);
    const float2* u = a.scratch + fl * M + k1a * (Q * P2);
    for (int e = tid; e < P2 * 4; e += NT) {
        const int r = e >> 2, q = e & 3;
        const float4 d = *reinterpret_cast<const float4*>(u + (uint64_t)r * Q + c0 + 2 * q);
        sbuf[(2 * q) * BS + K::pd(r)] = make_float2(d.x, d.y);
        sbuf[(2 * q + 1) * BS + K::pd(r)] = make_float2(d.z, d.w);
    }
    __syncthreads();
    const int col = tid / T, t = tid % T;
    float2* buf = sbuf + col * BS;
    const uint64_t c = c0 + col;
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = buf[K::pd(t + i * T)];
    K::fft(v, buf, a.tw3, t);  // slot i: output k1b = t + i T
    __syncthreads();
    // W_M^{c (k1a + P1 k1b)}: a two-level lookup at i = 0 and 8, products with
    // W_M^{c P1 T} between (exponents below M: c < Q, k1a + P1 k1b < P1 P2)
    const float2 step = tw2l(a.twm_lo, a.twm_hi, c * P1 * (uint64_t)T);
    float2 w = make_float2(1.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int k1b = t + i * T;
        w = (i % 8 == 0) ? tw2l(a.twm_lo, a.twm_hi, c * (k1a + P1 * (uint64_t)k1b)) : cmul(w, step);
        buf[K::pd(k1b)] = cmul(v[i], w);
    }
    __syncthreads();
    float2* y = a.scratch2 + fl * M;
    for (int e = tid; e < P2 * 4; e += NT) {
        const int kb = e >> 2, q = e & 3;
        const float2 lo = sbuf[(2 * q) * BS + K::pd(kb)], hi = sbuf[(2 * q + 1) * BS + K::pd(kb)];
        *reinterpret_cast<float4*>(y + (k1a + P1 * (uint64_t)kb) * Q + c0 + 2 * q) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
}

__global__ void build_two_level_kernel(float2* lo, float2* hi, uint64_t L, uint64_t nhi)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < 1024 + nhi;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t j = i < 1024 ? i : (i - 1024) * 1024;
        double s, c;
        sincospi(-2.0 * (double)(j % L) / (double)L, &s, &c);
        const float2 w = make_float2((float)c, (float)s);
        if (i < 1024) lo[i] = w;
        else hi[i - 1024] = w;
    }
}

template <int EXP1>
cudaError_t launch_columns_t(const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    constexpr int T = fused_M(EXP1) / fused_cfg(EXP1).R;
    constexpr int TC = large_col_tile(EXP1);
    constexpr size_t smem = (size_t)TC * large_col_stride_t(EXP1, TC) * sizeof(float2);
    auto k = large_columns_kernel<EXP1>;
    const cudaError_t e = ensure_smem_attr<large_columns_kernel<EXP1>>(smem);
    if (e != cudaSuccess) return e;
    constexpr int FPC = large_col_frames(EXP1);
    const uint64_t grid = (frames + FPC - 1) / FPC * (a.m2 / TC);
    LargeArgs b = a;
    b.frames_launch = frames;
    k<<<(unsigned)grid, TC * T, smem, st>>>(b);
    return cudaGetLastError();
}

template <int EXP2>
cudaError_t launch_rows_e(int outk, const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    switch (outk) {
    case OUT_POWER: return launch_rows_t<EXP2, OUT_POWER>(a, frames, st);
    case OUT_POWER_SERIAL: return launch_rows_t<EXP2, OUT_POWER_SERIAL>(a, frames, st);
    case OUT_HALF:
        if constexpr (EXP2 == 11) return launch_rows_half_11(a, frames, st);
        else return launch_rows_t<EXP2, OUT_HALF>(a, frames, st);
    case OUT_PLANES: return launch_rows_t<EXP2, OUT_PLANES>(a, frames, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int EXPM>
cudaError_t launch_middle_t(const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    constexpr int T = fused_M(EXPM) / fused_cfg(EXPM).R;
    constexpr size_t smem = (size_t)kTileC * large_col_stride(EXPM) * sizeof(float2);
    const cudaError_t e = ensure_smem_attr<large_middle_kernel<EXPM>>(smem);
    if (e != cudaSuccess) return e;
    const uint64_t grid = frames * a.m1 * (a.m2 / kTileC);
    large_middle_kernel<EXPM><<<(unsigned)grid, kTileC * T, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_columns(int l1, const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    switch (l1 + 1) {  // EXP1: the column FFT is the core of window 2^EXP1
    case 9: return launch_columns_t<9>(a, frames, st);
    case 10: return launch_columns_t<10>(a, frames, st);
    case 11: return launch_columns_t<11>(a, frames, st);
    case 12: return launch_columns_t<12>(a, frames, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rows(int l3, int outk, const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    switch (l3 + 1) {
    case 10: return launch_rows_e<10>(outk, a, frames, st);
    case 11: return launch_rows_e<11>(outk, a, frames, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_middle(int l2, const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    switch (l2 + 1) {
    case 6: return launch_middle_t<6>(a, frames, st);
    case 7: return launch_middle_t<7>(a, frames, st);
    case 8: return launch_middle_t<8>(a, frames, st);
    case 9: return launch_middle_t<9>(a, frames, st);
    case 10: return launch_middle_t<10>(a, frames, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// windows of the tiled kernels (stft_large_tiled.cuh)
static constexpr bool large_tiled(int exp) { return exp >= 16 && exp <= 19; }
cudaError_t launch_large_tiled(int l1, int l2, int outk, const LargeArgs& a, uint64_t frames, cudaStream_t st);

bool large_supports(int exp) { return exp >= kLargeMinExp && exp <= kLargeMaxExp; }

// Two passes up to 2^22 (column FFT 2^(exp/2), rows of the rest).  Above,
// rows of Q = 2^l3 points (the largest row pass, 2^10, but at 2^23), a column FFT
// of 2^l1 and a middle FFT of 2^l2, l1 >= l2 as close as l1 >= 8 allows.
static constexpr LargePlan plan_of(int exp)
{
    if (large_tiled(exp)) {
        const int l2 = exp == 16 ? 7 : 8;
        return LargePlan{2, exp - 1 - l2, 0, l2};
    }
    if (exp <= 22) return LargePlan{2, large_l1(exp), 0, large_l2(exp)};
    for (int l3 = 10; l3 >= 9; --l3) {
        const int rest = exp - 1 - l3;
        const int l1 = (rest + 1) / 2 < 8 ? 8 : (rest + 1) / 2;
        if (rest - l1 >= 5) return LargePlan{3, l1, rest - l1, l3};
    }
    return LargePlan{0, 0, 0, 0};
}
// every window's passes are among the ones launch_columns, launch_middle and
// launch_rows hold
static constexpr bool plans_held()
{
    for (int exp = 20; exp <= kLargeMaxExp; ++exp) {
        const LargePlan p = plan_of(exp);
        if (p.passes == 0 || p.l1 < 8 || p.l1 > 11 || p.l3 < 9 || p.l3 > 10) return false;
        if (p.passes == 3 && (p.l2 < 5 || p.l2 > 9)) return false;
        if (p.l1 + p.l2 + p.l3 != exp - 1) return false;
    }
    return true;
}
static_assert(plans_held(), "");
LargePlan large_plan(int exp) { return plan_of(exp); }

cudaError_t build_two_level(float2* lo, float2* hi, uint64_t L, cudaStream_t st)
{
    const uint64_t nhi = (L + 1023) / 1024;
    build_two_level_kernel<<<64, 256, 0, st>>>(lo, hi, L, nhi);
    return cudaGetLastError();
}

namespace {

// the passes of frames [a.f0, a.f0 + frames) over a.scratch (and a.scratch2)
cudaError_t launch_passes(int exp, int outk, const LargeArgs& a, uint64_t frames, cudaStream_t st)
{
    const LargePlan pl = large_plan(exp);
    if (large_tiled(exp)) return launch_large_tiled(pl.l1, pl.l3, outk, a, frames, st);
    const uint64_t q = 1ull << pl.l3;
    LargeArgs c = a;  // column pass: FFT of 2^l1, columns = M / 2^l1
    c.m1 = 1ull << pl.l1;
    c.m2 = 1ull << (pl.l2 + pl.l3);
    c.col_mask = pl.passes == 3 ? ~(q - 1) : ~0ull;
    cudaError_t e = launch_columns(pl.l1, c, frames, st);
    if (e != cudaSuccess) return e;
    LargeArgs r = a;  // row pass: rows of Q points, M / Q of them
    r.m1 = 1ull << (pl.l1 + pl.l2);
    r.m2 = q;
    if (pl.passes == 3) {
        LargeArgs m = a;
        m.m1 = 1ull << pl.l1;
        m.m2 = q;
        e = launch_middle(pl.l2, m, frames, st);
        if (e != cudaSuccess) return e;
        r.scratch = a.scratch2;
    }
    return launch_rows(pl.l3, outk, r, frames, st);
}

// Scratch comes from a memory pool of this library's own, so that the memory
// of one request serves the next: the device's default pool gives it back to
// the system at every synchronisation, and a request alone then paid 1.9 ms to
// map 800 MB again (2^18, 1e8 samples: 2.6 ms of which 0.7 ran).  The pool is
// stream-ordered (requests of several streams and threads never share a block
// at one time), keeps at most kPoolKeep bytes idle, and goes at
// large_release().  A captured request allocates from the default pool, whose
// allocations the graph owns.
constexpr uint64_t kPoolKeep = 1ull << 30;

struct LargeState {
    std::mutex mu;
    std::map<int, cudaMemPool_t> pools;  // device -> pool
};
LargeState& state()
{
    static LargeState* s = new LargeState();  // outlives static teardown
    return *s;
}

cudaError_t pool_get(int device, cudaMemPool_t* out)
{
    LargeState& s = state();
    std::lock_guard<std::mutex> lk(s.mu);
    auto it = s.pools.find(device);
    if (it != s.pools.end()) {
        *out = it->second;
        return cudaSuccess;
    }
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = device;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &p);
    if (e != cudaSuccess) return e;
    uint64_t keep = kPoolKeep;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
        cudaMemPoolDestroy(pool);
        return e;
    }
    s.pools[device] = pool;
    *out = pool;
    return cudaSuccess;
}

}  // namespace

// gives the pools back (ocs_shutdown; a pool goes once its last block is free)
void large_release()
{
    LargeState& s = state();
    std::lock_guard<std::mutex> lk(s.mu);
    for (auto& kv : s.pools) cudaMemPoolDestroy(kv.second);
    s.pools.clear();
}

// Frames [a.f0, a.f0 + frames) in chunks whose scratch is at most the budget
// (one frame at a time when a frame needs more).
cudaError_t launch_large(int exp, int outk, const LargeArgs& args, uint64_t frames, cudaStream_t st)
{
    if (!large_supports(exp) || frames == 0) return cudaErrorInvalidValue;
    const LargePlan pl = large_plan(exp);
    if (pl.passes == 0) return cudaErrorInvalidValue;
    // Chunks small enough for the scratch to stay in L2 lose to fewer, fuller
    // launches, also with the row pass of one chunk on a second stream beside
    // the column pass of the next (2^18, 1e8 samples: 1024 MB 554 us, 96 MB
    // 655, 48 MB 712; 2^16 505, 567, 633): a chunk's launches fill one or two
    // waves only.
    uint64_t budget = 1024ull << 20;
    if (const char* sb = std::getenv("OCS_LARGE_SCRATCH_MB"))
        budget = (uint64_t)std::min(std::max(1L, std::atol(sb)), 1L << 20) << 20;  // 1 MB .. 1 TB
    const uint64_t bytes = (1ull << (exp - 1)) * sizeof(float2);  // per frame
    const uint64_t per = std::max<uint64_t>(1, std::min<uint64_t>(frames, budget / bytes));
    const uint64_t chunks = (frames + per - 1) / per;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (e == cudaSuccess) e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return e;
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    const int bufs = pl.passes == 3 ? 2 : 1;
    float2* buf[2] = {nullptr, nullptr};
    cudaMemPool_t pool = nullptr;
    if (!capturing) e = pool_get(device, &pool);
    for (int i = 0; i < bufs && e == cudaSuccess; ++i)
        e = capturing ? cudaMallocAsync(reinterpret_cast<void**>(&buf[i]), per * bytes, st)
                      : cudaMallocFromPoolAsync(reinterpret_cast<void**>(&buf[i]), per * bytes, pool, st);
    for (uint64_t i = 0; i < chunks && e == cudaSuccess; ++i) {
        LargeArgs a = args;
        a.f0 = args.f0 + i * per;
        const uint64_t n = std::min(per, frames - i * per);
        a.scratch = buf[0];
        a.scratch2 = buf[1];
        e = launch_passes(exp, outk, a, n, st);
    }
    for (float2* b : buf)
        if (b) {
            const cudaError_t fe = cudaFreeAsync(b, st);
            if (e == cudaSuccess) e = fe;
        }
    return e;
}

}  // namespace ocs

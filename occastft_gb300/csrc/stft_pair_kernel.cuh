// Paired-frame fused STFT kernel (windows 2^6 and 2^8 .. 2^10, sm_103a).
//
// Two consecutive real frames a = 2p and b = 2p+1 ride in one N-point complex
// FFT, z[c] = y_a[c] + i y_b[c] (the classic "two real FFTs for one" identity):
//   A[k] = (Z[k] + conj Z[N-k]) / 2,   B[k] = (Z[k] - conj Z[N-k]) / (2i).
// Compared with one N/2-point FFT per frame plus the real-input untangle this
// needs no untangle twiddles, reads each window coefficient once for two
// frames, and with 32 values per thread needs a single shared-memory exchange
// up to N = 1024.  The 1/2 factors are folded into the window table (the
// table is pre-scaled by 1/2, an exact operation).
//
// Per frame it implements the same pipeline as the reference's
// Overlap_Common -> Window_* -> DCRemove_Common -> Stockham FFT -> toPower /
// toHalfComplexFormat (OKL/EXPCommon.okl:7-245, OKL/kernel.okl:178-218).
#pragma once
#include "stft_fused_kernel.cuh"

namespace ocs {

// ------------------------------------------------------------ plan
// Windows 2^8 (16 values per thread), 2^9 and 2^10 (32): a pair is one exchange
// inside a warp, and 16 or 32 lanes store 64 or 128 bytes of a row at a time.
// 2^8 runs it only when asked to (OCS_KERNEL=pair), because two frames in one
// FFT round relative to the louder of the two: 1e8 samples, power, overlap 0.5 /
// 0.75 / 0.3, the lanes-per-frame kernel 240 / 459 / 204 us, this 204 / 367 /
// 162; with 32 values and 8 lanes here 296 / 548 / 223.  At 2^7 the
// lanes-per-frame kernel stays (205 us against 290 here with 16 values and 276
// with 8, which take a second exchange), and at 2^6 (204; the pair plan is for
// outputs that do not start on 16 bytes, which that kernel cannot write: 440
// against 705 us for the one-frame kernel); at 2^11 the one-frame kernel is
// faster (one exchange; 241 against 330 us), above it the mirror-group kernel.
__host__ __device__ constexpr int pair_R(int pid) { return pid <= 8 ? 16 : 32; }

__host__ __device__ constexpr FusedCfg pair_cfg(int pid)
{
    FusedCfg c{pid, pair_R(pid), 0, {1, 1, 1, 1, 1, 1}};
    const int lr = c.R == 32 ? 5 : 4;
    int left = pid;  // log2 of the complex FFT size N
    int s = 0;
    while (left >= lr) { c.radix[s++] = 1 << lr; left -= lr; }
    if (left > 0) c.radix[s++] = 1 << left;
    c.nstages = s;
    return c;
}
__host__ __device__ constexpr int pair_T(int pid) { return (1 << pid) / pair_R(pid); }
__host__ __device__ constexpr int pair_Ns(int pid, int s)
{
    int ns = 1;
    for (int i = 0; i < s; ++i) ns *= pair_cfg(pid).radix[i];
    return ns;
}
// twiddle table: for each stage s >= 1, (r_s - 1) * Ns(s) entries, (m-1)*Ns + j = W_{Ns r}^{j m}
__host__ __device__ constexpr int pair_tw_offset(int pid, int s)
{
    int off = 0;
    for (int i = 1; i < s; ++i) off += (pair_cfg(pid).radix[i] - 1) * pair_Ns(pid, i);
    return off;
}
__host__ __device__ constexpr int pair_tw_size(int pid)
{
    return pair_tw_offset(pid, pair_cfg(pid).nstages) > 0 ? pair_tw_offset(pid, pair_cfg(pid).nstages) : 1;
}
__host__ __device__ constexpr int pair_cta_threads(int) { return 256; }
__host__ __device__ constexpr int pair_ppc(int pid) { return pair_cta_threads(pid) / pair_T(pid); }  // pairs per CTA
__host__ __device__ constexpr int pair_buf_stride(int pid)
{
    return (1 << pid) + (1 << pid) / pair_R(pid) + 1;
}
__host__ __device__ constexpr bool pair_supported(int pid) { return pid == 6 || (pid >= 8 && pid <= 10); }
// 2 x 256 threads per SM; 3 at 2^8, whose 16 values fit 80 registers (overlap
// 0.5 / 0.75 / dense: two CTAs 204 / 387 / 182 us, three 204 / 367 / 172, four
// 213 / 384 / 173).  At 2^10, 16 values per thread and three CTAs of up to 80
// registers measured 300 against 390 Gsamples/s: the extra block-wide exchange
// costs more than the occupancy gains.
__host__ __device__ constexpr int pair_min_blocks(int pid) { return pid == 8 ? 3 : 2; }
__host__ __device__ constexpr size_t pair_tab_bytes(int pid)
{
    return (size_t)pair_tw_size(pid) * 8 + (size_t)(1 << pid) * 4;
}
__host__ __device__ constexpr size_t pair_smem_bytes_ct(int pid)
{
    return (size_t)pair_ppc(pid) * pair_buf_stride(pid) * 8 + pair_tab_bytes(pid);
}

template <int EXP>
struct PairCore {
    static constexpr FusedCfg C = pair_cfg(EXP);
    static constexpr int N = 1 << EXP;
    static constexpr int R = C.R;
    static constexpr int T = N / R;
    static constexpr int NS = C.nstages;
    static constexpr int LP = ilog2(R);
    static constexpr unsigned FULL = 0xffffffffu;
    static __device__ __forceinline__ int pd(int i) { return padl<LP>(i); }

    // subtract each frame's mean: frame a is the real part, frame b the imaginary part
    static __device__ __forceinline__ void remove_dc(float2 (&v)[R])
    {
        float sa = 0.0f, sb = 0.0f;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            sa += v[u].x;
            sb += v[u].y;
        }
#pragma unroll
        for (int o = T / 2; o > 0; o >>= 1) {
            sa += __shfl_xor_sync(FULL, sa, o);
            sb += __shfl_xor_sync(FULL, sb, o);
        }
        const float ma = sa * (1.0f / (float)N), mb = sb * (1.0f / (float)N);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            v[u].x -= ma;
            v[u].y -= mb;
        }
    }

    // tw: the plan's twiddles in shared memory
    static __device__ __forceinline__ void fft(float2 (&v)[R], float2* buf, const float2* tw, int t)
    {
        {
            constexpr int r = C.radix[0];
            static_for<0, R / r>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                dft_inreg<R, r, q, R / r>(v);
            });
        }
        static_for<1, NS>([&](auto sc) {
            constexpr int s = decltype(sc)::value;
            constexpr int rp = C.radix[s - 1];
            constexpr int nsp = pair_Ns(EXP, s - 1);
            constexpr int r = C.radix[s];
            constexpr int ns = pair_Ns(EXP, s);
            constexpr int toff = pair_tw_offset(EXP, s);
            group_sync<T>();
            static_for<0, R / rp>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                const int g = t + q * T;
                const int base = (g / nsp) * nsp * rp + (g % nsp);
                static_for<0, rp>([&](auto mc) {
                    constexpr int m = decltype(mc)::value;
                    buf[pd(base + m * nsp)] = v[q + m * (R / rp)];
                });
            });
            group_sync<T>();
#pragma unroll
            for (int u = 0; u < R; ++u) v[u] = buf[pd(t + u * T)];
            static_for<0, R / r>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                const int j = (t + q * T) % ns;
                static_for<1, r>([&](auto mc) {
                    constexpr int m = decltype(mc)::value;
                    v[q + m * (R / r)] = cmul(v[q + m * (R / r)], tw[toff + (m - 1) * ns + j]);
                });
                dft_inreg<R, r, q, R / r>(v);
            });
        });
    }

    // Z[N - (t + U*T)]; src is partner_lane
    template <int U>
    static __device__ __forceinline__ float2 partner_at(const float2 (&v)[R], int t, int src)
    {
        float2 p;
        p.x = __shfl_sync(FULL, v[R - 1 - U].x, src);
        p.y = __shfl_sync(FULL, v[R - 1 - U].y, src);
        return (t == 0) ? v[(R - U) % R] : p;
    }
    static __device__ __forceinline__ int partner_lane(int tid, int t)
    {
        const int lane = tid & 31;
        return (lane & ~(T - 1)) | ((T - t) & (T - 1));
    }
};

// the plan's twiddles and the window behind them
template <int EXP>
__device__ __forceinline__ const float* pair_tables(const FusedArgs& a, float2* s_tab, int tid)
{
    constexpr int TWN = pair_tw_size(EXP);
    for (int i = tid; i < TWN; i += blockDim.x) s_tab[i] = a.tw[i];
    float* sw = reinterpret_cast<float*>(s_tab + TWN);
    for (int i = tid; i < (1 << EXP); i += blockDim.x) sw[i] = a.win[i];
    __syncthreads();
    return sw;
}

template <int EXP, int OUTK>
__device__ __forceinline__ void pair_group(const FusedArgs& a, uint64_t pbase, float2* buf, const float2* tws,
                                           const float* win, int tid, int lp, int t);

template <int EXP, int OUTK>
__global__ void __launch_bounds__(pair_cta_threads(EXP), pair_min_blocks(EXP))
stft_pair_kernel(const FusedArgs a)
{
    using K = PairCore<EXP>;
    constexpr int T = K::T;
    constexpr int PPC = pair_ppc(EXP);
    constexpr int BS = pair_buf_stride(EXP);

    extern __shared__ float2 smem[];
    const int tid = threadIdx.x;
    const int lp = tid / T;
    const int t = tid - lp * T;
    float2* buf = smem + lp * BS;
    float2* s_tab = smem + PPC * BS;
    pdl_trigger();
    const float* win = pair_tables<EXP>(a, s_tab, tid);
    pdl_wait();

    const uint64_t pairs = (a.frames + 1) / 2;
    // pairs to prefetch.  2^10, whose registers are full, prefetches always: with the
    // rule its overlap 0.5 takes 200.6 us instead of 199.9 (overlap 0: 128 for 152)
    const uint64_t ahead = EXP == 10 || a.hop < (uint64_t)(1 << EXP) ? pairs : 0;
    for (uint64_t pbase = (uint64_t)blockIdx.x * PPC; pbase < pairs; pbase += (uint64_t)gridDim.x * PPC) {
        // L2 prefetch of the pair this group takes next: samples of frames 2q and
        // 2q + 1, where frames overlap (see the one-frame kernel)
        const uint64_t q = pbase + (uint64_t)gridDim.x * PPC + lp;
        if (t == 0 && q < ahead) {
            const uint64_t s0 = 2 * q * a.hop;
            const uint64_t end = s0 + a.hop + (uint64_t)(1 << EXP);
            prefetch_l2_span(a.x, s0, end < a.n ? end : a.n);
        }
        pair_group<EXP, OUTK>(a, pbase, buf, s_tab, win, tid, lp, t);
    }
}

// One CTA iteration: pairs pbase .. pbase + PPC - 1 (frames 2p, 2p + 1 below
// a.frames); buf is this thread's pair buffer, tws the shared-memory twiddles.
template <int EXP, int OUTK>
__device__ __forceinline__ void pair_group(const FusedArgs& a, uint64_t pbase, float2* buf, const float2* tws,
                                           const float* win, int tid, int lp, int t)
{
    using K = PairCore<EXP>;
    constexpr int N = K::N, R = K::R, T = K::T;
    constexpr int H = N / 2;
    {
        const uint64_t p = pbase + lp;
        const uint64_t fa = 2 * p, fb = 2 * p + 1;
        const bool act_a = fa < a.frames;
        const bool act_b = fb < a.frames;
        float2 v[R];

        // ---------------- framing + window of both frames
        {
            const uint64_t sa = fa * a.hop;
            const uint64_t sb = sa + a.hop;
            const float* xa = a.x + sa;
            const float* xb = a.x + sb;
            if (act_b && sb + N <= a.n && a.hop == (uint64_t)(N / 2)) {
                // frame b starts N/2 = (R/2) T samples after frame a: its slots
                // u < R/2 are frame a's slots u + R/2, so only half of them load
                // (1e8 samples, power: 2^9 377 -> 386, 2^10 392 -> 393 Gsamples/s)
#pragma unroll
                for (int u = 0; u < R; ++u) v[u].x = xa[t + u * T];
#pragma unroll
                for (int u = R / 2; u < R; ++u) v[u].y = xb[t + u * T];
#pragma unroll
                for (int u = 0; u < R / 2; ++u) v[u].y = v[u + R / 2].x;
            } else if (act_b && sb + N <= a.n && a.hop == (uint64_t)(N / 4)) {
                // overlap 0.75: frame b's slots u < 3R/4 are frame a's slots u + R/4
#pragma unroll
                for (int u = 0; u < R; ++u) v[u].x = xa[t + u * T];
#pragma unroll
                for (int u = 3 * R / 4; u < R; ++u) v[u].y = xb[t + u * T];
#pragma unroll
                for (int u = 0; u < 3 * R / 4; ++u) v[u].y = v[u + R / 4].x;
            } else if (act_b && sb + N <= a.n) {
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const int c = t + u * T;
                    v[u] = make_float2(xa[c], xb[c]);
                }
            } else {
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const int c = t + u * T;
                    const float ra = (act_a && sa + c < a.n) ? xa[c] : 0.0f;
                    const float rb = (act_b && sb + c < a.n) ? xb[c] : 0.0f;
                    v[u] = make_float2(ra, rb);
                }
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const float w = win[t + u * T];
                v[u].x *= w;
                v[u].y *= w;
            }
        }
        if (a.remove_dc) K::remove_dc(v);
        K::fft(v, buf, tws, t);
        const int src = K::partner_lane(tid, t);

        // ---------------- separate the two spectra and store
        // slots u < R/2 carry k = t + u*T < N/2; thread 0 also owns k = N/2 (slot R/2)
        auto bins = [&](auto& power) __attribute__((always_inline)) {
            static_for<0, R / 2 + 1>([&](auto uc) {
                constexpr int u = decltype(uc)::value;
                const float2 pz = K::template partner_at<u>(v, t, src);
                if (u == R / 2 && t != 0) return;
                const int k = t + u * T;
                const float2 z = v[u];
                const float2 A = make_float2(z.x + pz.x, z.y - pz.y);  // frame a, bin k
                const float2 B = make_float2(z.y + pz.y, pz.x - z.x);  // frame b, bin k
                if constexpr (OUTK == OUT_POWER || OUTK == OUT_POWER_SERIAL) {
                    bool wa, wb;
                    const float pa = power.of(A, wa), pb = power.of(B, wb);
                    if (!a.dense) {
                        float* ra = a.out + fa * (uint64_t)N;
                        // slots 0 < u < R/2 hold T <= k < H: both mirror bins exist
                        constexpr bool inner = u != 0 && u != R / 2;
                        const bool mirror = inner || (k != 0 && k != H);
                        if (act_b) {  // both frames of the pair (act_b implies act_a)
                            stcs_if(wa, ra + k, pa);
                            stcs_if(wb, ra + N + k, pb);
                            if (mirror) {
                                stcs_if(wa, ra + (N - k), pa);
                                stcs_if(wb, ra + N + (N - k), pb);
                            }
                        } else if (act_a) {
                            stcs_if(wa, ra + k, pa);
                            if (mirror) stcs_if(wa, ra + (N - k), pa);
                        }
                    } else {
                        float* ra = a.out + fa * (uint64_t)(H + 1);
                        if (act_a) stcs_if(wa, ra + k, pa);
                        if (act_b) stcs_if(wb, ra + (H + 1) + k, pb);
                    }
                } else if constexpr (OUTK == OUT_HALF) {
                    float2* o2 = reinterpret_cast<float2*>(a.out);
                    if (!a.dense) {
                        const uint64_t fla = fa * (uint64_t)N;
                        const uint64_t flb = fla + N;
                        if (act_a && fla + k < a.ohalf) __stcs(o2 + fla + k, A);
                        if (act_a && k != 0 && k != H && fla + (N - k) < a.ohalf)
                            __stcs(o2 + fla + (N - k), make_float2(A.x, -A.y));
                        if (act_b && flb + k < a.ohalf) __stcs(o2 + flb + k, B);
                        if (act_b && k != 0 && k != H && flb + (N - k) < a.ohalf)
                            __stcs(o2 + flb + (N - k), make_float2(B.x, -B.y));
                    } else {
                        float2* ra = o2 + fa * (uint64_t)(H + 1);
                        if (act_a) __stcs(ra + k, A);
                        if (act_b) __stcs(ra + (H + 1) + k, B);
                    }
                }
            });
        };
        BinPower<OUTK, false> power;
        bins(power);
        if constexpr (OUTK == OUT_POWER) {
            // the partners travel by shuffle: the whole warp takes the second pass
            if (__any_sync(0xffffffffu, act_a && power.again())) {
                BinPower<OUTK, true> fix;
                bins(fix);
            }
        }
    }
}

template <int EXP, int OUTK>
cudaError_t launch_pair_t(const FusedArgs& a, int grid, cudaStream_t st)
{
    if constexpr (pair_supported(EXP) && OUTK != OUT_PLANES) {
        constexpr int threads = pair_cta_threads(EXP);
        constexpr size_t sm = pair_smem_bytes_ct(EXP);
        auto k = stft_pair_kernel<EXP, OUTK>;
        const cudaError_t e = ensure_smem_attr<stft_pair_kernel<EXP, OUTK>>(sm);
        if (e != cudaSuccess) return e;
        return launch_pdl(k, grid, threads, sm, st, a);
    } else {
        return cudaErrorInvalidValue;
    }
}

template <int EXP, int OUTK>
int occupancy_pair_t()
{
    int blocks = 0;
    if constexpr (pair_supported(EXP) && OUTK != OUT_PLANES) {
        auto k = stft_pair_kernel<EXP, OUTK>;
        constexpr size_t sm = pair_smem_bytes_ct(EXP);
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, pair_cta_threads(EXP), sm) != cudaSuccess)
            return 0;
    }
    return blocks;
}

template <int EXP>
cudaError_t launch_pair_exp(int outk, const FusedArgs& a, int grid, cudaStream_t st)
{
    switch (outk) {
    case OUT_POWER: return launch_pair_t<EXP, OUT_POWER>(a, grid, st);
    case OUT_POWER_SERIAL: return launch_pair_t<EXP, OUT_POWER_SERIAL>(a, grid, st);
    case OUT_HALF: return launch_pair_t<EXP, OUT_HALF>(a, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int EXP>
int occupancy_pair_exp(int outk)
{
    switch (outk) {
    case OUT_POWER: return occupancy_pair_t<EXP, OUT_POWER>();
    case OUT_POWER_SERIAL: return occupancy_pair_t<EXP, OUT_POWER_SERIAL>();
    case OUT_HALF: return occupancy_pair_t<EXP, OUT_HALF>();
    default: return 0;
    }
}

}  // namespace ocs

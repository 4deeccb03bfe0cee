// Two-launch STFT of windows 2^16 .. 2^19 with a tiled scratch (sm_103a).
//
// The transform is the four-step FFT of stft_large.cu, M = M1 M2 complex
// points, m = c + M2 m1, k = k1 + M1 k2:
//   column pass  Y[k1][c] = W_M^{c k1} sum_{m1} z[c + M2 m1] W_{M1}^{m1 k1}
//   row pass     Z[k1 + M1 k2] = sum_c Y[k1][c] W_{M2}^{c k2}, untangle, store.
// What differs is how the points travel.  Both passes keep 16 neighbouring
// columns (or rows) in the 16 lanes of a half-warp, so that every global
// access moves whole 128-byte lines straight between memory and the registers
// of the FFT, and shared memory carries one exchange per pass:
//   column pass  loads with lanes over c; the exchange turns the lanes to k1,
//                and Y goes out as Y'[k1 / 16][c][k1 mod 16]
//   row pass     a CTA owns the 16 rows of a tile and their mirrors M1 - k1;
//                lanes over k1 from the load to the store, whose bins k1 ..
//                k1 + 15 are 16 consecutive floats.  A thread runs group t of
//                a row and group T - 1 - t of its mirror, which holds the
//                partners Z[M - k], so the untangle reads registers.
// The kernels before moved every point through shared memory two more times
// per pass (staging of the rows read and written), took the untangle's partners
// from shared memory and stored 8 consecutive bins; their L1 pipe was 73-83%
// busy, now 61% in the column pass and 53% in the row pass (2^18).  1e8 samples, Hamming, overlap 0.5, power / half-complex,
// before -> after (us): 2^16 660 -> 502 / 430 -> 370; 2^17 655 -> 510 / 430 ->
// 369; 2^18 716 -> 532 / 475 -> 376; 2^19 720 -> 652 / 480 -> 441.  The scratch's
// round trip makes the DRAM bytes 2.3 times the request's (2.8 GB, 412 us).
//
// Scratch loads and output stores take the default cache policy: a line of
// mirror rows is read by two CTAs and a line of outputs written by two, so
// evict-first on either made them travel again (2^16: loads 604 -> 507 us).
// For the same reason more CTAs per SM (80 registers) lose: 502 -> 568.
//
// Row 0 and row M1/2 pair with themselves.  They are lane 0 of the first tile
// (row M1/2 in the place of row 0's mirror), whose threads exchange their
// results through shared memory.
#pragma once
#include "stft_mirror_kernel.cuh"

namespace ocs {

constexpr int kLtTile = 16;  // rows per tile

// ---------------------------------------------------------------- column pass
// M1 = RA RB points, 32 (M1 = 256: 16) per thread; stage 1 DFT over RA points
// m1 = q + RB p of every q, stage 2 over RB points of every k0 < RA; k1 = k0 +
// RA kk.  TC columns per CTA of 256 threads.
template <int L1>
struct LtCol {
    static constexpr int M1 = 1 << L1;
    static constexpr int RA = L1 == 8 ? 16 : 32;
    static constexpr int RB = M1 / RA;             // 16, 16, 32
    static constexpr int T = RB;                   // threads per column
    static constexpr int TC = 256 / T;             // 16, 16, 8
    static constexpr int GR = RA / RB;             // stage-2 groups per thread
    static constexpr int ROWS = mirror_rows(RB);   // twiddle rows of stage 2
    // Columns of 256 points take four consecutive frames per CTA, keep their
    // window coefficients in registers and load the next frame's samples while
    // stage 2 works on this one's (2^16: one frame 591, two 516, four 502, eight
    // 503 us for 1e8 samples, power).  With 32 values per thread that spills
    // (2^18: one frame 532, four 554).
    static constexpr bool MULTI = L1 == 8;
    static constexpr int FPC = MULTI ? 4 : 1;
    static constexpr size_t SMEM = (size_t)M1 * TC * 8 + (size_t)ROWS * RA * 8;
};

// W_{M1}^e, e < M1, from the plan table of window 2 M1 (tw[k] = W_{2 M1}^k, k < M1)
__device__ __forceinline__ float2 lt_w(const float2* tw, int m1, int e)
{
    const int i = 2 * (e & (m1 - 1));
    const float2 w = tw[i & (m1 - 1)];
    return i < m1 ? w : make_float2(-w.x, -w.y);
}
__device__ __forceinline__ float2 lt_two_level(const float2* lo, const float2* hi, uint32_t j)
{
    return cmul(lo[j & 1023u], hi[j >> 10]);
}

template <int L1>
__global__ void __launch_bounds__(256, 2) large_tiled_columns_kernel(const LargeArgs a)
{
    using C = LtCol<L1>;
    constexpr int M1 = C::M1, RA = C::RA, RB = C::RB, TC = C::TC, GR = C::GR;
    extern __shared__ float2 sbuf[];
    float2* const s_tw = sbuf + M1 * TC;  // [row][k0]: W_{M1}^{m k0}
    const int tid = threadIdx.x;
    const uint32_t M2 = (uint32_t)a.m2;
    const uint32_t M = M1 * M2;
    const uint32_t N = 2 * M;
    const uint32_t tiles = M2 / TC;
    const uint64_t fg = blockIdx.x / tiles;
    const uint32_t c0 = (blockIdx.x % tiles) * TC;
    pdl_trigger();
    pdl_wait();
    for (int i = tid; i < C::ROWS * RA; i += 256) s_tw[i] = lt_w(a.tw1, M1, mirror_row_m(i / RA) * (i % RA));
    // stage 1: column c0 + sc, rows q + RB p
    const int sc = tid % TC, q = tid / TC;
    // stage 2: k0 = kt + 16 kh (RB = 32) or kt (+ 16 g), column c0 + dc
    const int kt = tid & 15, dc = (tid >> 4) % TC;
    const int k0 = kt + 16 * (tid / (16 * TC));
    float2 wv[C::MULTI ? RA : 1];
    const uint32_t i0 = 2 * (c0 + sc + M2 * (uint32_t)q);  // real index of point p = 0
    const uint32_t istep = 2 * M2 * RB;
    auto win_at = [&](int p) {
        return a.win ? *reinterpret_cast<const float2*>(a.win + i0 + istep * p) : make_float2(0.5f, 0.5f);
    };
    if constexpr (C::MULTI) {
#pragma unroll
        for (int p = 0; p < RA; ++p) wv[p] = win_at(p);
    }
    const bool vec2 = (a.hop & 1) == 0 && (reinterpret_cast<uintptr_t>(a.x) & 7) == 0;
    // W_M^{c k1}, k1 = k0 + 16 g + RA kk: W_M^{c k0} times powers of W_M^{c RA} (and of W_M^{16 c})
    const uint32_t c = c0 + dc;

    // samples of frame fl of the launch (zeros past the signal's end)
    auto load = [&](float2 (&v)[RA], uint64_t fl) __attribute__((always_inline)) {
        const uint64_t f = a.f0 + fl;
        const uint64_t s0 = f * a.hop;
        const float* x = a.x + s0 + i0;
        if (f < a.frames_total && s0 + N <= a.n) {
            if (vec2) {
#pragma unroll
                for (int p = 0; p < RA; ++p) v[p] = *reinterpret_cast<const float2*>(x + (size_t)istep * p);
            } else {
#pragma unroll
                for (int p = 0; p < RA; ++p) v[p] = make_float2(x[(size_t)istep * p], x[(size_t)istep * p + 1]);
            }
        } else {
#pragma unroll
            for (int p = 0; p < RA; ++p) {
                const uint64_t g = s0 + i0 + (uint64_t)istep * p;
                v[p] = make_float2(f < a.frames_total && g < a.n ? x[(size_t)istep * p] : 0.0f,
                                   f < a.frames_total && g + 1 < a.n ? x[(size_t)istep * p + 1] : 0.0f);
            }
        }
    };
    float2 v[RA];
    if (fg * C::FPC < a.frames_launch) load(v, fg * C::FPC);
#pragma unroll 1
    for (int ff = 0; ff < C::FPC; ++ff) {
        const uint64_t fl = fg * C::FPC + ff;
        if (fl >= a.frames_launch) break;
        // the exchange places are formed anew for each frame: kept over the
        // loop they would take the registers the loads in flight need
        int so = sc, dd = dc;
        asm volatile("" : "+r"(so), "+r"(dd));
#pragma unroll
        for (int p = 0; p < RA; ++p) {
            if constexpr (C::MULTI) v[p] = mul2(v[p], wv[p]);
            else v[p] = mul2(v[p], win_at(p));
        }
        dft_inreg<RA, RA, 0, 1>(v);
        __syncthreads();  // the previous frame's reads of the buffer (and the table's writes) are over
        // point (k0, q) of column sc: the column XORed by k0 (and, with 8
        // columns, q's low bit by k0's bit 3), so that both the 16 columns of
        // stage 1's half-warps and the 16 k0 of stage 2's lie in 16 banks
        auto place = [&](int kk0, int qq, int cc) {
            if constexpr (TC == 16) return (kk0 * RB + qq) * 16 + (cc ^ (kk0 & 15));
            else return (kk0 * RB + (qq ^ ((kk0 >> 3) & 1))) * 8 + (cc ^ (kk0 & 7));
        };
#pragma unroll
        for (int k = 0; k < RA; ++k) sbuf[place(k, q, so)] = v[k];
        __syncthreads();
        // the next frame's samples travel while stage 2 works on this one's
        if constexpr (C::MULTI) {
            if (ff + 1 < C::FPC && fl + 1 < a.frames_launch) load(v, fl + 1);
        }
        // ---------------- stage 2, times W_M^{c k1}, out
        const float2 stepg = lt_two_level(a.twm_lo, a.twm_hi, c * (uint32_t)RA);  // W_M^{c RA}
        const float2 step2 = lt_two_level(a.twm_lo, a.twm_hi, 2 * c * (uint32_t)RA);
        const float2 step4 = lt_two_level(a.twm_lo, a.twm_hi, 4 * c * (uint32_t)RA);
        const float2 step3 = cmul(step2, stepg);
        float2* const y = a.scratch + fl * (uint64_t)M;
        static_for<0, GR>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            const int kg = k0 + 16 * g;
            float2 u[RB];
            u[0] = sbuf[place(kg, 0, dd)];
            mirror_twiddles<RB>(s_tw + kg, RA, [&](auto mc, float2 w) {
                constexpr int m = decltype(mc)::value;
                u[m] = cmul(sbuf[place(kg, m, dd)], w);
            });
            dft_inreg<RB, RB, 0, 1>(u);
            // kk = 4 i + j: W_M^{c kg} W^{4 i} W^j, a table lookup every 8th kk
            float2 b = make_float2(1.0f, 0.0f);
            static_for<0, RB / 4>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                if constexpr (i % 2 == 0) b = lt_two_level(a.twm_lo, a.twm_hi, c * (uint32_t)(kg + 4 * i * RA));
                else b = cmul(b, step4);
                auto put = [&](int j, float2 w) {
                    const uint32_t k1 = kg + RA * (4 * i + j);
                    y[((uint64_t)(k1 / kLtTile) * M2 + c) * kLtTile + (kt & 15)] = cmul(u[4 * i + j], w);
                };
                put(0, b);
                put(1, cmul(b, stepg));
                put(2, cmul(b, step2));
                put(3, cmul(b, step3));
            });
        });
    }
}

// ---------------------------------------------------------------- row pass
// M2 = 16 RB points per row, 16 per thread and row: stage 1 DFT over the 16
// points c = t + T u, stage 2 over RB = T points; k2 = t + T u in slot u.
template <int L2>
struct LtRow {
    static constexpr int M2 = 1 << L2;
    static constexpr int RB = M2 / 16;             // 8, 16
    static constexpr int T = RB;
    static constexpr int THREADS = kLtTile * T;    // 128, 256
    static constexpr int GR = 16 / RB;             // stage-2 groups per thread and row
    static constexpr int ROWS = mirror_rows(RB);
    static constexpr size_t SMEM = (size_t)M2 * kLtTile * 8 + (size_t)ROWS * 16 * 8;
};

template <int L2, int OUTK>
__global__ void __launch_bounds__(LtRow<L2>::THREADS, 512 / LtRow<L2>::THREADS)
large_tiled_rows_kernel(const LargeArgs a)
{
    using R = LtRow<L2>;
    constexpr int M2 = R::M2, RB = R::RB, T = R::T, GR = R::GR;
    extern __shared__ float2 sbuf[];  // [k0 RB + q][16]
    float2* const s_tw = sbuf + M2 * kLtTile;
    const int tid = threadIdx.x;
    const uint32_t M1 = (uint32_t)a.m1;
    const uint32_t M = M1 * M2, N = 2 * M;
    const uint32_t blocks = M1 / (2 * kLtTile);
    const uint64_t fl = blockIdx.x / blocks;
    const uint32_t b = blockIdx.x % blocks;
    const uint64_t f = a.f0 + fl;
    pdl_trigger();
    pdl_wait();
    for (int i = tid; i < R::ROWS * 16; i += R::THREADS) s_tw[i] = lt_w(a.tw2, M2, mirror_row_m(i / 16) * (i % 16));
    const int r = tid & 15, t = tid >> 4;
    const uint32_t k1 = kLtTile * b + r;
    const bool special = k1 == 0;
    float2 v[32];  // slots 0 .. 15 the row, 16 .. 31 its mirror
    {
        const float2* y = a.scratch + fl * (uint64_t)M;
        const uint32_t km = special ? M1 / 2 : M1 - k1;  // the mirror row
        const float2* yd = y + ((uint64_t)b * M2 + t) * kLtTile + r;
        const float2* ym = y + ((uint64_t)(km / kLtTile) * M2 + t) * kLtTile + km % kLtTile;
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = yd[(size_t)u * T * kLtTile];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[16 + u] = ym[(size_t)u * T * kLtTile];
    }
    dft_inreg<32, 16, 0, 1>(v);
    dft_inreg<32, 16, 16, 1>(v);
    // the row's points, then its mirror's, go through one exchange buffer
    float2* const bd = sbuf + r;
    // group k0 = t + T g of the row, (T - 1 - t) + T g of the mirror; slot g + GR kk
    static_for<0, 2>([&](auto mc) {
        constexpr int h = decltype(mc)::value;
        if constexpr (h == 1) __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) bd[(k * RB + t) * kLtTile] = v[16 * h + k];
        __syncthreads();
        static_for<0, GR>([&](auto gc) {
            constexpr int g = decltype(gc)::value;
            const int kg = (h ? T - 1 - t : t) + T * g;
            const float2* const src = bd + kg * RB * kLtTile;
            float2 u[RB];
            u[0] = src[0];
            mirror_twiddles<RB>(s_tw + kg, 16, [&](auto mm, float2 w) {
                constexpr int m = decltype(mm)::value;
                u[m] = cmul(src[m * kLtTile], w);
            });
            dft_inreg<RB, RB, 0, 1>(u);
#pragma unroll
            for (int kk = 0; kk < RB; ++kk) v[16 * h + g + GR * kk] = u[kk];
        });
    });
    if (f >= a.frames_total) return;

    // ---------------- untangle and store: k = k1 + M1 (t + T u), M2 = 16 T
    const bool dc = a.remove_dc != 0;
    float* const ro = a.out + f * (uint64_t)(a.dense ? M + 1 : N);
    float2* const o2 = reinterpret_cast<float2*>(a.out);
    const uint64_t flc = f * (uint64_t)N;
    const bool whole = flc + N <= a.ohalf;
    // bins k, M - k, M + k and N - k of one pair; self: 1 at k = 0 (bins 0 and
    // M), 2 at k = M/2 (bins M/2 and 3M/2)
    auto emit = [&](uint32_t k, float2 A, float2 B, float2 w, int self) {
        const float2 e = make_float2(A.x + B.x, A.y - B.y);
        const float2 wo = cmul(make_float2(A.y + B.y, B.x - A.x), w);
        float2 X0 = cadd(e, wo);        // X[k]
        const float2 X1 = csub(e, wo);  // X[k + M]
        if (dc && k == 0) X0 = make_float2(0.0f, 0.0f);
        if constexpr (OUTK == OUT_POWER || OUTK == OUT_POWER_SERIAL) {
            const float p0 = power_of<OUTK>(X0), p1 = power_of<OUTK>(X1);
            if (!a.dense) {
                ro[k] = p0;
                if (self != 1) ro[N - k] = p0;
                if (self != 2) ro[M + k] = p1;
                if (self == 0) ro[M - k] = p1;
            } else {
                ro[k] = p0;
                if (self != 2) ro[M - k] = p1;
            }
        } else if constexpr (OUTK == OUT_PLANES) {
            auto put = [&](uint32_t bin, float re, float im) {
                a.out[flc + bin] = re;
                a.out_im[flc + bin] = im;
            };
            put(k, X0.x, X0.y);
            if (self != 1) put(N - k, X0.x, -X0.y);
            if (self != 2) put(M + k, X1.x, X1.y);
            if (self == 0) put(M - k, X1.x, -X1.y);
        } else {
            if (!a.dense) {
                auto put = [&](uint32_t bin, float re, float im) {
                    if (whole || flc + bin < a.ohalf) o2[flc + bin] = make_float2(re, im);
                };
                put(k, X0.x, X0.y);
                if (self != 1) put(N - k, X0.x, -X0.y);
                if (self != 2) put(M + k, X1.x, X1.y);
                if (self == 0) put(M - k, X1.x, -X1.y);
            } else {
                float2* const rc = o2 + f * (uint64_t)(M + 1);
                rc[k] = X0;
                if (self != 2) rc[M - k] = self == 1 ? X1 : make_float2(X1.x, -X1.y);
            }
        }
    };
    // W_N^k = W_N^{k1} W_{2 M2}^t W_32^u (N = 2 M1 M2, M2 = 16 T)
    const float2 wt = a.tw2[t];
    if (b == 0) {
        // the first tile: lane 0's rows pair with themselves
        __syncthreads();
        float2* const sd = sbuf;         // row 0's results, then row M1/2's
        float2* const sm = sbuf + M2;
        if (special) {
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                sd[t + T * u] = v[u];
                sm[T - 1 - t + T * u] = v[16 + u];
            }
        }
        __syncthreads();
        if (special) {
            const float2 wh = cmul(lt_two_level(a.twn_lo, a.twn_hi, M1 / 2), wt);
            static_for<0, 8>([&](auto uc) {
                constexpr int u = decltype(uc)::value;
                const int k2 = t + T * u;
                emit(M1 * k2, sd[k2], sd[(M2 - k2) & (M2 - 1)], twc<u, 32>(wt), k2 == 0 ? 1 : 0);
                emit(M1 / 2 + M1 * k2, sm[k2], sm[M2 - 1 - k2], twc<u, 32>(wh), 0);
            });
            if (t == 0) {
                const float2 z = sd[M2 / 2];
                emit(M / 2, z, z, make_float2(0.0f, -1.0f), 2);
            }
            return;
        }
    }
    const float2 wk = cmul(lt_two_level(a.twn_lo, a.twn_hi, k1), wt);
    static_for<0, 16>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        emit(k1 + M1 * (uint32_t)(t + T * u), v[u], v[16 + 15 - u], twc<u, 32>(wk), 0);
    });
}

}  // namespace ocs

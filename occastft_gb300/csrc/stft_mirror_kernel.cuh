// Mirror-group STFT kernel (windows 2^12 .. 2^15, sm_103a).
//
// A complex FFT of P points carries either two consecutive real frames of
// N = P samples (z = y_a + i y_b, "pair") or one frame of N = 2P samples
// (z[m] = y[2m] + i y[2m+1], "single"; mirror_paired says which calls take
// which).  P = r1 r2 16, 32 points per thread,
// T = P / 32 threads per transform, in three stages with two exchanges through
// shared memory.  With n = n0 + 16 n1 + 16 r2 n2 and k = k0 + r1 k1 + G k2
// (G = r1 r2 = P / 16):
//   stage 1  DFT over n2 (r1 points) of every (n0, n1)
//   stage 2  times W_G^{n1 k0}, DFT over n1 (r2 points) of every (n0, k0)
//   stage 3  times W_P^{n0 g}, DFT over n0 (16 points) of every g = k0 + r1 k1:
//            Z[g + G k2]
// Both separations pair Z[k] with Z[P - k].  Groups g and G - g of stage 3
// hold each other's partners, so a thread runs those two groups, t and G - t:
// the partners are its own registers and no third exchange is needed.  Since
// W_P^{n0 (G - t)} = W_16^{n0} conj(W_P^{n0 t}) and a factor W_16^{n0} only
// shifts k2 by one, both groups use one set of twiddles, the second their
// conjugates, and its output slot j is Z[G - t + G (j - 1)].  Groups 0 and G/2
// pair with themselves: thread 0 runs them, with the extra factor W_32^{n0} of
// group G/2.
//
// What bounds it: latency at 16 warps per SM, with the L1/shared-memory pipe at
// 51% and issue at 51% (ncu, 2^12, overlap 0.75).  A transform's 32 points per thread take
// half the registers of an SM, so the plan saves wavefronts, instructions and
// barriers per sample: no third exchange (a third of the exchange traffic);
// the twiddles of a stage from a few table entries and products (6 loads of
// 15, 10 of 31, one rounding more each); the exchanges in place, which takes
// three barriers per transform instead of five and no padding.
// 1e8 samples, Hamming, before -> after (us; power at overlap 0.5, power at
// 0.75, half-complex at 0.5): 2^12 312 -> 275, 601 -> 530, 206 -> 185; 2^13
// 339 -> 298, 653 -> 567, 209 -> 200; 2^14 388 -> 319, 730 -> 621, 256 -> 203;
// 2^15 402 -> 361, 777 -> 699, 269 -> 239.  At 2^11 a frame is one warp of the
// one-frame kernel, which has a single exchange and no barrier: 242 us against
// 254 for this plan.  Half-complex at 2^12 and 2^13 as a pair: 177 and 192 us, but
// a quiet frame beside a loud one then loses digits (8e-4 of its norm at 1e-4 of
// its neighbour's level, 1.4e-7 in the single form).
//
// Per frame it implements the reference's Overlap_Common -> Window_* ->
// DCRemove_Common -> Stockham FFT -> toPower / toHalfComplexFormat
// (OKL/EXPCommon.okl:7-245, OKL/kernel.okl:178-218).
#pragma once
#include "stft_fused_kernel.cuh"

namespace ocs {

// ------------------------------------------------------------ plan
struct MirrorCfg {
    int lp;      // log2 P
    int r1, r2;  // stage radices; the third is 16
};
__host__ __device__ constexpr MirrorCfg mirror_cfg(int lp)
{
    return lp == 11   ? MirrorCfg{11, 16, 8}
           : lp == 12 ? MirrorCfg{12, 16, 16}
           : lp == 13 ? MirrorCfg{13, 32, 16}
                      : MirrorCfg{14, 32, 32};
}
__host__ __device__ constexpr bool mirror_supported(int exp) { return exp >= 12 && exp <= 15; }
__host__ __device__ constexpr int mirror_T(int lp) { return 1 << (lp - 5); }

// A stage of r points takes its twiddles w^m, m < r, from the rows
// m = 1, 2, 3, 4, 8, 12, .. of its table and products w^(4a) w^b.
__host__ __device__ constexpr int mirror_rows(int r) { return 3 + r / 4 - 1; }
__host__ __device__ constexpr int mirror_row_m(int i) { return i < 3 ? i + 1 : 4 * (i - 2); }  // row i's m
// Table of a transform of 2^lp points, in float2:
//   stage 2  [row][k0 < r1]: W_G^{m k0}
//   stage 3  [row][t < T]: W_P^{m t}
//   [t < T]: W_2P^t, the untangle's factor of the single form
__host__ __device__ constexpr int mirror_tw2_size(int lp) { return mirror_rows(mirror_cfg(lp).r2) * mirror_cfg(lp).r1; }
__host__ __device__ constexpr int mirror_tw3_size(int lp) { return mirror_rows(16) * mirror_T(lp); }
__host__ __device__ constexpr int mirror_tab_size(int lp)
{
    return mirror_tw2_size(lp) + mirror_tw3_size(lp) + mirror_T(lp);
}
// transforms per CTA of 256 threads (512 at P = 2^14)
__host__ __device__ constexpr int mirror_threads(int lp) { return mirror_T(lp) > 256 ? mirror_T(lp) : 256; }
__host__ __device__ constexpr int mirror_gpc(int lp) { return mirror_threads(lp) / mirror_T(lp); }
// The window joins the tables in shared memory at 2^12 (16 KB: 283 -> 275 us).
// Above it stays in global memory: its size would come out of the L1 that the
// loads in flight need (2^13 298 -> 319 us; 2^15, half of it, 364 -> 404).
__host__ __device__ constexpr bool mirror_smem_window(int exp) { return exp == 12; }
__host__ __device__ constexpr size_t mirror_smem_bytes(int exp, bool pair)
{
    const int lp = mirror_lp(exp, pair);
    return ((size_t)mirror_gpc(lp) * 8 << lp) + (size_t)mirror_tab_size(lp) * 8 +
           (mirror_smem_window(exp) ? (size_t)4 << exp : 0) + (size_t)(mirror_threads(lp) / 32) * 8;
}

// barrier of the T threads of one transform
template <int LP>
__device__ __forceinline__ void mirror_sync(int lp)
{
    if constexpr (mirror_gpc(LP) == 1) {
        __syncthreads();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(lp + 1), "n"(mirror_T(LP)) : "memory");
    }
}

// f(m, w^m) for m = 1 .. R-1 from the table rows at tab (stride floats2 apart)
template <int R, typename F>
__device__ __forceinline__ void mirror_twiddles(const float2* tab, int stride, F f)
{
    float2 b[4];
    static_for<1, 4>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        b[m] = tab[(m - 1) * stride];
        f(mc, b[m]);
    });
    static_for<1, R / 4>([&](auto ac) {
        constexpr int a = decltype(ac)::value;
        const float2 w = tab[(2 + a) * stride];
        f(std::integral_constant<int, 4 * a>{}, w);
        static_for<1, 4>([&](auto mc) {
            constexpr int m = decltype(mc)::value;
            f(std::integral_constant<int, 4 * a + m>{}, cmul(w, b[m]));
        });
    });
}

template <int EXP, bool PAIR_>
struct Mirror {
    static constexpr bool PAIR = PAIR_;
    static constexpr int N = 1 << EXP, H = N / 2;
    static constexpr int LP = mirror_lp(EXP, PAIR), P = 1 << LP;
    static constexpr int R1 = mirror_cfg(LP).r1, R2 = mirror_cfg(LP).r2;
    static constexpr int T = mirror_T(LP), G = P / 16;

    // Register of point t + T u, u < 32: stage 1's groups in runs of r1 (r1 =
    // 16: group t, then group t + T).
    static __host__ __device__ constexpr int slot(int u) { return R1 == 16 ? (u & 1) * 16 + (u >> 1) : u; }

    // ---------------- framing + window
    static __device__ __forceinline__ void load_pair(float2 (&v)[32], const FusedArgs& a, uint64_t fa, bool act_b,
                                                     const float* win, int t)
    {
        const uint64_t sa = fa * a.hop, sb = sa + a.hop;
        const float* xa = a.x + sa + t;
        const float* xb = a.x + sb + t;
        if (act_b && sb + N <= a.n) {
            // frame b's samples that frame a has loaded already are copied
            // (overlap 0.5 and 0.75)
#pragma unroll
            for (int u = 0; u < 32; ++u) v[slot(u)].x = xa[T * u];
            if (a.hop == (uint64_t)H) {
#pragma unroll
                for (int u = 0; u < 32; ++u) v[slot(u)].y = u < 16 ? v[slot((u + 16) & 31)].x : xb[T * u];
            } else if (a.hop == (uint64_t)(N / 4)) {
#pragma unroll
                for (int u = 0; u < 32; ++u) v[slot(u)].y = u < 24 ? v[slot((u + 8) & 31)].x : xb[T * u];
            } else {
#pragma unroll
                for (int u = 0; u < 32; ++u) v[slot(u)].y = xb[T * u];
            }
        } else {
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                v[slot(u)].x = sa + t + T * u < a.n ? xa[T * u] : 0.0f;
                v[slot(u)].y = act_b && sb + t + T * u < a.n ? xb[T * u] : 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < 32; ++u) {
            v[slot(u)] = mul2(v[slot(u)], bc2(win[t + T * u]));
        }
    }
    static __device__ __forceinline__ void load_single(float2 (&v)[32], const FusedArgs& a, uint64_t f, const float* win,
                                                       int t)
    {
        const uint64_t s = f * a.hop;
        const float* x = a.x + s + 2 * t;
        if (s + N <= a.n) {
            if (a.vec2) {
#pragma unroll
                for (int u = 0; u < 32; ++u) v[slot(u)] = *reinterpret_cast<const float2*>(x + 2 * T * u);
            } else {
#pragma unroll
                for (int u = 0; u < 32; ++u) v[slot(u)] = make_float2(x[2 * T * u], x[2 * T * u + 1]);
            }
        } else {
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                const uint64_t i = s + 2 * (t + T * u);
                v[slot(u)] = make_float2(i < a.n ? x[2 * T * u] : 0.0f, i + 1 < a.n ? x[2 * T * u + 1] : 0.0f);
            }
        }
        const float2* w2 = reinterpret_cast<const float2*>(win) + t;
#pragma unroll
        for (int u = 0; u < 32; ++u) {
            v[slot(u)] = mul2(v[slot(u)], w2[T * u]);
        }
    }
    // subtract the windowed frames' means (DCRemove_Common semantics)
    static __device__ __forceinline__ void remove_dc(float2 (&v)[32], float2* red, int lp, int t)
    {
        float2 s = v[0], s1 = v[1];
#pragma unroll
        for (int j = 2; j < 32; j += 2) {
            s = add2(s, v[j]);
            s1 = add2(s1, v[j + 1]);
        }
        s = add2(s, s1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if ((t & 31) == 0) red[t >> 5] = s;
        mirror_sync<LP>(lp);
        s = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int w = 0; w < T / 32; ++w) s = add2(s, red[w]);
        if constexpr (!PAIR) s = bc2(s.x + s.y);
        const float2 mean = mul2(s, bc2(-1.0f / (float)N));
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = add2(v[j], mean);
    }

    // Place of a point in the exchange buffer: n0 + 16 d1 + (P / r1) d2, d2
    // being n2 and then k0, d1 n1 and then k1, with the low four bits XORed by
    // a function of d2 so that the 16 points a half-warp touches lie in 16
    // banks in every stage: (n0), (n0 mod 8 or 4, low bits of d2) or (n0), and (d2).
    // (Stage 3's mirrored groups step d1 in one lane of 16: one conflict.)
    static __host__ __device__ constexpr int swz(int d2)
    {
        if (R2 == 8) return (d2 >> 2) | ((d2 & 2) << 1) | ((d2 & 1) << 3);  // d2 < 16
        return ((d2 >> 1) & 7) | ((d2 & 1) << 3);
    }

    // In: the windowed points (slot()).  Out: v[k2] = Z[t + G k2] and v[16 + j] =
    // Z[G - t + G ((j - 1) mod 16)] (thread 0: Z[G/2 + ..]).
    //
    // The exchanges work in place: a stage writes its results where it read its
    // points, so only the hand-overs need barriers, three per transform.
    static __device__ __forceinline__ void fft(float2 (&v)[32], float2* buf, const float2* tw2, const float2* tw3,
                                               int lp, int t)
    {
        constexpr int S = P / R1;  // step of d2
        // ---------------- stage 1: group q = (n0, n1) = t (and t + T)
        dft_inreg<32, R1, 0, 1>(v);
        if constexpr (R1 == 16) dft_inreg<32, 16, 16, 1>(v);
        mirror_sync<LP>(lp);  // the previous transform's reads of the buffer are over
        static_for<0, R1>([&](auto kc) {
            constexpr int k0 = decltype(kc)::value;
            const int i = t ^ swz(k0);
            buf[i + S * k0] = v[k0];
            if constexpr (R1 == 16) buf[i + T + S * k0] = v[16 + k0];
        });
        mirror_sync<LP>(lp);
        // ---------------- stage 2
        if constexpr (R2 == 32) {
            const int k0 = t >> 4;
            float2* const b = buf + S * k0 + ((t & 15) ^ swz(k0));
            v[0] = b[0];
            mirror_twiddles<32>(tw2 + k0, R1, [&](auto mc, float2 w) {
                constexpr int m = decltype(mc)::value;
                v[m] = cmul(b[16 * m], w);
            });
            dft_inreg<32, 32, 0, 1>(v);
#pragma unroll
            for (int k1 = 0; k1 < 32; ++k1) b[16 * k1] = v[k1];
        } else if constexpr (R2 == 8) {
            // groups (n0 + 4 i, k0), n0 < 4, i < 4, of one set of twiddles
            const int k0 = t >> 2, m0 = swz(k0);
            float2* const b = buf + S * k0 + ((t & 3) ^ (m0 & 3));
            const int h = m0 & 12;  // place of n0 + 4 i in a run of 16: (4 i) ^ h from b
#pragma unroll
            for (int i = 0; i < 4; ++i) v[8 * i] = b[(4 * i) ^ h];
            mirror_twiddles<8>(tw2 + k0, R1, [&](auto mc, float2 w) {
                constexpr int m = decltype(mc)::value;
#pragma unroll
                for (int i = 0; i < 4; ++i) v[8 * i + m] = cmul(b[((4 * i) ^ h) + 16 * m], w);
            });
            static_for<0, 4>([&](auto ic) { dft_inreg<32, 8, 8 * decltype(ic)::value, 1>(v); });
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k1 = 0; k1 < 8; ++k1) b[((4 * i) ^ h) + 16 * k1] = v[8 * i + k1];
        } else {
            // groups (n0, k0) and (n0 + 8, k0), n0 < 8, of one set of twiddles
            const int k0 = t >> 3, m0 = swz(k0);
            float2* const b = buf + S * k0 + ((t & 7) ^ (m0 & 7));
            const int lo = m0 & 8, hi = lo ^ 8;  // places of n0 < 8 and n0 >= 8 in a run of 16
            v[0] = b[lo];
            v[16] = b[hi];
            mirror_twiddles<16>(tw2 + k0, R1, [&](auto mc, float2 w) {
                constexpr int m = decltype(mc)::value;
                v[m] = cmul(b[lo + 16 * m], w);
                v[16 + m] = cmul(b[hi + 16 * m], w);
            });
            dft_inreg<32, 16, 0, 1>(v);
            dft_inreg<32, 16, 16, 1>(v);
#pragma unroll
            for (int k1 = 0; k1 < 16; ++k1) {
                b[lo + 16 * k1] = v[k1];
                b[hi + 16 * k1] = v[16 + k1];
            }
        }
        mirror_sync<LP>(lp);
        // ---------------- stage 3: groups g = t and G - t (thread 0: 0 and G/2)
        const int gb = t == 0 ? G / 2 : G - t;
        auto place = [&](int g) {
            const int d2 = g % R1;
            return S * d2 + 16 * (g / R1) + swz(d2);  // ^ n0
        };
        const int ia = place(t), ib = place(gb);
        v[0] = buf[ia];
        v[16] = buf[ib];
        mirror_twiddles<16>(tw3 + t, T, [&](auto mc, float2 w) {
            constexpr int m = decltype(mc)::value;
            v[m] = cmul(buf[ia ^ m], w);
            v[16 + m] = cmul(buf[ib ^ m], make_float2(w.x, -w.y));
        });
        if (t == 0) {
            // group G/2: W_P^{n0 G/2} = W_32^{n0}, and the shift's W_16^{-n0}
            static_for<1, 16>([&](auto nc) {
                constexpr int n0 = decltype(nc)::value;
                v[16 + n0] = twc<-n0, 32>(v[16 + n0]);
            });
        }
        __syncwarp();
        dft_inreg<32, 16, 0, 1>(v);
        dft_inreg<32, 16, 16, 1>(v);
    }

    // f(j, k, Z[k], Z[P - k]) for this thread's pairs but the one of slot 0:
    // j < 8 are bins t + G j and j >= 8 bins hi + G (j - 8), hi = t + 8 G.
    // Thread 0's groups pair with themselves (group 0: slots j and 16 - j;
    // group G/2, whose output i sits in slot 16 + (i + 1) mod 16: i and 15 - i,
    // hi = G/2); its values are selected into the same pairs, so that every
    // thread stores by the same code.  (A branch with stores of its own made
    // that warp a quarter longer than the others, which waited for it at the
    // barriers: window 2^12, overlap 0.5, 318 -> 292 us.)
    template <typename F>
    static __device__ __forceinline__ void for_pairs(const float2 (&v)[32], int t, F f)
    {
        const bool own = t == 0;
        const int hi = own ? G / 2 : t + 8 * G;
        auto sel = [&](const float2& x, const float2& y) { return make_float2(own ? x.x : y.x, own ? x.y : y.y); };
        static_for<1, 16>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            if constexpr (j < 8) f(jc, t + G * j, v[j], sel(v[16 - j], v[32 - j]));
            else f(jc, hi + G * (j - 8), sel(v[16 + j - 7], v[j]), sel(v[16 + ((24 - j) & 15)], v[32 - j]));
        });
    }
};

// Separates the pair of frames fa, fa + 1 and stores.
template <int EXP, int OUTK>
__device__ __forceinline__ void mirror_store_pair(const float2 (&v)[32], const FusedArgs& a, uint64_t fa, bool act_b, int t)
{
    using K = Mirror<EXP, true>;
    constexpr int N = K::N, H = K::H;
    float2* const o2 = reinterpret_cast<float2*>(a.out);
    const uint64_t fla = fa * (uint64_t)N, flb = fla + N;
    // reference half-complex layout: both frames lie below OHalfSize
    const bool whole = OUTK == OUT_HALF && act_b && flb + N <= a.ohalf;
    // bins k and N - k of both frames from Z[k] and Z[N - k]; self: k = N - k
    auto emit = [&](int k, float2 z, float2 pz, auto self_c) {
        constexpr bool self = decltype(self_c)::value;
        const float2 A = make_float2(z.x + pz.x, z.y - pz.y);  // frame a, bin k
        const float2 B = make_float2(z.y + pz.y, pz.x - z.x);  // frame b, bin k
        if constexpr (OUTK == OUT_POWER || OUTK == OUT_POWER_SERIAL) {
            float pa, pb;
            power_pair<OUTK>(A, B, pa, pb);
            if (!a.dense) {
                float* r = a.out + fla;
                __stcs(r + k, pa);
                if constexpr (!self) __stcs(r + (N - k), pa);
                if (act_b) {
                    __stcs(r + N + k, pb);
                    if constexpr (!self) __stcs(r + N + (N - k), pb);
                }
            } else {
                // the pair's bin in 0 .. N/2
                float* r = a.out + fa * (uint64_t)(H + 1) + (k <= H ? k : N - k);
                __stcs(r, pa);
                if (act_b) __stcs(r + (H + 1), pb);
            }
        } else {
            const float2 Ac = make_float2(A.x, -A.y), Bc = make_float2(B.x, -B.y);
            if (!a.dense) {
                auto put = [&](uint64_t flat, float2 x, bool act) {
                    if (whole || (act && flat < a.ohalf)) __stcs(o2 + flat, x);
                };
                put(fla + k, A, true);
                put(flb + k, B, act_b);
                if constexpr (!self) {
                    put(fla + (N - k), Ac, true);
                    put(flb + (N - k), Bc, act_b);
                }
            } else {
                const bool low = k <= H;
                float2* r = o2 + fa * (uint64_t)(H + 1) + (low ? k : N - k);
                __stcs(r, low ? A : Ac);
                if (act_b) __stcs(r + (H + 1), low ? B : Bc);
            }
        }
    };
    if (t != 0) {
        emit(t, v[0], v[16], std::false_type{});
    } else {
        emit(0, v[0], v[0], std::true_type{});
        emit(H, v[8], v[8], std::true_type{});
    }
    K::for_pairs(v, t, [&](auto, int k, float2 z, float2 pz) { emit(k, z, pz, std::false_type{}); });
}

// Untangles frame f and stores: X[k] = e + W_N^k o, X[P - k] = conj(e - W_N^k o).
// wt: W_N^t.
template <int EXP, int OUTK>
__device__ __forceinline__ void mirror_store_single(const float2 (&v)[32], const FusedArgs& a, uint64_t f, float2 wt, int t)
{
    using K = Mirror<EXP, false>;
    constexpr int N = K::N, M = K::H;
    float2* const o2 = reinterpret_cast<float2*>(a.out);
    const uint64_t fl = f * (uint64_t)N;
    const bool whole = OUTK == OUT_HALF && fl + N <= a.ohalf;
    // bins k, M - k, M + k, N - k from Z[k], Z[M - k] and w = W_N^k.
    // kind 0: those; 1: k = 0 (bins 0 and M); 2: k = M/2 (bins M/2 and 3M/2)
    auto emit = [&](int k, float2 z, float2 pz, float2 w, auto kind_c) {
        constexpr int kind = decltype(kind_c)::value;
        const float2 e = make_float2(z.x + pz.x, z.y - pz.y);
        const float2 wo = cmul(make_float2(z.y + pz.y, pz.x - z.x), w);
        const float2 X0 = cadd(e, wo);  // X[k]
        const float2 X1 = csub(e, wo);  // X[k + M] = conj X[M - k]
        if constexpr (OUTK == OUT_POWER || OUTK == OUT_POWER_SERIAL) {
            if (!a.dense) {
                const float p0 = power_of<OUTK>(X0), p1 = power_of<OUTK>(X1);
                float* r = a.out + fl;
                __stcs(r + k, p0);
                if constexpr (kind != 1) __stcs(r + (N - k), p0);
                if constexpr (kind != 2) __stcs(r + (M + k), p1);
                if constexpr (kind == 0) __stcs(r + (M - k), p1);
            } else {
                float p0, p1;
                power_pair<OUTK>(X0, X1, p0, p1);
                float* r = a.out + f * (uint64_t)(M + 1);
                __stcs(r + k, p0);
                if constexpr (kind != 2) __stcs(r + (M - k), p1);
            }
        } else {
            const float2 c0 = make_float2(X0.x, -X0.y), c1 = make_float2(X1.x, -X1.y);
            if (!a.dense) {
                auto put = [&](int b, float2 x) {
                    if (whole || fl + b < a.ohalf) __stcs(o2 + fl + b, x);
                };
                put(k, X0);
                if constexpr (kind != 1) put(N - k, c0);
                if constexpr (kind != 2) put(M + k, X1);
                if constexpr (kind == 0) put(M - k, c1);
            } else {
                float2* r = o2 + f * (uint64_t)(M + 1);
                __stcs(r + k, X0);
                if constexpr (kind != 2) __stcs(r + (M - k), kind == 1 ? X1 : c1);
            }
        }
    };
    if (t != 0) {
        emit(t, v[0], v[16], wt, std::integral_constant<int, 0>{});
    } else {
        emit(0, v[0], v[0], make_float2(1.0f, 0.0f), std::integral_constant<int, 1>{});
        emit(M / 2, v[8], v[8], make_float2(0.0f, -1.0f), std::integral_constant<int, 2>{});
    }
    // W_N^k: W_N^t W_32^j in slots j < 8, W_N^kHi W_32^(j - 8) above
    const float2 whi = t == 0 ? make_float2((float)cx_cos(kTwoPi / 64), -(float)cx_sin(kTwoPi / 64))
                              : twc<8, 32>(wt);
    K::for_pairs(v, t, [&](auto jc, int k, float2 z, float2 pz) {
        constexpr int j = decltype(jc)::value;
        emit(k, z, pz, j < 8 ? twc<j, 32>(wt) : twc<j - 8, 32>(whi), std::integral_constant<int, 0>{});
    });
}

// shared memory of a CTA, and group lp's parts of it
template <int EXP, bool PAIR>
struct MirrorSmem {
    float2* buf;  // the group's exchange buffer
    float2* tab;  // twiddle tables
    float* win;   // the window (mirror_smem_window)
    float2* red;  // the group's partial means
    __device__ __forceinline__ MirrorSmem(float2* smem, int lp)
    {
        constexpr int LP = mirror_lp(EXP, PAIR);
        buf = smem + ((size_t)lp << LP);
        tab = smem + ((size_t)mirror_gpc(LP) << LP);
        win = reinterpret_cast<float*>(tab + mirror_tab_size(LP));
        red = reinterpret_cast<float2*>(win + (mirror_smem_window(EXP) ? 1 << EXP : 0)) + lp * (mirror_T(LP) / 32);
    }
};

// Transform p of the request by the T threads of group lp: frames 2p and 2p + 1
// (those below a.frames), or frame p in the single form.
template <int EXP, bool PAIR, int OUTK>
__device__ __forceinline__ void mirror_transform(const FusedArgs& a, uint64_t p, const MirrorSmem<EXP, PAIR>& sm,
                                                 const float* win, int lp, int t)
{
    using K = Mirror<EXP, PAIR>;
    constexpr int LP = K::LP;
    const float2* const tw2 = sm.tab;
    const float2* const tw3 = sm.tab + mirror_tw2_size(LP);
    float2 v[32];
    const bool act_b = 2 * p + 1 < a.frames;  // pair form
    if constexpr (K::PAIR) K::load_pair(v, a, 2 * p, act_b, win, t);
    else K::load_single(v, a, p, win, t);
    if (a.remove_dc) K::remove_dc(v, sm.red, lp, t);
    // the exchange places are formed anew each time: kept over a loop of
    // transforms they would take some 40 registers
    int tf = t;
    asm volatile("" : "+r"(tf));
    K::fft(v, sm.buf, tw2, tw3, lp, tf);
    if constexpr (K::PAIR) mirror_store_pair<EXP, OUTK>(v, a, 2 * p, act_b, t);
    else mirror_store_single<EXP, OUTK>(v, a, p, tw3[mirror_tw3_size(LP) + t], t);
    __syncwarp();  // thread 0 stored on a branch of its own; the barriers want whole warps
}

// threads of a CTA for an output kind
__host__ __device__ constexpr int mirror_cta(int exp, int outk)
{
    return mirror_threads(mirror_lp(exp, mirror_paired(exp, outk)));
}

template <int EXP, int OUTK>
__global__ void __launch_bounds__(mirror_cta(EXP, OUTK), 512 / mirror_cta(EXP, OUTK))
stft_mirror_kernel(const FusedArgs a)
{
    using K = Mirror<EXP, mirror_paired(EXP, OUTK)>;
    constexpr int LP = K::LP, T = K::T, N = K::N, GPC = mirror_gpc(LP);
    constexpr int NT = mirror_threads(LP);
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const int lp = tid / T, t = tid - lp * T;
    const MirrorSmem<EXP, K::PAIR> sm(reinterpret_cast<float2*>(smem4), lp);
    pdl_trigger();
    for (int i = tid; i < mirror_tab_size(LP); i += NT) sm.tab[i] = a.tw[i];
    const float* win = a.win;
    if constexpr (mirror_smem_window(EXP)) {
        for (int i = tid; i < N / 2; i += NT)
            reinterpret_cast<float2*>(sm.win)[i] = reinterpret_cast<const float2*>(a.win)[i];
        win = sm.win;
    }
    __syncthreads();
    pdl_wait();
    constexpr int FPT = K::PAIR ? 2 : 1;  // frames per transform
    const uint64_t count = (a.frames + FPT - 1) / FPT;
    const uint64_t stride = (uint64_t)gridDim.x * GPC;
    for (uint64_t p = (uint64_t)blockIdx.x * GPC + lp; p < count; p += stride) {
        // the samples of this group's next transform start toward L2
        if (t == 0 && p + stride < count) {
            const uint64_t s0 = FPT * (p + stride) * a.hop, end = s0 + (FPT - 1) * a.hop + N;
            prefetch_l2_span(a.x, s0, end < a.n ? end : a.n);
        }
        mirror_transform<EXP, K::PAIR, OUTK>(a, p, sm, win, lp, t);
    }
}

}  // namespace ocs

namespace ocs {
template <int EXP, int OUTK>
cudaError_t launch_mirror_t(const FusedArgs& a, int grid, cudaStream_t st)
{
    constexpr size_t sm = mirror_smem_bytes(EXP, mirror_paired(EXP, OUTK));
    const cudaError_t e = ensure_smem_attr<stft_mirror_kernel<EXP, OUTK>>(sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(stft_mirror_kernel<EXP, OUTK>, grid, mirror_cta(EXP, OUTK), sm, st, a);
}

template <int EXP>
cudaError_t launch_mirror_exp(int outk, const FusedArgs& a, int grid, cudaStream_t st)
{
    switch (outk) {
    case OUT_POWER: return launch_mirror_t<EXP, OUT_POWER>(a, grid, st);
    case OUT_POWER_SERIAL: return launch_mirror_t<EXP, OUT_POWER_SERIAL>(a, grid, st);
    case OUT_HALF: return launch_mirror_t<EXP, OUT_HALF>(a, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int EXP, int OUTK>
int occupancy_mirror_t()
{
    int blocks = 0;
    constexpr size_t sm = mirror_smem_bytes(EXP, mirror_paired(EXP, OUTK));
    auto k = stft_mirror_kernel<EXP, OUTK>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, mirror_cta(EXP, OUTK), sm) != cudaSuccess)
        return 0;
    return blocks;
}

template <int EXP>
int occupancy_mirror_exp(int outk)
{
    switch (outk) {
    case OUT_POWER: return occupancy_mirror_t<EXP, OUT_POWER>();
    case OUT_POWER_SERIAL: return occupancy_mirror_t<EXP, OUT_POWER_SERIAL>();
    case OUT_HALF: return occupancy_mirror_t<EXP, OUT_HALF>();
    default: return 0;
    }
}

// defined in stft_mirror_lo.cu / stft_mirror_hi.cu
cudaError_t launch_mirror_lo(int exp, int outk, const FusedArgs& a, int grid, cudaStream_t st);
cudaError_t launch_mirror_hi(int exp, int outk, const FusedArgs& a, int grid, cudaStream_t st);
int occupancy_mirror_lo(int exp, int outk);
int occupancy_mirror_hi(int exp, int outk);
}  // namespace ocs

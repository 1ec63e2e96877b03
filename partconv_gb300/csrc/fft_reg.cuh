// fft_reg.cuh -- complex Stockham FFT with 16 points per thread in registers,
// for kernels that run many transforms at once.
//
// The transform is the one of fft_smem.cuh (radix-4 stages, then one radix-2
// stage when log2 N is odd) with two consecutive radix-4 stages taken per
// shared-memory round trip: the 16 points a[t + m N/16] of thread t are
// closed under the stages of size Ns and 4 Ns, so a pass reads them, runs
// both stages in registers and writes them back.  N = 256 crosses shared
// memory once instead of four times, N = 16384 three times instead of seven.
// Every butterfly does the operations of stage_r4 / stage_r2 on the same
// twiddle values in the same order, so the results equal fft_smem's bit for
// bit.
//
// Twiddles are read from one global table (build_fft_tables) in which every
// stage's factors lie contiguously, so the threads of a warp read consecutive
// entries (L1 hits); the values are those of the 2^wlog table.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "fft_smem.cuh"

namespace pcg {

constexpr int kRegMinLog = 4;    // 16 .. 16384 points
constexpr int kRegMaxLog = 14;

// ---- layout of the table (float2 entries) ---------------------------------------
// w1(s): exp(-2 pi i k / 4^(s+1)), k < 4^s, stages s = 1 .. 6
// w2(s), w3(s): its squares and cubes (blocks up to 1024 points read all three
//   factors; larger ones do with FULL, else they form them by products as
//   fft_smem's conflict-free stages do, with about one rounding more each)
// r2(a): exp(-2 pi i k / (2 4^a)), k < 4^a, a = 2 .. 6 (the radix-2 stage)
// sp(l): exp(-2 pi i k / 2^(l+1)), k <= 2^(l-1), l = 4 .. 14 (the real split)
__host__ __device__ constexpr int ft_pow4(int s) { return 1 << (2 * s); }
__host__ __device__ constexpr int ft_w1(int s) { return (ft_pow4(s) - 4) / 3; }                // sum of 4^j, 1 <= j < s
__host__ __device__ constexpr int ft_w2(int s) { return ft_w1(7) + (ft_pow4(s) - 4) / 3; }
__host__ __device__ constexpr int ft_w3(int s) { return ft_w2(7) + (ft_pow4(s) - 4) / 3; }
__host__ __device__ constexpr int ft_r2(int a) { return ft_w3(7) + (ft_pow4(a) - 16) / 3; }
__host__ __device__ constexpr int ft_sp(int l) { return ft_r2(7) + (1 << (l - 1)) - 8 + 2 * (l - 4); }
constexpr int kFftTabEntries = ft_sp(15);

// The entries for transforms up to 2^max_log points, from W[m] =
// exp(-2 pi i m / 2^wlog) (quarter-turn symmetry as in Twiddles::get, so the
// values are the ones fft_smem's stages use), by thread t of nt.
__host__ __device__ inline void fill_fft_tables(float2* tab, const float2* W, int wlog, int max_log, int t, int nt) {
    auto w = [&](long long a, int lg) {   // exp(-2 pi i a / 2^lg)
        const long long i = a << (wlog - lg);
        const int q = (int)(i >> (wlog - 2));
        const float2 v = W[(size_t)(i & ((1LL << (wlog - 2)) - 1))];
        const bool odd = (q & 1) != 0;
        const float sg = (q & 2) ? -1.0f : 1.0f;
        return make_float2(sg * (odd ? v.y : v.x), sg * (odd ? -v.x : v.y));
    };
    for (int s = 1; s <= 6 && 2 * s + 2 <= max_log; ++s)
        for (int k = t; k < ft_pow4(s); k += nt) {
            tab[ft_w1(s) + k] = w(k, 2 * s + 2);
            tab[ft_w2(s) + k] = w(2 * k, 2 * s + 2);
            tab[ft_w3(s) + k] = w(3 * k, 2 * s + 2);
        }
    for (int a = 2; a <= 6 && 2 * a + 1 <= max_log; ++a)
        for (int k = t; k < ft_pow4(a); k += nt) tab[ft_r2(a) + k] = w(k, 2 * a + 1);
    for (int l = kRegMinLog; l <= max_log; ++l)
        for (int k = t; k <= (1 << (l - 1)); k += nt) tab[ft_sp(l) + k] = w(k, l + 1);
}
inline std::vector<float2> build_fft_tables(const std::vector<float2>& W, int wlog) {
    std::vector<float2> tab((size_t)kFftTabEntries, make_float2(1.f, 0.f));
    fill_fft_tables(tab.data(), W.data(), wlog, kRegMaxLog, 0, 1);
    return tab;
}

// Shared-memory index of point i: one spare element per 16, so the strided
// writes of a pass (16 or 16 Ns apart) spread over the banks.
__device__ __forceinline__ int rpad(int i) { return i + (i >> 4); }

// Threads per transform, and the barrier among them (a named one per transform
// where a CTA of NT threads runs several, so transforms do not wait for one
// another; at most 16, 1024 threads / 64).
template <int LOGN, int NT>
struct RegFft {
    static constexpr int N = 1 << LOGN;
    static constexpr int TPT = N / 16;          // threads per transform
    static constexpr int SM = N + N / 16;       // shared float2 per transform
    __device__ static __forceinline__ void sync() {
        if constexpr (TPT <= 32) {
            __syncwarp();
        } else if constexpr (TPT == NT) {
            __syncthreads();
        } else if constexpr (2 * TPT == NT) {   // constant names: a CTA then holds two barriers, not sixteen
            if ((int)threadIdx.x < TPT) asm volatile("bar.sync 0, %0;" ::"n"(TPT) : "memory");
            else asm volatile("bar.sync 1, %0;" ::"n"(TPT) : "memory");
        } else {
            asm volatile("bar.sync %0, %1;" ::"r"((int)threadIdx.x / TPT), "n"(TPT) : "memory");
        }
    }
};

template <bool INV>
__device__ __forceinline__ float2 tw_dir(float2 w) {
    return INV ? make_float2(w.x, -w.y) : w;
}

template <bool INV>
__device__ __forceinline__ void bfly4(float2& v0, float2& v1, float2& v2, float2& v3) {
    const float2 a0 = cadd(v0, v2);
    const float2 a1 = csub(v0, v2);
    const float2 a2 = cadd(v1, v3);
    const float2 d = csub(v1, v3);
    const float2 a3 = INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
    v0 = cadd(a0, a2);
    v1 = cadd(a1, a3);
    v2 = csub(a0, a2);
    v3 = csub(a1, a3);
}

// the three factors of stage S (Ns = 4^S) at index k
template <int S, bool FULL, bool INV>
__device__ __forceinline__ void stage_tw(const float2* __restrict__ T, int k, float2& w1, float2& w2, float2& w3) {
    w1 = tw_dir<INV>(__ldg(T + ft_w1(S) + k));
    if constexpr (FULL) {
        w2 = tw_dir<INV>(__ldg(T + ft_w2(S) + k));
        w3 = tw_dir<INV>(__ldg(T + ft_w3(S) + k));
    } else {
        w2 = cmul(w1, w1);
        w3 = cmul(w2, w1);
    }
}

// Stages S and S + 1 on v[m] = a[t + m TPT]; afterwards v[r + 4 e] is the
// element 16 (t - k) + k + (r + 4 e) Ns, k = t mod Ns.
template <int LOGN, int NT, int S, bool INV, bool F>
__device__ __forceinline__ void pass16(float2 (&v)[16], int t, const float2* __restrict__ T) {
    constexpr int Ns = 1 << (2 * S);
    constexpr bool FULL = F || LOGN <= 10;   // all three factors of a butterfly from the table
    const int k = t & (Ns - 1);
    if constexpr (S > 0) {
        float2 w1, w2, w3;
        stage_tw<S, FULL, INV>(T, k, w1, w2, w3);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q + 4] = cmul(v[q + 4], w1);
            v[q + 8] = cmul(v[q + 8], w2);
            v[q + 12] = cmul(v[q + 12], w3);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) bfly4<INV>(v[q], v[q + 4], v[q + 8], v[q + 12]);   // v[q + 4 r]: output r of butterfly q
    float2 o[16];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float2 a0 = v[4 * r], a1 = v[4 * r + 1], a2 = v[4 * r + 2], a3 = v[4 * r + 3];
        if (S > 0 || r > 0) {
            float2 w1, w2, w3;
            stage_tw<S + 1, FULL, INV>(T, k + r * Ns, w1, w2, w3);
            a1 = cmul(a1, w1);
            a2 = cmul(a2, w2);
            a3 = cmul(a3, w3);
        }
        bfly4<INV>(a0, a1, a2, a3);
        o[r] = a0;
        o[r + 4] = a1;
        o[r + 8] = a2;
        o[r + 12] = a3;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = o[i];
}

// The last stages after the radix-16 passes, in place on v[m] = a[t + m TPT]
// (the results lie at the same places): radix 8 (4 then 2), 4 or 2.
template <int LOGN, int NT, bool INV, bool F>
__device__ __forceinline__ void pass_tail(float2 (&v)[16], int t, const float2* __restrict__ T) {
    constexpr int N4 = LOGN / 2, TPT = RegFft<LOGN, NT>::TPT;
    constexpr bool odd4 = (N4 & 1) != 0, r2 = (LOGN & 1) != 0;
    constexpr bool FULL = F || LOGN <= 10;   // all three factors of a butterfly from the table
    if constexpr (odd4) {   // the last radix-4 stage, Ns = 4^(N4 - 1)
        constexpr int S = N4 - 1;
        constexpr int Ns = 1 << (2 * S);
        // without a radix-2 stage after it Ns = N / 4: four butterflies t + g TPT;
        // with one Ns = N / 8: butterflies t + g TPT and N / 8 further, same factors
        constexpr int G = r2 ? 2 : 4;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2 w1, w2, w3;
            const int k = (t + g * TPT) & (Ns - 1);
            if constexpr (S > 0) stage_tw<S, FULL, INV>(T, k, w1, w2, w3);
#pragma unroll
            for (int q = 0; q < (r2 ? 2 : 1); ++q) {
                const int b = g + 2 * q;   // inputs b + 4 r
                if constexpr (S > 0) {
                    v[b + 4] = cmul(v[b + 4], w1);
                    v[b + 8] = cmul(v[b + 8], w2);
                    v[b + 12] = cmul(v[b + 12], w3);
                }
                bfly4<INV>(v[b], v[b + 4], v[b + 8], v[b + 12]);
            }
        }
        if constexpr (r2) {   // output r of butterfly (g, q) is element t + g TPT + r 2 TPT + q N / 2
            float2 o[16];
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 w = tw_dir<INV>(__ldg(T + ft_r2(N4) + t + g * TPT + r * 2 * TPT));
                    const float2 a = v[g + 4 * r], b = cmul(v[g + 2 + 4 * r], w);
                    o[g + 2 * r] = cadd(a, b);
                    o[g + 2 * r + 8] = csub(a, b);
                }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = o[i];
        }
    } else if constexpr (r2) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            const float2 w = tw_dir<INV>(__ldg(T + ft_r2(N4) + t + g * TPT));
            const float2 a = v[g], b = cmul(v[g + 8], w);
            v[g] = cadd(a, b);
            v[g + 8] = csub(a, b);
        }
    }
}

// write a radix-16 pass's results, read the next pass's points
template <int LOGN, int NT, int S>
__device__ __forceinline__ void exchange(float2 (&v)[16], int t, float2* s) {
    using F = RegFft<LOGN, NT>;
    constexpr int Ns = 1 << (2 * S);
    const int k = t & (Ns - 1);
    const int base = 16 * (t - k) + k;
#pragma unroll
    for (int i = 0; i < 16; ++i) s[rpad(base + i * Ns)] = v[i];
    F::sync();
#pragma unroll
    for (int m = 0; m < 16; ++m) v[m] = s[rpad(t + m * F::TPT)];
}

// N-point transform of one group of TPT threads: in and out v[m] = a[t + m TPT].
// s: this transform's shared memory (RegFft::SM float2), free on entry; a
// caller that writes it afterwards syncs first.  FULL: see the table above.
template <int LOGN, int NT, bool INV, bool FULL>
__device__ __forceinline__ void fft_reg(float2 (&v)[16], int t, float2* s, const float2* __restrict__ T) {
    using F = RegFft<LOGN, NT>;
    constexpr int NP = LOGN / 4;   // radix-16 passes (LOGN / 2 radix-4 stages in pairs)
    constexpr bool tail = (LOGN & 3) != 0;
    pass16<LOGN, NT, 0, INV, FULL>(v, t, T);
    if constexpr (NP > 1) {
        exchange<LOGN, NT, 0>(v, t, s);
        pass16<LOGN, NT, 2, INV, FULL>(v, t, T);
    }
    if constexpr (NP > 2) {
        F::sync();
        exchange<LOGN, NT, 2>(v, t, s);
        pass16<LOGN, NT, 4, INV, FULL>(v, t, T);
    }
    if constexpr (tail) {
        if constexpr (NP > 1) F::sync();
        exchange<LOGN, NT, 2 * (NP - 1)>(v, t, s);
        pass_tail<LOGN, NT, INV, FULL>(v, t, T);
    }
}

}  // namespace pcg

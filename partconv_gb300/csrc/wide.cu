// wide.cu -- block-parallel processing: a long call's base steps, many at once.
//
// pc_process and pc_process_device see all of a call's input at once, and
// nothing in partitioned convolution feeds back, so the blocks of every level
// can be computed side by side instead of one dependent launch per base
// block.  A chunk of base steps is
//   1. wide_fft   per block size: the window of every block that completes in
//                 the chunk, real FFT, spectrum ring row b mod slots;
//   2. wide_mac   all levels: Y_b = sum_p X_{b-p} H_p for runs of a few
//                 consecutive blocks per thread and bin, with the run's window
//                 of spectra in registers (each spectrum row is read once per
//                 run and part instead of once per block and part, each
//                 filter row once per run);
//   3. wide_ifft  per block size, level 0 last: inverse FFT, output ring, and
//                 for level 0 the sum of the levels' due samples and the output;
//   4. wide_mix   outputs fed by several PCs, in PC order.
// After the last chunk of a call the input rings and the partial sums of the
// blocks in progress are brought to where one-block steps would have left
// them (wide_ring, wide_partials), so pc_run can continue.
//
// Every block is computed with the float operations of the one-block steps
// (step_kernels.cu) in the same order -- same butterflies and twiddles
// (fft_reg.cuh), same grouping of the parts -- so a call's result does not
// depend on how its steps were executed, bit for bit.
//
// (the reference's counterpart of a long call is a loop over
// PartConvMulti::run, src/partconvMulti.cpp:815-928 of ebattenberg/partconv)
#include <cuda_runtime.h>

#include <algorithm>

#include "engine_types.h"
#include "fft_reg.cuh"
#include "kernels.h"
#include "wide.h"

namespace pcg {

namespace {

__device__ __forceinline__ int wmod(long long a, int m) {
    const long long r = a % m;
    return (int)(r < 0 ? r + m : r);
}

// blocks of level l completed before step c0, and during the chunk
__device__ __forceinline__ long long blocks_before(const WLevel& l, long long c) { return (c + l.s_blocks) >> l.logT; }

// ---------------------------------------------------------------------------
// 1. window, forward real FFT, spectrum row
// ---------------------------------------------------------------------------
template <int LOGN>
__global__ void __launch_bounds__(RegFft<LOGN>::NT) wide_fft_kernel(const int2* __restrict__ map, WArgs a) {
    using F = RegFft<LOGN>;
    constexpr int N = F::N, TPT = F::TPT;
    extern __shared__ float4 dyn_smem[];
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = reinterpret_cast<float2*>(dyn_smem) + tr * F::SM;
    const long long b0 = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - b0);
    if (e.y >= nb) return;                     // the whole CTA
    const bool live = e.y + tr < nb;
    const long long b = b0 + min(e.y + tr, nb - 1);
    // window [t_end - 2 N, t_end) of the channel; samples before t_in0 (the
    // call's first) are in the PC's input ring, already scaled
    const long long t_end = ((b + 1) << LOGN) - (long long)l.s_blocks * a.N0;
    const long long w0 = t_end - 2LL * N, t_in0 = a.io.step0 * (long long)a.N0;
    const float* in = a.io.in + (long long)l.in_ch * a.io.in_ch;
    const float scale = l.scale;
    float2 v[16];
    if (w0 >= t_in0 && a.vec_in) {
        const float2* p = reinterpret_cast<const float2*>(in + (w0 - t_in0));
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const float2 x = __ldg(p + t + m * TPT);
            v[m] = make_float2(x.x * scale, x.y * scale);
        }
    } else {
        const long long isamp = a.io.in_sample;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const long long ta = w0 + 2LL * (t + m * TPT);
            if (ta >= t_in0) {
                const float* p = in + (ta - t_in0) * isamp;
                v[m] = make_float2(p[0] * scale, p[isamp] * scale);
            } else {
                v[m] = __ldcg(reinterpret_cast<const float2*>(l.xring + (ta & l.rin_mask)));
            }
        }
    }
    fft_reg<LOGN, false>(v, t, s, a.tab);
    // the split pairs k < N / 2 (this thread's v[0 .. 7]) with N - k, which
    // lies in another thread's upper half
    F::sync();
#pragma unroll
    for (int m = 8; m < 16; ++m) s[rpad(t + m * TPT)] = v[m];
    F::sync();
    if (!live) return;
    float2* Xs = l.X + (size_t)wmod(b, l.slots) * l.cs;
    const float2* sp = a.tab + ft_sp(LOGN);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int k = t + m * TPT;
        float2 xk, xnk;
        if (m == 0 && t == 0) split_zero(v[0], xk, xnk);
        else split_w(v[m], s[rpad(N - k)], __ldg(sp + k), xk, xnk);
        Xs[k] = xk;
        Xs[N - k] = xnk;
    }
    if (t == 0) {
        float2 xk, xnk;
        split_w(v[8], v[8], __ldg(sp + N / 2), xk, xnk);
        Xs[N / 2] = xk;
    }
}

// ---------------------------------------------------------------------------
// 2. the sum over parts.  G: part groups per partial-sum row of the handle's
// spread tasks (the parts p_lo + q tp + g, + G, ... of row q form one running
// sum; a row is its groups added in order).
// ---------------------------------------------------------------------------
template <int G>
__global__ void __launch_bounds__(kWideMacNT) wide_mac_kernel(const int2* __restrict__ map, WArgs a, int tp) {
    constexpr int RB = wide_run(G);
    constexpr int U = G > 8 ? G : 8;   // parts per unrolled batch
    static_assert(U % RB == 0 && U % G == 0, "constant window rotation and groups");
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    const long long bf = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - bf);
    const int cs = l.cs, P = l.P, R = l.slots;
    const int item = e.y + threadIdx.x;
    const int run = item / cs, k = item - run * cs;
    const int i0 = run * RB;
    if (i0 >= nb) return;
    const float2* __restrict__ H = l.H + k;
    const float2* X = l.X + k;
    const int sl0 = wmod(bf + i0, R);
    // row of block (run's first) + d, -R <= d < R
    auto xat = [&](int d) {
        int sl = sl0 + d;
        if (sl < 0) sl += R;
        if (sl >= R) sl -= R;
        return __ldcg(X + (size_t)sl * cs);
    };
    const bool rows = P > l.p_lo;
    float2 y[RB];
    float2 part[RB];   // kFormFire: the part the fire adds to X_b H_0
    if (l.form == kFormMulti) {
        // p < p_lo in one running sum
#pragma unroll
        for (int j = 0; j < RB; ++j) y[j] = make_float2(0.f, 0.f);
        float2 w[RB];
#pragma unroll
        for (int j = 0; j < RB; ++j) w[j] = xat(j);
        const int Q = l.p_lo;
        for (int p0 = 0; p0 < Q; p0 += RB) {
            float2 h[RB], nx[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u)
                if (p0 + u < Q) {
                    h[u] = __ldg(H + (size_t)(p0 + u) * cs);
                    nx[u] = xat(-(p0 + u + 1));
                }
#pragma unroll
            for (int u = 0; u < RB; ++u)
                if (p0 + u < Q) {
#pragma unroll
                    for (int j = 0; j < RB; ++j) y[j] = cmac(y[j], w[(j - u + RB) % RB], h[u]);
                    w[(RB - 1 - u + RB) % RB] = nx[u];
                }
        }
    } else {
        const float2 h0 = __ldg(H);
        const bool x1 = l.two && P >= 2;
        float2 w[RB + 1];
#pragma unroll
        for (int j = 0; j < RB; ++j) w[j + 1] = xat(j);
        w[0] = x1 ? xat(-1) : make_float2(0.f, 0.f);
        const float2 h1 = x1 ? __ldg(H + cs) : make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            y[j] = cmul(w[j + 1], h0);
            part[j] = x1 ? cmul(w[j], h1) : make_float2(0.f, 0.f);
            if (l.form == kFormCluster && x1) y[j] = cadd(y[j], part[j]);
        }
    }
    if (rows) {
        float2 ys[RB];
        for (int q = 0; q < l.nrows; ++q) {
            const int pb = l.p_lo + q * tp, n = min(tp, P - pb);
            float2 acc[G][RB];
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int j = 0; j < RB; ++j) acc[g][j] = make_float2(0.f, 0.f);
            float2 w[RB];   // block (run's first) + d at w[d mod RB]
#pragma unroll
            for (int j = 0; j < RB; ++j) w[j] = xat(j - pb);
            for (int p0 = 0; p0 < n; p0 += U) {
                float2 h[U], nx[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (p0 + u < n) {
                        h[u] = __ldg(H + (size_t)(pb + p0 + u) * cs);
                        nx[u] = xat(-(pb + p0 + u + 1));
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (p0 + u < n) {
#pragma unroll
                        for (int j = 0; j < RB; ++j) acc[u % G][j] = cmac(acc[u % G][j], w[(j - u + U) % RB], h[u]);
                        w[(RB - 1 - u + U) % RB] = nx[u];
                    }
            }
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                float2 r = acc[0][j];
#pragma unroll
                for (int g = 1; g < G; ++g) r = cadd(r, acc[g][j]);
                if (l.form == kFormCluster) y[j] = cadd(y[j], r);
                else ys[j] = q == 0 ? r : cadd(ys[j], r);
            }
        }
        if (l.form == kFormFire) {
#pragma unroll
            for (int j = 0; j < RB; ++j) part[j] = cadd(part[j], ys[j]);
        } else if (l.form == kFormMulti) {
#pragma unroll
            for (int j = 0; j < RB; ++j) y[j] = cadd(y[j], ys[j]);
        }
    }
    float2* Y = l.Yw + (size_t)i0 * cs + k;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        if (i0 + j >= nb) break;
        if (l.form == kFormFire) y[j] = cadd(y[j], part[j]);
        Y[(size_t)j * cs] = y[j];
    }
}

// ---------------------------------------------------------------------------
// 3. inverse merge, inverse FFT, output ring or the call's output
// ---------------------------------------------------------------------------
template <int LOGN, bool L0>
__global__ void __launch_bounds__(RegFft<LOGN>::NT) wide_ifft_kernel(const int2* __restrict__ map, WArgs a) {
    using F = RegFft<LOGN>;
    constexpr int N = F::N, TPT = F::TPT;
    extern __shared__ float4 dyn_smem[];
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = reinterpret_cast<float2*>(dyn_smem) + tr * F::SM;
    const long long b0 = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - b0);
    if (e.y >= nb) return;
    const bool live = e.y + tr < nb;
    const int i = min(e.y + tr, nb - 1);
    const long long b = b0 + i;
    const float2* Y = l.Yw + (size_t)i * l.cs;
    const float2* sp = a.tab + ft_sp(LOGN);
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {   // Z'[n] from Y[n] and Y[N - n]
        const int n = t + m * TPT;
        float2 yn = __ldcg(Y + n), yc = __ldcg(Y + N - n);
        float2 other;
        if (m < 8) {
            if (m == 0 && t == 0) yn.y = yc.y = 0.0f;
            merge_w(yn, yc, __ldg(sp + n), v[m], other);
        } else {
            merge_w(yc, yn, __ldg(sp + N - n), other, v[m]);
        }
    }
    fft_reg<LOGN, true>(v, t, s, a.tab);
    if (!live) return;
    // real samples 2 n, 2 n + 1 of the block in v[m], n = t + m TPT < N / 2
    if constexpr (!L0) {
        const long long t0 = b << LOGN;
#pragma unroll
        for (int m = 0; m < 8; ++m)
            *reinterpret_cast<float2*>(l.yring + ((t0 + 2 * (t + m * TPT)) & l.rmask)) = v[m];
    } else {
        const long long t0 = b << LOGN;   // PC time = global time; N = N0, b = base step
        if (l.M > 1) {
            if constexpr (LOGN <= 10) {   // the larger levels' due samples summed first, then added
                float2 em[8];
                for (int L = 1; L < l.M; ++L) {
                    const WLevel& u = a.lv[l.lv0 + L];
                    const float* yr = u.yring;
                    const int mk = u.rmask;
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float2 y = __ldcg(reinterpret_cast<const float2*>(yr + ((t0 + 2 * (t + m * TPT)) & mk)));
                        em[m] = L == 1 ? y : cadd(em[m], y);
                    }
                }
#pragma unroll
                for (int m = 0; m < 8; ++m) v[m] = cadd(v[m], em[m]);
            } else {
                for (int L = 1; L < l.M; ++L) {
                    const WLevel& u = a.lv[l.lv0 + L];
                    const float* yr = u.yring;
                    const int mk = u.rmask;
#pragma unroll
                    for (int m = 0; m < 8; ++m)
                        v[m] = cadd(v[m], __ldcg(reinterpret_cast<const float2*>(yr + ((t0 + 2 * (t + m * TPT)) & mk))));
                }
            }
        }
        if (l.mix_mode == 2) {
            float2* o = reinterpret_cast<float2*>(l.pcw + ((size_t)i << LOGN));
#pragma unroll
            for (int m = 0; m < 8; ++m) o[t + m * TPT] = v[m];
        } else if (l.mix_mode == 1) {
            const long long os = a.io.out_sample;
            float* o = a.io.out + (long long)l.out_ch * a.io.out_ch + (t0 - a.io.step0 * (long long)a.N0) * os;
            if (a.vec_out) {
#pragma unroll
                for (int m = 0; m < 8; ++m) reinterpret_cast<float2*>(o)[t + m * TPT] = v[m];
            } else {
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    o[2LL * (t + m * TPT) * os] = v[m].x;
                    o[(2LL * (t + m * TPT) + 1) * os] = v[m].y;
                }
            }
        }
    }
}

// 4. outputs fed by several PCs (summed in PC order) and outputs without any
__global__ void wide_mix_kernel(Bank bank, int n_zero, int mixed, WArgs a) {
    const int len = a.nsteps * a.N0;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= len) return;
    const long long os = a.io.out_sample;
    float* o = a.io.out + ((a.c0 - a.io.step0) * (long long)a.N0 + j) * os;
    if (mixed)
        for (int ch = 0; ch < bank.n_out; ++ch) {
            const int q0 = bank.out_off[ch], q1 = bank.out_off[ch + 1];
            if (q1 - q0 < 2) continue;
            float v = 0.0f;
            for (int q = q0; q < q1; ++q) v += __ldcg(a.lv[bank.pcs[bank.out_pcs[q]].lv0].pcw + j);
            o[(long long)ch * a.io.out_ch] = v;
        }
    for (int z = 0; z < n_zero; ++z) o[(long long)bank.zero_list[z] * a.io.out_ch] = 0.0f;
}

// the call's newest samples (at most a ring's worth) to every PC's input ring
__global__ void wide_ring_kernel(const WLevel* __restrict__ lv, const int* __restrict__ lv0, WArgs a, long long t_end,
                                 long long frames) {
    const WLevel& l = lv[lv0[blockIdx.y]];
    const long long n = min(frames, (long long)l.rin_mask + 1);
    const float* in = a.io.in + (long long)l.in_ch * a.io.in_ch;
    const long long t_in0 = a.io.step0 * (long long)a.N0;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
        const long long ta = t_end - n + j;
        l.xring[ta & l.rin_mask] = in[(ta - t_in0) * a.io.in_sample] * l.scale;
    }
}

template <int LOGN>
size_t reg_smem() {
    return sizeof(float2) * (size_t)RegFft<LOGN>::SM * RegFft<LOGN>::TPC;
}

template <int LOGN>
cudaError_t prepare_one() {
    const int b = (int)reg_smem<LOGN>();
    cudaError_t e = cudaFuncSetAttribute(wide_fft_kernel<LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wide_ifft_kernel<LOGN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wide_ifft_kernel<LOGN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    return e;
}

// f.template operator()<LOGN>() for log2 N
template <class Fn>
cudaError_t by_log(int N, Fn&& f) {
    switch (N) {
        case 16: return f.template operator()<4>();
        case 32: return f.template operator()<5>();
        case 64: return f.template operator()<6>();
        case 128: return f.template operator()<7>();
        case 256: return f.template operator()<8>();
        case 512: return f.template operator()<9>();
        case 1024: return f.template operator()<10>();
        case 2048: return f.template operator()<11>();
        case 4096: return f.template operator()<12>();
        case 8192: return f.template operator()<13>();
        case 16384: return f.template operator()<14>();
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

int wide_transforms_per_cta(int N) { return N >= 2048 ? 1 : 2048 / N; }

struct WidePrepare {
    template <int L>
    cudaError_t operator()() const { return prepare_one<L>(); }
};
cudaError_t prepare_wide_kernels() {
    for (int N = 8192; N <= 16384; N *= 2) {   // the others fit the default shared memory
        cudaError_t e = by_log(N, WidePrepare{});
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

struct WideFft {
    int grid;
    const int2* map;
    const WArgs& a;
    cudaStream_t st;
    template <int L>
    cudaError_t operator()() const {
        wide_fft_kernel<L><<<grid, RegFft<L>::NT, reg_smem<L>(), st>>>(map, a);
        return cudaGetLastError();
    }
};
cudaError_t launch_wide_fft(int N, int grid, const int2* map, const WArgs& a, cudaStream_t st) {
    return grid > 0 ? by_log(N, WideFft{grid, map, a, st}) : cudaSuccess;
}

struct WideIfft {
    bool l0;
    int grid;
    const int2* map;
    const WArgs& a;
    cudaStream_t st;
    template <int L>
    cudaError_t operator()() const {
        if (l0) wide_ifft_kernel<L, true><<<grid, RegFft<L>::NT, reg_smem<L>(), st>>>(map, a);
        else wide_ifft_kernel<L, false><<<grid, RegFft<L>::NT, reg_smem<L>(), st>>>(map, a);
        return cudaGetLastError();
    }
};
cudaError_t launch_wide_ifft(int N, bool l0, int grid, const int2* map, const WArgs& a, cudaStream_t st) {
    return grid > 0 ? by_log(N, WideIfft{l0, grid, map, a, st}) : cudaSuccess;
}

cudaError_t launch_wide_mac(int G, int tp, int grid, const int2* map, const WArgs& a, cudaStream_t st) {
    if (grid <= 0) return cudaSuccess;
    switch (G) {
        case 1: wide_mac_kernel<1><<<grid, kWideMacNT, 0, st>>>(map, a, tp); break;
        case 2: wide_mac_kernel<2><<<grid, kWideMacNT, 0, st>>>(map, a, tp); break;
        case 4: wide_mac_kernel<4><<<grid, kWideMacNT, 0, st>>>(map, a, tp); break;
        case 8: wide_mac_kernel<8><<<grid, kWideMacNT, 0, st>>>(map, a, tp); break;
        case 16: wide_mac_kernel<16><<<grid, kWideMacNT, 0, st>>>(map, a, tp); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_wide_mix(const Bank& bank, int n_zero, bool mixed, const WArgs& a, cudaStream_t st) {
    const int len = a.nsteps * a.N0;
    wide_mix_kernel<<<(len + 255) / 256, 256, 0, st>>>(bank, n_zero, mixed ? 1 : 0, a);
    return cudaGetLastError();
}

cudaError_t launch_wide_ring(const WLevel* lv, const int* lv0, int npc, const WArgs& a, long long t_end,
                             long long frames, int max_ring, cudaStream_t st) {
    const long long n = std::min<long long>(frames, max_ring);
    for (int p = 0; p < npc; p += 65535) {
        const dim3 grid((unsigned)std::min<long long>((n + 1023) / 1024, 64), (unsigned)std::min(npc - p, 65535));
        wide_ring_kernel<<<grid, 256, 0, st>>>(lv, lv0 + p, a, t_end, frames);
    }
    return cudaGetLastError();
}

}  // namespace pcg

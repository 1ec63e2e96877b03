// wide.cu -- block-parallel processing: a long call's base steps, many at once.
//
// pc_process and pc_process_device see all of a call's input at once, and
// nothing in partitioned convolution feeds back, so the blocks of every level
// can be computed side by side instead of one dependent launch per base
// block.  A chunk of base steps is
//   1. wide_fft   all block sizes: the window of every block that completes in
//                 the chunk, real FFT, spectrum ring row b mod slots;
//   2. wide_mac   all levels: Y_b = sum_p X_{b-p} H_p, a tile of bins through
//                 a segment of blocks per CTA, filter and spectrum rows in
//                 shared memory and the window of a run of blocks in registers
//                 (each row is read once per segment instead of once per block
//                 and part);
//   3. wide_ifft  levels >= 1: inverse FFT, output ring;
//      wide_out   level 0: inverse FFT, the levels' due samples, the output;
//   4. wide_mix   outputs fed by several PCs, in PC order.
// After the last chunk of a call the input rings and the partial sums of the
// blocks in progress are brought to where one-block steps would have left
// them (wide_state_kernel in step_kernels.cu), so pc_run can continue.
//
// Every block is computed with the float operations of the one-block steps
// (step_kernels.cu) in the same order -- same butterflies and twiddles
// (fft_reg.cuh), same grouping of the parts -- so a call's result does not
// depend on how its steps were executed, bit for bit.
//
// The launches of a call overlap by programmatic dependent launch: a kernel
// reads its CTA map and level descriptor, which no kernel writes, and then
// waits for the kernel before it, in every CTA and before anything else.
//
// (the reference's counterpart of a long call is a loop over
// PartConvMulti::run, src/partconvMulti.cpp:815-928 of ebattenberg/partconv)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "engine_types.h"
#include "fft_reg.cuh"
#include "kernels.h"
#include "wide.h"

namespace pcg {

namespace {

__device__ __forceinline__ int wmod(long long a, int m) {
    if ((unsigned long long)a < 0x80000000ULL) return (int)((unsigned)a % (unsigned)m);   // a 32-bit division
    const long long r = a % m;
    return (int)(r < 0 ? r + m : r);
}

// blocks of level l completed before step c0, and during the chunk
__device__ __forceinline__ long long blocks_before(const WLevel& l, long long c) { return (c + l.s_blocks) >> l.logT; }

// ---------------------------------------------------------------------------
// 1. window, forward real FFT, spectrum row: one launch for all block sizes.
// A CTA of NT threads runs 16 NT / N transforms of one level; every CTA has
// the same amount of work whatever its block size.  Bound: shared-memory and
// L1 traffic of the radix-16 exchanges (L1 65 %, issue 54 % busy): 32 streams of
// 2^18 samples, blocks of 256 and 2048 in 54 us, of 16384 in 44 us, 200 MB of
// spectra written; the same transforms by one-block steps were part of a chain
// of 1024 launches of 3 us.
// ---------------------------------------------------------------------------
template <int LOGN, int NT, bool FULL>
__device__ __forceinline__ void fft_body(const WLevel& l, int first, const WArgs& a, float2* smem) {
    using F = RegFft<LOGN, NT>;
    constexpr int N = F::N, TPT = F::TPT;
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = smem + tr * F::SM;
    const long long b0 = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - b0);
    const bool live = first + tr < nb;
    if (TPT >= 32 && !live) return;            // whole warps, whole barriers
    const long long b = b0 + min(first + tr, nb - 1);
    // window [t_end - 2 N, t_end) of the channel; samples before t_in0 (the
    // call's first) are in the PC's input ring, already scaled
    const long long t_end = ((b + 1) << LOGN) - (long long)l.s_blocks * a.N0;
    const long long w0 = t_end - 2LL * N, t_in0 = a.io.step0 * (long long)a.N0;
    const float* in = a.io.in + (long long)l.in_ch * a.io.in_ch;
    const float scale = l.scale;
    float2 v[16];
    if (w0 >= t_in0 && a.vec_in && (a.len == 0 || t_end - t_in0 <= a.len)) {
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
                const long long i = ta - t_in0, left = a.len == 0 ? 2 : a.len - i;
                const float* p = in + i * isamp;
                v[m] = make_float2(left > 0 ? p[0] * scale : 0.0f, left > 1 ? p[isamp] * scale : 0.0f);
            } else if (l.xring) {
                v[m] = __ldcg(reinterpret_cast<const float2*>(l.xring + (ta & l.rin_mask)));
            } else {
                v[m] = make_float2(0.f, 0.f);
            }
        }
    }
    fft_reg<LOGN, NT, false, FULL>(v, t, s, a.tab);
    // the split pairs k < N / 2 (this thread's v[0 .. 7]) with N - k, which
    // lies in another thread's upper half
    F::sync();
#pragma unroll
    for (int m = 8; m < 16; ++m) s[rpad(t + m * TPT)] = v[m];
    F::sync();
    if (!live) return;
    float2* Xs = wide_at(l.X, a.rel) + (size_t)wmod(b, l.slots) * l.cs;
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

// f.template operator()<LOGN>() for log2 N, up to 16 NT points
template <int NT, class Fn>
__device__ __forceinline__ void by_log_dev(int logN, Fn&& f) {
    switch (logN) {
        case 4: f.template operator()<4>(); break;
        case 5: f.template operator()<5>(); break;
        case 6: f.template operator()<6>(); break;
        case 7: f.template operator()<7>(); break;
        case 8: f.template operator()<8>(); break;
        case 9: f.template operator()<9>(); break;
        case 10: f.template operator()<10>(); break;
        case 11: f.template operator()<11>(); break;
        default:
            if constexpr (NT == 256) {
                f.template operator()<12>();
            } else if constexpr (NT >= 1024) {
                if (logN == 12) f.template operator()<12>();
                else if (logN == 13) f.template operator()<13>();
                else f.template operator()<14>();
            }
    }
}

template <int NT, bool FULL>
struct FftBody {
    const WLevel& l;
    int first;
    const WArgs& a;
    float2* smem;
    template <int LOGN>
    __device__ __forceinline__ void operator()() const { fft_body<LOGN, NT, FULL>(l, first, a, smem); }
};
template <int NT, bool FULL>
__global__ void __launch_bounds__(NT) wide_fft_kernel(const int2* __restrict__ map, WArgs a) {
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    cudaGridDependencySynchronize();
    if (e.y >= (int)(blocks_before(l, a.c0 + a.nsteps) - blocks_before(l, a.c0))) return;
    by_log_dev<NT>(l.logN, FftBody<NT, FULL>{l, e.y, a, reinterpret_cast<float2*>(dyn_smem)});
}

// ---------------------------------------------------------------------------
// 2. the sum over parts: one thread per bin and run of RB consecutive blocks.
// ---------------------------------------------------------------------------
// One bin's column of a level in global memory: filter rows and spectrum
// rows, walked from one part to the next (offsets in elements).
struct MacCol {
    const float2* H;   // row of the part at hand
    const float2* X;
    int cs, wrap;      // row stride; ring size in elements
    int ox;            // spectrum of block (run's first) - p, for the part p at hand
    __device__ __forceinline__ int back(int o) const {   // the block before
        o -= cs;
        return o < 0 ? o + wrap : o;
    }
    __device__ __forceinline__ int fwd(int o) const {
        o += cs;
        return o >= wrap ? o - wrap : o;
    }
    __device__ __forceinline__ f32x2 x(int o) const { return __ldcg(reinterpret_cast<const f32x2*>(X + o)); }
    __device__ __forceinline__ float2 h() const { return __ldg(H); }
};

// Sums X_{b+j-p} H_p, j < RB, over n consecutive parts, last to first, in groups
// of tg, a group in running sums of `unit` parts (running sums added in order
// into the group, groups in order into row); c stands at the last part on entry.
// The run's RB spectra under part p stay in registers: part p - 1 needs one new
// one.  The loads of four parts go together.
template <int RB>
__device__ __forceinline__ void sum_parts(MacCol c, int n, int tg, int unit, f32x2 (&row)[RB]) {
    constexpr int U = 4;
    static_assert(RB % U == 0, "constant window rotation");
    f32x2 acc[RB], w[RB], ws[RB];   // window: block (run's first) + d - last part at w[d mod RB], and its swapped pairs
    f32x2 grp[RB];
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        row[j] = acc[j] = grp[j] = 0;
        w[j] = c.x(c.ox);
        ws[j] = swap2(w[j]);
        c.ox = c.fwd(c.ox);
    }
    int left = tg, run = unit;   // parts until the group and the running sum end
    for (int i0 = 0; i0 < n; i0 += RB) {
#pragma unroll
        for (int s = 0; s < RB / U; ++s) {
            if (i0 + s * U >= n) break;
            float2 h[U];
            f32x2 nx[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + s * U + u < n) {
                    h[u] = c.h();
                    c.H -= c.cs;
                    nx[u] = c.x(c.ox);   // (not used after the last one)
                    c.ox = c.fwd(c.ox);
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (i0 + s * U + u >= n) break;
                const int r = s * U + u;   // r-th part from the last, mod RB
                const f32x2 hr = pack2(h[u].x, h[u].x), hi = pack2(-h[u].y, h[u].y);
#pragma unroll
                for (int j = 0; j < RB; ++j) {
                    const int q = (j + r) % RB;
                    acc[j] = cmac2(acc[j], w[q], ws[q], hr, hi);
                }
                w[r % RB] = nx[u];
                ws[r % RB] = swap2(nx[u]);
                --left;
                if (--run == 0 || left == 0 || i0 + r + 1 == n) {
                    run = unit;
#pragma unroll
                    for (int j = 0; j < RB; ++j) {
                        grp[j] = add2(grp[j], acc[j]);
                        acc[j] = 0;
                    }
                    if (left == 0 || i0 + r + 1 == n) {
                        left = tg;
#pragma unroll
                        for (int j = 0; j < RB; ++j) {
                            row[j] = add2(row[j], grp[j]);
                            grp[j] = 0;
                        }
                    }
                }
            }
        }
    }
}

// row[j] = sum of X_{b+j-p} H_p over the first n parts, one by one with each
// product rounded before it is added (fire_multi's sum)
template <int RB>
__device__ __forceinline__ void chain_parts(MacCol c, int n, float2 (&y)[RB]) {
#pragma unroll
    for (int j = 0; j < RB; ++j) y[j] = make_float2(0.f, 0.f);
    for (int p = 0; p < n; ++p) {
        const float2 h = c.h();
        int o = c.ox;
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            y[j] = cadd(y[j], cmul(unpack2(c.x(o)), h));
            o = c.fwd(o);
        }
        c.H += c.cs;
        c.ox = c.back(c.ox);
    }
}

// y = X_b H_0 + (X_{b-1} H_1 + rows) for the run's blocks, c at part 0 (first:
// the run begins with block 0, before which there is silence)
template <int RB>
__device__ __forceinline__ void finish_run(const MacCol& c, const WLevel& l, const f32x2 (&ys)[RB], float2* Y,
                                           int live, bool first = false) {
    const bool rows = l.P > l.p_lo, x1 = l.two && l.P >= 2;
    const float2 h0 = c.h();
    const float2 h1 = x1 ? __ldg(c.H + c.cs) : make_float2(0.f, 0.f);
    float2 xm = x1 && !first ? unpack2(c.x(c.back(c.ox))) : make_float2(0.f, 0.f);
    int o = c.ox;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        const float2 x = unpack2(c.x(o));
        float2 s = unpack2(ys[j]);
        if (x1) s = rows ? cadd(cmul(xm, h1), s) : cmul(xm, h1);
        const float2 y = cadd(cmul(x, h0), s);
        if (j < live) Y[(size_t)j * l.cs] = y;
        xm = x;
        o = c.fwd(o);
    }
}

// (zeros when !on)
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool on = true) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// row[j] = sum of X_{b+j-p} H_p over n consecutive parts, last to first, in groups
// of four, from shared memory; x: the spectrum of the run's first block under the
// last of them, h: that part's row.  The window of a run under one part (RB spectra
// and their swapped pairs) stays in registers: the part before needs one new one.
// Shared rows are kMacTile apart, so every row is at a constant offset.  The
// loads of four parts go together (the spectrum after the first part is not used:
// it may be the shared row after the newest one).
template <int RB>
__device__ __forceinline__ void sum_groups(const f32x2* x, const float2* h, int n, f32x2 (&row)[RB]) {
    constexpr int U = 4, W = kMacTile;
    static_assert(RB % U == 0, "constant window rotation");
    f32x2 w[RB], ws[RB];   // the block of run index j under the r-th part from the last at w[(j + r) mod RB]
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        w[j] = x[j * W];
        ws[j] = swap2(w[j]);
    }
    for (int i0 = 0; i0 < n; i0 += RB, x += RB * W, h -= RB * W) {
#pragma unroll
        for (int s = 0; s < RB; s += U) {
            if (i0 + s >= n) break;
            float2 hv[U];
            f32x2 nx[U], acc[RB];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + s + u < n) {
                    hv[u] = h[-(s + u) * W];
                    nx[u] = x[(RB + s + u) * W];
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (i0 + s + u >= n) break;
                const f32x2 hr = pack2(hv[u].x, hv[u].x), hi = pack2(-hv[u].y, hv[u].y);
#pragma unroll
                for (int j = 0; j < RB; ++j) {
                    const int q = (j + s + u) % RB;
                    acc[j] = u == 0 ? fma2(ws[q], hi, mul2(w[q], hr)) : cmac2(acc[j], w[q], ws[q], hr, hi);
                }
                w[s + u] = nx[u];
                ws[s + u] = swap2(nx[u]);
            }
#pragma unroll
            for (int j = 0; j < RB; ++j) row[j] = i0 + s == 0 ? acc[j] : add2(row[j], acc[j]);
        }
    }
}

// Y = X_b H_0 + (X_{b-1} H_1 + row) for the run, X_{b-1} H_1 with x1 and the row
// with rows; x, h: the shared rows of the run's first block and of part 0.
// Products as cmul(X, H).
template <int RB>
__device__ __forceinline__ void mac_finish(const f32x2* x, const float2* h, bool x1, bool rows, const f32x2 (&row)[RB],
                                           float2* Y, int cs, int live) {
    constexpr int W = kMacTile;
    const float2 h0 = h[0], h1 = x1 ? h[W] : make_float2(0.f, 0.f);
    const f32x2 hr0 = pack2(h0.x, h0.x), hi0 = pack2(-h0.y, h0.y), hr1 = pack2(h1.x, h1.x), hi1 = pack2(-h1.y, h1.y);
    f32x2 xm = x1 ? x[-W] : 0, xms = swap2(xm);
    f32x2* y = reinterpret_cast<f32x2*>(Y);
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        const f32x2 xj = x[j * W], xs = swap2(xj);
        f32x2 s = row[j];
        if (x1) {
            const f32x2 m1 = fma2(xms, hi1, mul2(xm, hr1));
            s = rows ? add2(m1, s) : m1;
        }
        if (j < live) y[(size_t)j * cs] = add2(fma2(xs, hi0, mul2(xj, hr0)), s);
        xm = xj;
        xms = xs;
    }
}

// The default tiles: a CTA takes a tile of at most kMacTile bins of one level
// through a segment of kMacSeg blocks, kWideRun at a time, from shared memory.
// With at most kMacRes parts the filter rows of the tile stay there, and the
// segment's spectra with the P - 1 before them (up to 14 parts all 32, then 24)
// are all on their way before the first run is waited for; with more, every run
// takes the parts a partial-sum row at a time.
// Bound: latency, with twelve warps per SM: instructions are issued in 53 % of the
// cycles (stalls per issue: wait 1.6, long scoreboard 0.9), 41 % of them for the
// packed products (their pipe 45 % busy).  32 streams of 2^18 samples (14 | 14 |
// 1 .. 31 parts, 300 M products, 201 MB of spectra in and out): 154 us with rows
// in a ring of shared memory walked with wrapped offsets and the first two parts
// one float at a time, 136 us with constant offsets and packed ends; serialised
// 148 us first part to last, 142 us last to first.  Four CTAs per SM with 152
// registers a thread beat five with 128 (424 against 432 us for the call).
__global__ void __launch_bounds__(kMacTile, 4) wide_mac_kernel(const int4* __restrict__ map, WArgs a) {
    constexpr int RB = kWideRun, W = kMacTile;
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const int4 e = map[blockIdx.x];   // level, first bin, blocks [z, w) of the chunk
    const WLevel& l = a.lv[e.x];
    cudaGridDependencySynchronize();
    const long long bf = blocks_before(l, a.c0);
    const int nb = min(e.w, (int)(blocks_before(l, a.c0 + a.nsteps) - bf));
    if (e.z >= nb) return;
    const int cs = l.cs, P = l.P, R = l.slots, k0 = e.y;
    const int w2 = min(W, cs - k0) >> 1;   // pairs of bins in the tile
    const int tid = threadIdx.x, lr = tid / (W / 2), lc = tid % (W / 2);
    const bool live = tid < 2 * w2;
    const float2* Hg = wide_at(l.H, a.rel) + k0;
    const float2* Xg = wide_at(l.X, a.rel) + k0;
    float2* Y = wide_at(l.Yw, a.rel) + k0 + tid;
    int sl = wmod(bf, R) + e.z;   // ring row of block e.z of the chunk
    if (sl >= R) sl -= R;
    float2* Hs = reinterpret_cast<float2*>(dyn_smem);
    // filter rows [p, p + n) to shared rows dst ..
    auto copy_h = [&](float2* dst, int p, int n) {
        if (lc < w2)
            for (int i = lr; i < n; i += 2) cp_async16(dst + i * W + 2 * lc, Hg + (size_t)(p + i) * cs + 2 * lc);
    };
    // ring rows s + i (mod R), i0 <= i < i1, to shared rows dst + i; zeros for i < nz (blocks before 0)
    auto copy_x = [&](float2* dst, int s, int i0, int i1, int nz) {
        if (s < 0) s += R;
        if (lc < w2)
            for (int i = i0 + lr; i < i1; i += 2) {
                const int r = s + i;
                cp_async16(dst + i * W + 2 * lc, Xg + (size_t)(r >= R ? r - R : r) * cs + 2 * lc, i >= nz);
            }
    };
    if (P <= kMacRes) {
        float2* Xs = Hs + P * W;
        const int hist = P - 1;
        const int S = min(kMacSeg, (kMacRows - P - hist) & -RB);   // blocks whose spectra fit
        copy_h(Hs, 0, P);
        for (int s0 = e.z; s0 < nb; s0 += S) {
            const int n = min(S, nb - s0);
            const int nz = (int)max(0LL, hist - (bf + s0));
            if (s0 > e.z) __syncthreads();   // the rows before are still being read
#pragma unroll
            for (int g = 0; g < kMacSeg / RB; ++g) {
                copy_x(Xs, sl - hist, g == 0 ? 0 : hist + g * RB, hist + min((g + 1) * RB, n), nz);
                cp_async_commit();
            }
            const f32x2* x = reinterpret_cast<const f32x2*>(Xs + hist * W) + tid;
            float2* y = Y + (size_t)s0 * cs;
            for (int i = 0; i < n; i += RB, x += RB * W, y += (size_t)RB * cs) {
                switch (i / RB) {   // the copies of the later runs may be under way
                    case 0: cp_async_wait<kMacSeg / RB - 1>(); break;
                    case 1: cp_async_wait<kMacSeg / RB - 2>(); break;
                    case 2: cp_async_wait<kMacSeg / RB - 3>(); break;
                    default: cp_async_wait<0>();
                }
                __syncthreads();
                if (!live) continue;
                f32x2 row[RB];
#pragma unroll
                for (int j = 0; j < RB; ++j) row[j] = 0;
                if (P > l.p_lo) {
                    const int n1 = min(P, l.p_lo + kMacRes - 2);   // end of the first partial-sum row
                    sum_groups<RB>(x - (n1 - 1) * W, Hs + tid + (n1 - 1) * W, n1 - l.p_lo, row);
                    if (n1 < P) {   // (p_lo = 1: a part is left)
                        const float2 h = Hs[tid + n1 * W];
                        const f32x2 hr = pack2(h.x, h.x), hi = pack2(-h.y, h.y);
#pragma unroll
                        for (int j = 0; j < RB; ++j) {
                            const f32x2 xj = x[(j - n1) * W];
                            row[j] = add2(row[j], fma2(swap2(xj), hi, mul2(xj, hr)));
                        }
                    }
                }
                mac_finish<RB>(x, Hs + tid, l.two && P > 1, P > l.p_lo, row, y, cs, n - i);
            }
            sl += S;
            if (sl >= R) sl -= R;
        }
        return;
    }
    // shared rows: filter rows 0 and 1, the run's spectra and the one before them,
    // its partial sums so far, then the row of parts at hand
    constexpr int XH = 2, YS = XH + 1 + RB, HS = YS + RB;
    static_assert(HS + 2 * (kMacRes - 2) + RB <= kMacRows, "a partial-sum row's parts, and the row after them");
    f32x2* ys = reinterpret_cast<f32x2*>(Hs + YS * W) + tid;
    for (int i0 = e.z; i0 < nb; i0 += RB) {
        for (int q = 0; q < l.nrows; ++q) {
            const int pb = l.p_lo + q * l.tp, n = min(l.tp, P - pb);
            float2* Xs = Hs + (HS + n) * W;
            if (q == 0) {
                if (i0 == e.z) copy_h(Hs, 0, 2);
                copy_x(Hs + XH * W, sl - 1, 0, 1 + min(RB, nb - i0), bf + i0 == 0 ? 1 : 0);
            }
            // blocks (run's first) - pb - (n - 1) .. (run's first) - pb + RB - 1
            copy_h(Hs + HS * W, pb, n);
            // (before block 0 only in the first blocks of all: the ring holds no more than R of them)
            copy_x(Xs, sl - pb - (n - 1), 0, n - 1 + RB, (int)max(0LL, pb + n - 1 - (bf + i0)));
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            if (live) {
                f32x2 row[RB];
                sum_groups<RB>(reinterpret_cast<const f32x2*>(Xs) + tid, Hs + (HS + n - 1) * W + tid, n, row);
                if (q > 0) {
#pragma unroll
                    for (int j = 0; j < RB; ++j) row[j] = add2(ys[j * W], row[j]);
                }
                if (q + 1 < l.nrows) {
#pragma unroll
                    for (int j = 0; j < RB; ++j) ys[j * W] = row[j];
                } else {
                    mac_finish<RB>(reinterpret_cast<const f32x2*>(Hs + (XH + 1) * W) + tid, Hs + tid, l.two, true, row,
                                   Y + (size_t)i0 * cs, cs, nb - i0);
                }
            }
            __syncthreads();
        }
        sl += RB;
        if (sl >= R) sl -= R;
    }
}

// Other tile shapes and several base blocks per step: one thread per bin and
// run, rows from L2.
__global__ void __launch_bounds__(kMacAnyNT, 3) wide_mac_any_kernel(const int4* __restrict__ map, WArgs a) {
    constexpr int RB = kWideRun;
    cudaTriggerProgrammaticLaunchCompletion();
    const int4 e = map[blockIdx.x];   // level, first (run, bin) item
    const WLevel& l = a.lv[e.x];
    cudaGridDependencySynchronize();
    const long long bf = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - bf);
    const int cs = l.cs, P = l.P, R = l.slots;
    const int item = e.y + threadIdx.x;
    const int run = item / cs, k = item - run * cs;
    const int i0 = run * RB;
    if (i0 >= nb) return;
    int sl = wmod(bf, R) + i0;   // ring row of the run's first block
    if (sl >= R) sl -= R;
    MacCol c{l.H + k, l.X + k, cs, R * cs, 0};
    f32x2 ys[RB];   // partial-sum rows of the parts >= p_lo
#pragma unroll
    for (int j = 0; j < RB; ++j) ys[j] = 0;
    const bool rows = P > l.p_lo;
    if (rows) {
        for (int q = 0; q < l.nrows; ++q) {
            f32x2 row[RB];
            const int n = min(l.tp, P - l.p_lo - q * l.tp), p = l.p_lo + q * l.tp + n - 1;   // the row's last part
            c.H = l.H + (size_t)p * cs + k;
            c.ox = (sl < p ? sl - p + R : sl - p) * cs;
            sum_parts<RB>(c, n, l.tpg, l.multi ? 2 : 4, row);
#pragma unroll
            for (int j = 0; j < RB; ++j) ys[j] = q == 0 ? row[j] : add2(ys[j], row[j]);
        }
    }
    c.H = l.H + k;
    c.ox = sl * cs;
    float2* Y = l.Yw + (size_t)i0 * cs + k;
    if (l.multi) {   // parts < p_lo one by one
        float2 y[RB];
        chain_parts<RB>(c, l.p_lo, y);
#pragma unroll
        for (int j = 0; j < RB; ++j)
            if (i0 + j < nb) Y[(size_t)j * cs] = rows ? cadd(y[j], unpack2(ys[j])) : y[j];
    } else {
        finish_run(c, l, ys, Y, nb - i0);
    }
}

// ---------------------------------------------------------------------------
// 3. inverse merge, inverse FFT, output ring (levels >= 1, one launch for all
// block sizes) or the call's output (level 0, after them).  Bound: as the
// forward transforms, the output also by the latency of the levels' due
// samples: 32 streams of 2^18 samples 39 (2048), 44 (16384) and 38 us (output).
// ---------------------------------------------------------------------------
template <int LOGN, int NT, bool L0, bool FULL>
__device__ __forceinline__ void ifft_body(const WLevel& l, int first, const WArgs& a, float2* smem) {
    using F = RegFft<LOGN, NT>;
    constexpr int N = F::N, TPT = F::TPT;
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = smem + tr * F::SM;
    const long long b0 = blocks_before(l, a.c0);
    const int nb = (int)(blocks_before(l, a.c0 + a.nsteps) - b0);
    const bool live = first + tr < nb;
    if (TPT >= 32 && !live) return;
    const int i = min(first + tr, nb - 1);
    const long long b = b0 + i;
    const float2* Y = wide_at(l.Yw, a.rel) + (size_t)i * l.cs;
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
    fft_reg<LOGN, NT, true, FULL>(v, t, s, a.tab);
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
            const long long left = a.len == 0 ? N : a.len - (t0 - a.io.step0 * (long long)a.N0);   // samples of the block to write
            if (left < N) {
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const long long i = 2 * (t + m * TPT);
                    if (i < left) o[i * os] = v[m].x;
                    if (i + 1 < left) o[(i + 1) * os] = v[m].y;
                }
            } else if (a.vec_out) {
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

template <int NT, bool FULL>
struct IfftBody {
    const WLevel& l;
    int first;
    const WArgs& a;
    float2* smem;
    template <int LOGN>
    __device__ __forceinline__ void operator()() const { ifft_body<LOGN, NT, false, FULL>(l, first, a, smem); }
};
template <int NT, bool FULL>
__global__ void __launch_bounds__(NT) wide_ifft_kernel(const int2* __restrict__ map, WArgs a) {
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    cudaGridDependencySynchronize();
    if (e.y >= (int)(blocks_before(l, a.c0 + a.nsteps) - blocks_before(l, a.c0))) return;
    by_log_dev<NT>(l.logN, IfftBody<NT, FULL>{l, e.y, a, reinterpret_cast<float2*>(dyn_smem)});
}

__host__ __device__ constexpr int out_threads(int logN) { return logN <= 11 ? 128 : 1 << (logN - 4); }
template <int LOGN, bool FULL>
__global__ void __launch_bounds__(out_threads(LOGN)) wide_out_kernel(const int2* __restrict__ map, WArgs a) {
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const int2 e = map[blockIdx.x];
    const WLevel& l = a.lv[e.x];
    cudaGridDependencySynchronize();
    if (e.y >= a.nsteps) return;
    ifft_body<LOGN, out_threads(LOGN), true, FULL>(l, e.y, a, reinterpret_cast<float2*>(dyn_smem));
}

// 0. interleaved input, frames of C samples, to rows of one channel each
// (pitch apart).  Each channel is read by every level of every PC on it, twice
// per window; from the interleaved frames those reads touch C times the memory
// they use.  A tile of up to 32 channels, 1024 samples at most, goes through
// shared memory.  Bound: the latency of one load and one store (6 inputs,
// 128128 frames: 3 us; the transforms of 12 paths after it 24 us instead of
// 37).
__host__ __device__ constexpr int planar_frames(int cw) { return 1024 / cw & ~31; }
__global__ void __launch_bounds__(256) wide_planar_kernel(const float* __restrict__ in, float* __restrict__ out, int C,
                                                          long long pitch, long long frames) {
    __shared__ float tile[1024 + 1024 / 2];   // frames cw | 1 apart
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int c0 = blockIdx.y * 32, cw = min(32, C - c0), F = planar_frames(min(32, C)), ld = cw | 1;
    const long long f0 = (long long)blockIdx.x * F;
    const int nf = (int)min((long long)F, frames - f0);
    const float* src = in + f0 * C + c0;
    float* dst = out + c0 * pitch + f0;
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = threadIdx.x + u * 256, f = i / cw, c = i - f * cw;
        if (f < nf) v[u] = __ldg(src + (long long)f * C + c);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = threadIdx.x + u * 256, f = i / cw, c = i - f * cw;
        if (f < nf) tile[f * ld + c] = v[u];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = threadIdx.x + u * 256, c = i / F, f = i - c * F;
        if (c < cw && f < nf) dst[c * pitch + f] = tile[f * ld + c];
    }
}

// 4. outputs fed by several PCs (summed in PC order) and outputs without any
__global__ void wide_mix_kernel(Bank bank, int n_zero, int mixed, WArgs a) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
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

// What a run from the start reads before writing it: the spectrum rows of
// the P - 1 blocks before the first one, and the output ring up to the first
// block's samples (the rest of both is written first); and the state region
// of n16 16-byte words, cleared by the CTAs after the levels'.
__global__ void wide_reset_kernel(const WLevel* __restrict__ lv, int nlv, float4* state, size_t n16) {
    const int nt = gridDim.y * blockDim.x, t = blockIdx.y * blockDim.x + threadIdx.x;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((int)blockIdx.x >= nlv) {
        const size_t step = (size_t)(gridDim.x - nlv) * nt;
        for (size_t i = (size_t)(blockIdx.x - nlv) * nt + t; i < n16; i += step) state[i] = z;
        return;
    }
    const WLevel& l = lv[blockIdx.x];
    const long long b0 = blocks_before(l, 0);
    const long long n4 = l.cs >> 1, ring = l.slots * n4;   // float4 per row (rows are 16-byte aligned) and ring
    const long long first = wmod(b0 - (l.P - 1), l.slots) * n4;
    float4* X = reinterpret_cast<float4*>(l.X);
    for (long long i = t; i < (l.P - 1) * n4; i += nt) X[first + i < ring ? first + i : first + i - ring] = z;
    const int ny = (int)min((long long)l.rmask + 1, b0 << l.logN) >> 2;
    for (int i = t; i < ny; i += nt) reinterpret_cast<float4*>(l.yring)[i] = z;
}

// What a step c from which the rings go on reads of them: the spectrum rows of
// the P - 1 blocks before its first one and the output ring from its first sample
// to the last block's end, from the rings of lv to those of to.
__global__ void wide_move_kernel(const WLevel* __restrict__ lv, const WLevel* __restrict__ to, long long c, int N0) {
    const int nt = gridDim.y * blockDim.x, t = blockIdx.y * blockDim.x + threadIdx.x;
    const WLevel &l = lv[blockIdx.x], &m = to[blockIdx.x];
    const long long b0 = blocks_before(l, c);
    const int n4 = l.cs >> 1;
    int sl = wmod(b0, l.slots), sm = wmod(b0, m.slots);
    for (int p = 1; p < l.P; ++p) {
        sl = sl == 0 ? l.slots - 1 : sl - 1;
        sm = sm == 0 ? m.slots - 1 : sm - 1;
        const float4* src = reinterpret_cast<const float4*>(l.X + (size_t)sl * l.cs);
        float4* dst = reinterpret_cast<float4*>(m.X + (size_t)sm * l.cs);
        for (int i = t; i < n4; i += nt) dst[i] = __ldcg(src + i);
    }
    const long long end = l.yring ? b0 << l.logN : 0;
    for (long long x = c * N0 + 4LL * t; x < end; x += 4LL * nt)
        *reinterpret_cast<float4*>(m.yring + (x & m.rmask)) = __ldcg(reinterpret_cast<const float4*>(l.yring + (x & l.rmask)));
}

// launch that may overlap the previous kernel's tail (see above)
template <class... KA, class... A>
cudaError_t launch_dep(void (*k)(KA...), dim3 grid, int nt, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, KA(args)...);
}

// shared memory of a CTA of nt threads, 16 points each
constexpr size_t fft_smem_of(int nt) { return sizeof(float2) * 17 * (size_t)nt; }

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

template <class K>
cudaError_t allow_smem(K* k, int nt) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fft_smem_of(nt));
}
struct OutPrepare {
    template <int L>
    cudaError_t operator()() const {
        const cudaError_t e = allow_smem(wide_out_kernel<L, false>, out_threads(L));
        return e == cudaSuccess ? allow_smem(wide_out_kernel<L, true>, out_threads(L)) : e;
    }
};

}  // namespace

static std::vector<float2> make_twiddles(int wlog) {
    std::vector<float2> W((size_t)1 << wlog);
    for (size_t m = 0; m < W.size(); ++m) {
        const double a = -2.0 * M_PI * (double)m / (double)W.size();
        W[m] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    return W;
}
const std::vector<float2>& host_twiddles(int wlog) {
    static const std::vector<float2> w15 = make_twiddles(15), w17 = make_twiddles(17);
    return wlog == 15 ? w15 : w17;
}
const std::vector<float2>& host_fft_tables() {
    static const std::vector<float2> t = build_fft_tables(host_twiddles(15), 15);
    return t;
}

static __global__ void fft_tables_kernel(float2* tab, const float2* W, int wlog) {
    fill_fft_tables(tab, W, wlog, kRegMaxLog, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
cudaError_t launch_fft_tables(float2* tab, const float2* W, int wlog, cudaStream_t st) {
    fft_tables_kernel<<<32, 256, 0, st>>>(tab, W, wlog);
    return cudaGetLastError();
}

cudaError_t prepare_wide_kernels() {
    cudaError_t e = allow_smem(wide_fft_kernel<1024, false>, 1024);
    if (e == cudaSuccess) e = allow_smem(wide_fft_kernel<1024, true>, 1024);
    if (e == cudaSuccess) e = allow_smem(wide_ifft_kernel<1024, false>, 1024);
    if (e == cudaSuccess) e = allow_smem(wide_ifft_kernel<1024, true>, 1024);
    for (int N = 8192; N <= 16384 && e == cudaSuccess; N *= 2) e = by_log(N, OutPrepare{});
    return e;
}

int wide_threads(int max_n) { return max_n <= 2048 ? 128 : 1024; }
int wide_out_blocks(int N0) { return N0 <= 2048 ? 2048 / N0 : 1; }

template <int NT, bool FULL>
static cudaError_t launch_fft(bool inverse, bool dep, int grid, const int2* map, const WArgs& a, cudaStream_t st) {
    if (inverse) {
        if constexpr (NT != 256) return launch_dep(wide_ifft_kernel<NT, FULL>, grid, NT, fft_smem_of(NT), st, map, a);
        return cudaErrorInvalidValue;
    }
    if (dep) return launch_dep(wide_fft_kernel<NT, FULL>, grid, NT, fft_smem_of(NT), st, map, a);
    wide_fft_kernel<NT, FULL><<<grid, NT, fft_smem_of(NT), st>>>(map, a);
    return cudaGetLastError();
}
cudaError_t launch_wide_fft(bool inverse, int nt, int grid, const int2* map, const WArgs& a, cudaStream_t st, bool dep) {
    if (grid <= 0) return cudaSuccess;
    if (nt == 256) return launch_fft<256, true>(inverse, dep, grid, map, a, st);
    if (nt == 128)
        return a.full ? launch_fft<128, true>(inverse, dep, grid, map, a, st)
                      : launch_fft<128, false>(inverse, dep, grid, map, a, st);
    return a.full ? launch_fft<1024, true>(inverse, dep, grid, map, a, st)
                  : launch_fft<1024, false>(inverse, dep, grid, map, a, st);
}

struct WideOut {
    int grid;
    const int2* map;
    const WArgs& a;
    cudaStream_t st;
    template <int L>
    cudaError_t operator()() const {
        // (blocks up to 1024 read every factor from the table either way)
        return L > 10 && a.full ? launch_dep(wide_out_kernel<L, true>, grid, out_threads(L), fft_smem_of(out_threads(L)), st, map, a)
                                : launch_dep(wide_out_kernel<L, false>, grid, out_threads(L), fft_smem_of(out_threads(L)), st, map, a);
    }
};
cudaError_t launch_wide_out(int N0, int grid, const int2* map, const WArgs& a, cudaStream_t st) {
    return grid > 0 ? by_log(N0, WideOut{grid, map, a, st}) : cudaSuccess;
}

constexpr size_t kMacSmem = sizeof(float2) * kMacTile * (size_t)kMacRows;
static_assert(kMacSeg == 4 * kWideRun, "four groups of copies");
static_assert(kMacRows >= 2 * kMacRes - 1 + kWideRun, "a run of the longest resident level");

cudaError_t launch_wide_mac(bool any, int grid, const int4* map, const WArgs& a, cudaStream_t st) {
    if (grid <= 0) return cudaSuccess;
    return any ? launch_dep(wide_mac_any_kernel, grid, kMacAnyNT, 0, st, map, a)
               : launch_dep(wide_mac_kernel, grid, kMacTile, kMacSmem, st, map, a);
}

cudaError_t launch_wide_mix(const Bank& bank, int n_zero, bool mixed, const WArgs& a, cudaStream_t st) {
    const int len = a.nsteps * a.N0;
    return launch_dep(wide_mix_kernel, (len + 255) / 256, 256, 0, st, bank, n_zero, mixed ? 1 : 0, a);
}

cudaError_t launch_wide_planar(const float* in, float* out, int channels, long long pitch, long long frames,
                               cudaStream_t st) {
    const int F = planar_frames(std::min(32, channels));
    return launch_dep(wide_planar_kernel, dim3((unsigned)((frames + F - 1) / F), (unsigned)((channels + 31) / 32)), 256, 0,
                      st, in, out, channels, pitch, frames);
}

cudaError_t launch_wide_move(const WLevel* lv, const WLevel* to, int nlv, long long step, int N0, cudaStream_t st) {
    wide_move_kernel<<<dim3(nlv, nlv > 512 ? 4 : 64), 256, 0, st>>>(lv, to, step, N0);
    return cudaGetLastError();
}

cudaError_t launch_wide_reset(const WLevel* lv, int nlv, size_t level_bytes, void* state, size_t bytes, cudaStream_t st) {
    // gy CTAs for each level, 64 KB of the largest one for each (64 for each level:
    // 32 us per reset of 64 streams of 64 | 512; so 15 us, an empty kernel being 10)
    const int gy = (int)std::min<size_t>(std::max<size_t>(1, (level_bytes + 65535) >> 16), nlv > 512 ? 4 : 64);
    const int extra = (int)std::min<size_t>(64, bytes / ((size_t)gy << 14) + 1);
    wide_reset_kernel<<<dim3(nlv + extra, gy), 256, 0, st>>>(lv, nlv, static_cast<float4*>(state), bytes >> 4);
    return cudaGetLastError();
}

}  // namespace pcg

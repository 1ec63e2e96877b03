// mimo.cu -- n_in x n_out MIMO partitioned convolution with per-bin channel
// sums: y_o = sum_i x_i * h_{i,o} over every (input, output) path.
//
// The reference would run one PartConvFilter per path and sum the outputs in
// time (src/partconvMulti.cpp:911-921), recomputing each input's spectrum for
// every output.  Here every input's block spectrum is computed once per
// level block and each output's FDL sums over inputs per bin:
//   Y_o[k] = sum_i sum_p X_i[b-p][k] H_{i,o,p}[k],
// followed by one inverse FFT per output and level block.  The level
// schedule is the engine's minimum-latency one (matlab/MFDL_part_conv.m
// structure; layouts must pass its relaxed check).
//
// A base step is three kernels (programmatic dependent launches):
//   K1 input FFTs     -- every (input, level) whose block completes: window,
//                        real FFT, spectrum ring slot b mod P (level 0 also
//                        appends the step's samples to the input ring);
//   K2 MAC tasks      -- fire sums for the (output, level) blocks due now:
//                        Yf_o = sum_i X_i[b] H_{i,o,0} (+ X_i[b-1] H_{i,o,1}
//                        for level 0) + the partial sums; and spread tasks
//                        that build the partial sums over the older parts for
//                        later blocks, split by output, bin tile and input
//                        range (reduced in a fixed order when consumed);
//   K3 output IFFTs   -- inverse FFT of Yf_o, output ring (levels >= 1) or
//                        the step's output: level 0 plus the due slices of
//                        the other levels, in level order.
// H is streamed once per block: the MAC is bound by HBM bandwidth.  It is
// stored tile-major, [output][bin tile][input][part][bins of the tile], with
// each level's bins cut into fixed tiles (the bin slices the MAC tasks take),
// so one MAC task streams one contiguous range of H (about 40 KB: its inputs'
// rows of the tile, parts adjacent, in the order it sums them) instead of a
// 0.4 KB segment of every (input, part) row.
//
// A call of many base steps runs block-parallel (wide.cu's transforms): the
// sum over inputs and parts is then, per bin, a product of the outputs' filter
// matrix with the spectra of many blocks, and H is read once per chunk of
// blocks instead of once per block (mimo_wide_mac_kernel).  It reads a second
// copy of H laid out for it, Hw: [output pair][tile of kTile bins][input][part]
// [bins of the tile] of (re0, re1, im0, im1), operands of packed (f32x2)
// multiply-adds as they lie (an odd last output is paired with zeros).  The first
// such call makes that copy and the rings and sums of its chunks (ensure_wide); a
// handle of short calls holds neither.  One
// layout for both was slower for one of them: the one-block kernel on the
// pairs ran 29.7 instead of 25.5 us per launch, the block-parallel one on the
// tiles of single outputs 727 instead of 640 us per 128 blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/partconv_gb300.h"
#include "engine_types.h"
#include "fft_reg.cuh"
#include "kernels.h"
#include "wide.h"

using namespace pcg;

namespace {

constexpr int kWlog = 15;
constexpr int kMacNT = 128;        // MAC CTA: threads = (bin-pair column, term group) pairs
constexpr int kMacMaxBins = 128;   // widest bin tile (64 columns of two bins: two term groups)
constexpr int kTile = 32;          // bins per tile of Hw (a warp's lanes); a row's last two bins, N
                                   // and its padding, belong to the tile before them
constexpr int kMaxMimoLevels = 8;
constexpr int kMaxMacTerms = 2048;  // (input, part) terms one MAC task sums
// block-parallel calls: from this many base steps on (small matrices would gain
// from four: block-parallel and one-block steps, 128x16 | 2048xP, 4, 8 and 16
// steps: 4 x 4 paths of 6001 taps 36, 41, 45 and 39, 70, 124 us; 32 x 32 of 2^15
// taps 101, 133, 141 and 64, 125, 231 us).  A level whose blocks take more steps
// than that is read twice in calls so short, once for the partial sums of the block
// in progress and as a whole when it completes: a step later per kWideStepBytes of
// its spectra (64 x 64 paths, 128x16 | 2048x15, 1 GB: 10, 14, 15 and 16 steps 389,
// 446, 460, 434 and 292, 407, 434, 464 us; 32 x 32, 0.25 GB: 10, 11 and 12 steps
// 152, 157, 155 and 139, 152, 165 us)
constexpr int kWideMinSteps = 10;
constexpr double kWideStepBytes = 165e6;
// base steps per chunk: as many as keep the chunk's spectra within kWideBytes
constexpr size_t kWideBytes = (size_t)64 << 20;
constexpr int kWideMinChunk = 32, kWideMaxChunk = 4096;
constexpr int kOB = 4;             // outputs a warp sums together
constexpr int kBB = 8;             // ... and consecutive blocks
constexpr int kSegBlocks = 2 * kBB;   // blocks per CTA of mimo_wide_mac_kernel (8, 16 or 32)

struct MLevel {
    int N, logN, P, T, s_blocks, cs, rmask, npart;
    int ntile;           // bin tiles of a row of H
    const int* tstart;   // [ntile + 1]: first bin of each tile (the last entry is cs)
    int slots;      // rows of an input's spectrum ring (block b in row b mod slots)
    int nbw;        // most blocks of a block-parallel chunk
    float2* H;      // [nO][tile][nI][P][tile width]
    float4* Hw;     // [output pair][tile of kTile][nI][P][tile width] (null before the first block-parallel call)
    float2* X;      // [nI][slots][cs]
    float2* Yp;     // [nO][npart][2][cs]
    float2* Yf;     // [nO][cs]
    float2* Yw;     // [nO][nbw][cs]
    float* yring;   // [nO][rmask + 1]
};

struct MBank {
    const float2* W;
    int wlog, N0, nI, nO, M, pad;
    MLevel lv[kMaxMimoLevels];
};

// tiles of Hw for a row of cs = N + 2 bins, and the tile that holds bin k: first bin, bins
__host__ __device__ __forceinline__ int tile_count(int cs) { return cs - 2 < kTile ? 1 : (cs - 2) / kTile; }
__host__ __device__ __forceinline__ int tile_start(int cs, int k) {
    const int t = k / kTile, n = tile_count(cs);
    return (t < n ? t : n - 1) * kTile;
}
__host__ __device__ __forceinline__ int tile_width(int cs, int k0) {
    return k0 == (tile_count(cs) - 1) * kTile ? cs - k0 : kTile;
}

// one task of one stage; kind: 0 input FFT, 1 fire sum, 2 spread, 3 output IFFT
struct MTask {
    int kind, level, ch, k0;
    int k1, i0, i1, part;
};

__device__ __forceinline__ long long imod(long long a, long long m) {
    long long r = a % m;
    return r < 0 ? r + m : r;
}
__device__ __forceinline__ f32x2 neg2(f32x2 v) { return v ^ 0x8000000080000000ULL; }
__device__ __forceinline__ float4 f4mac(float4 acc, float4 x, float4 h) {
    // the products rounded before they are added: one rounding of the long sum each
    const float2 lo = cmul(make_float2(x.x, x.y), make_float2(h.x, h.y));
    const float2 hi = cmul(make_float2(x.z, x.w), make_float2(h.z, h.w));
    return make_float4(acc.x + lo.x, acc.y + lo.y, acc.z + hi.x, acc.w + hi.y);
}
__device__ __forceinline__ float4 f4add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// L2 eviction policy for a MAC task's filter rows: the level-0 rows (read
// every base step) are evicted last, the larger levels' rows, which stream
// through once per level block, first
__device__ __forceinline__ unsigned long long l2_policy(bool keep) {
    unsigned long long p;
    if (keep)
        asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    else
        asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// 16-byte read-only load with an L2 cache policy, not kept in L1
__device__ __forceinline__ float4 ld_policy(const float4* ptr, unsigned long long pol) {
    float4 v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(ptr), "l"(pol));
    return v;
}

__device__ __forceinline__ long long block_of(const MLevel& l, long long c) {   // newest block fired by step c
    return (c + 1 + l.s_blocks) / l.T - 1;
}

// ---------------------------------------------------------------------------
// K1: input FFTs
// ---------------------------------------------------------------------------
template <int NT, int MAXB>
__global__ void __launch_bounds__(NT) mimo_xfft_kernel(const MBank* __restrict__ bank_p, const MTask* __restrict__ tasks,
                                                       RunState rs, float* __restrict__ xring, int rin_mask) {
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const MBank& bank = *bank_p;
    const MTask t = tasks[blockIdx.x];
    const MLevel& l = bank.lv[t.level];
    const int N = l.N, logN = l.logN, tid = threadIdx.x, N0 = bank.N0;
    float2* s = reinterpret_cast<float2*>(dyn_smem);
    float2* twt = s + N;
    const long long c = rs.step_base;
    const long long t_new = c * (long long)N0, t_end = t_new + N0;
    const float* in = rs.io.in + (c - rs.io.step0) * rs.io.in_step + (long long)t.ch * rs.io.in_ch;
    float* xr = xring + (size_t)t.ch * (rin_mask + 1);
    load_twiddles<NT>(twt, logN, bank.W, bank.wlog);
    const long long isamp = rs.io.in_sample;
    const long long b = block_of(l, c);
    float2* Xs = l.X + ((size_t)t.ch * l.slots + (size_t)imod(b, l.slots)) * l.cs;
    // A window that lies wholly in this call's input is transformed before
    // the dependency wait (it reads only the input), its spectrum held in
    // registers until after the wait, when the spectrum ring may be written.
    constexpr int KMAX = 2 * MAXB + 1;   // bin pairs per thread (N <= 4 NT MAXB)
    const bool early = MAXB <= 2 && (c - rs.io.step0) * N0 >= 2LL * N - N0;
    float2 xk_r[MAXB <= 2 ? KMAX : 1][2];
    if constexpr (MAXB <= 2) {
        if (early) {
            for (int n = tid; n < N; n += NT) {
                const long long j = t_end - 2LL * N + 2LL * n - t_new;   // may be negative: earlier blocks
                s[n] = make_float2(in[j * isamp], in[(j + 1) * isamp]);
            }
            __syncthreads();
            const Twiddles tw{twt, logN};
            fft_smem<NT, MAXB>(s, N, logN, tw, false);
#pragma unroll
            for (int q = 0; q < KMAX; ++q) {
                const int k = tid + q * NT;
                if (k <= N / 2) rfft_split(s[k], s[k == 0 ? 0 : N - k], k, logN, tw, xk_r[q][0], xk_r[q][1]);
            }
        }
    }
    cudaGridDependencySynchronize();
    if constexpr (MAXB <= 2) {
        if (early) {
#pragma unroll
            for (int q = 0; q < KMAX; ++q) {
                const int k = tid + q * NT;
                if (k <= N / 2) {
                    Xs[k] = xk_r[q][0];
                    if (N - k != k) Xs[N - k] = xk_r[q][1];
                }
            }
            if (t.level == 0)   // the ring keeps the input history for later calls
                for (int i = tid; i < N0; i += NT) xr[(t_new + i) & rin_mask] = in[i * isamp];
            return;
        }
    }
    for (int n = tid; n < N; n += NT) {
        const long long ta = t_end - 2LL * N + 2LL * n;
        float a, bb;
        if (ta >= t_new) {
            const long long j = ta - t_new;
            a = in[j * isamp];
            bb = in[(j + 1) * isamp];
            if (t.level == 0) {
                xr[ta & rin_mask] = a;
                xr[(ta + 1) & rin_mask] = bb;
            }
        } else {
            a = __ldcg(&xr[ta & rin_mask]);
            bb = __ldcg(&xr[(ta + 1) & rin_mask]);
        }
        s[n] = make_float2(a, bb);
    }
    __syncthreads();
    const Twiddles tw{twt, logN};
    fft_smem<NT, MAXB>(s, N, logN, tw, false);
    for (int k = tid; k <= N / 2; k += NT) {
        const int nk = (k == 0) ? 0 : N - k;
        float2 xk, xnk;
        rfft_split(s[k], s[nk], k, logN, tw, xk, xnk);
        Xs[k] = xk;
        if (N - k != k) Xs[N - k] = xnk;
    }
}

// ---------------------------------------------------------------------------
// K2: MAC tasks (fire sums and spread partial sums)
//
// Measured on the 64 x 64 workload (us per launch): this kernel 30.7; with
// at most four term groups of 32 columns (a third of the threads idle on
// 44-bin tiles) 31.0; with the row-major H before the tile-major one 32.5.
// Rejected:
//   * H streamed into shared memory by cp.async stages (4 x 8 KB per CTA, no
//     registers held by the copies): 67 -- the input-spectrum loads became a
//     chain of round trips per stage, behind two barriers each;
//   * a task's whole H tile copied into shared memory by cp.async before the
//     grid dependency wait, input spectra through registers one batch ahead:
//     46.6-48.6 -- 46 KB per CTA leaves four CTAs per SM, and each CTA's
//     input-spectrum round trips start only once its tile has landed;
//   * four outputs per task, one input-spectrum load feeding four filter
//     loads (twice the filter bytes in flight per thread, a quarter of the
//     CTAs): 32.4;
//   * terms in part-major order (consecutive inputs of one part; input
//     spectra then far apart): 35.1;
//   * the filter loads as ld.global.nc.L1::no_allocate with a 128- or
//     256-byte L2 prefetch size instead of __ldcs: 30.49 against 30.51;
//   * 256-thread CTAs (four per SM): 31.4; 64-thread CTAs: 47.8.
//   * the larger levels' tasks first in the launch (level 0's last): 30.6;
//   * input spectra through L1 (__ldg): 28.2 against 28.5, not worth relying
//     on the read-only path for data the previous kernel wrote;
//   * (probes) level-0 tasks alone 16.2, level-1 tasks alone 21.4, and 21.7
//     with the level-1 filter loads at the addresses of an interleaved
//     [term][task][column] layout: DRAM page locality is not what limits it.
// Kept: the level-0 filter rows (68 MB, read every base step) loaded with an
// L2 evict-last policy and the larger levels' rows with evict-first, so more
// of the level-0 rows survive in L2 between steps: 30.5 -> 28.5 (evict-normal
// for level 0: 28.8).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kMacNT, 8) mimo_mac_kernel(const MBank* __restrict__ bank_p,
                                                          const MTask* __restrict__ tasks, RunState rs) {
    __shared__ float4 red[kMacNT];
    cudaTriggerProgrammaticLaunchCompletion();
    const MBank& bank = *bank_p;
    const MTask t = tasks[blockIdx.x];
    const MLevel& l = bank.lv[t.level];
    // ncol bin-pair columns (a float4 each) x G term groups; consecutive
    // threads walk a row of the tile, then the next term's row, which
    // follows it in memory
    const int ncol = (t.k1 - t.k0) >> 1;
    const int G = kMacNT / ncol;
    const int lane = threadIdx.x % ncol, g = threadIdx.x / ncol;
    const int k = t.k0 + 2 * lane;
    const bool active = g < G;
    const int o = t.ch, P = l.P, cs = l.cs, nI = bank.nI;
    const long long c = rs.step_base;

    // (input, part) iteration space
    long long bt;
    int p_lo, np, i0, ni;
    if (t.kind == 1) {   // fire sum: parts 0 (and 1 for level 0) of the block due now
        bt = block_of(l, c);
        p_lo = 0;
        np = (l.T == 1 && P >= 2) ? 2 : 1;
        i0 = 0;
        ni = nI;
    } else {             // spread: parts p >= p_lo of a later block
        bt = (l.T == 1) ? c + 1 : (c + 1 + l.s_blocks) / l.T;
        p_lo = (l.T == 1) ? 2 : 1;
        np = P - p_lo;
        i0 = t.i0;
        ni = t.i1 - t.i0;
    }
    const int J = ni * np;
    // row offsets (in float4 units) of every (input, part) term, computed
    // once per CTA so the streaming loop carries no index arithmetic
    __shared__ int xoff[kMaxMacTerms], hoff[kMaxMacTerms];
    const int R = l.slots, slot_bt = (int)imod(bt, R);
    for (int j = threadIdx.x; j < J; j += kMacNT) {
        const int i = i0 + j / np;
        const int p = p_lo + j % np;
        int sl = slot_bt - p;
        if (sl < 0) sl += R;
        xoff[j] = ((i * R + sl) * cs) >> 1;
        hoff[j] = ((i * P + p) * (t.k1 - t.k0)) >> 1;
    }
    __syncthreads();
    // the tables depend only on the task and the step: built before the
    // wait for the input spectra of this step
    cudaGridDependencySynchronize();
    // this task's tile of H: [input][part][width] at o nI P cs + k0 nI P
    const float4* H4 = reinterpret_cast<const float4*>(l.H + (size_t)o * nI * P * cs + (size_t)t.k0 * nI * P + (k - t.k0));
    const float4* X4 = reinterpret_cast<const float4*>(l.X + k);
    const unsigned long long hpol = l2_policy(t.level == 0);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
        // eight 128-thread CTAs per SM (64 registers): more, smaller CTAs in
        // flight hide HBM latency better than deeper per-thread unrolling
        constexpr int U = 4;
        for (int j0 = g; j0 < J; j0 += U * G) {
            float4 xv[U], hv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u * G;
                if (j < J) {
                    xv[u] = __ldcg(X4 + xoff[j]);
                    hv[u] = ld_policy(H4 + hoff[j], hpol);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j0 + u * G < J) acc = f4mac(acc, xv[u], hv[u]);
        }
    }
    if (g > 0 && active) red[(g - 1) * ncol + lane] = acc;
    __syncthreads();
    if (g != 0) return;
    for (int j = 1; j < G; ++j) acc = f4add(acc, red[(j - 1) * ncol + lane]);
    if (t.kind == 1) {
        const bool has_spread = (l.T == 1) ? P >= 3 : P >= 2;
        if (has_spread) {
            const int buf = (l.T == 1) ? (int)(bt & 1) : 0;
            for (int q = 0; q < l.npart; ++q)
                acc = f4add(acc, __ldcg(reinterpret_cast<const float4*>(
                                     l.Yp + (((size_t)o * l.npart + q) * 2 + buf) * cs + k)));
        }
        *reinterpret_cast<float4*>(l.Yf + (size_t)o * cs + k) = acc;
    } else {
        const int buf = (l.T == 1) ? (int)(bt & 1) : 0;
        *reinterpret_cast<float4*>(l.Yp + (((size_t)o * l.npart + t.part) * 2 + buf) * cs + k) = acc;
    }
}

// ---------------------------------------------------------------------------
// Block-parallel sum over inputs and parts, Y_o[b] = sum_i sum_p X_i[b-p]
// H_{i,o,p} per bin.  Lane = bin; a warp keeps kOB outputs x kBB consecutive
// blocks in registers (packed pairs), so an H value loaded once serves kBB
// blocks and an X value kOB outputs, and the window of kBB spectra moves by
// one row per part.  The CTA's four warps take four groups of blocks (the same
// H, from L1), or with fewer blocks split the inputs; a tile of 2 bins splits
// the inputs over the lanes instead.  An input's parts are summed last to first
// (a response decays, so the small terms come first) and folded into a second
// sum in shared memory: a plain chain over 64 inputs x 16 parts would round
// four times as much as the one-block kernel's short ones.
// Bound: float32 multiply-adds (8.3 us per billion cmacs at the packed rate)
// where H is reused over many blocks, else HBM reading H.
// ---------------------------------------------------------------------------
constexpr int kOP = kOB / 2;            // pairs of outputs a warp sums together
constexpr int kStages = 4;              // pipeline stages of two parts (or an input's window)
constexpr int kStageBytes = 2 * (16 * kOP + 8) * 32;   // per warp: H and X of two parts
static_assert(8 * 32 * kBB <= kStageBytes, "a window is one stage");
struct WideMacSmem {
    char ring[4][kStages][kStageBytes];
    f32x2 so[4][kOB * kBB][32];
};
// global -> shared copies, each lane its own column; X zero-filled when !on
__device__ __forceinline__ void cp_async8(unsigned dst, const void* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(on ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

__global__ void __launch_bounds__(128, 3) mimo_wide_mac_kernel(const MBank* __restrict__ bank_p,
                                                               const int4* __restrict__ map, long long c0, int nsteps) {
    extern __shared__ float4 dyn_smem[];
    WideMacSmem& sm = *reinterpret_cast<WideMacSmem*>(dyn_smem);
    cudaTriggerProgrammaticLaunchCompletion();
    const MBank& bank = *bank_p;
    const int4 e = map[blockIdx.x];   // level, first bin, first output, first block of the chunk
    const MLevel& l = bank.lv[e.x];
    const int nI = bank.nI, nO = bank.nO, P = l.P, cs = l.cs, R = l.slots;
    const long long bf = (c0 + l.s_blocks) / l.T;
    const int nb = (int)((c0 + nsteps + l.s_blocks) / l.T - bf) - e.w;   // blocks from the CTA's first on
    cudaGridDependencySynchronize();
    if (nb <= 0) return;
    const int t0 = tile_start(cs, e.y), tw = tile_width(cs, t0);   // the tile in memory
    const int w = min(min(kTile, t0 + tw - e.y), cs - 2 > kTile && e.y < cs - 2 ? cs - 2 - e.y : kTile);
    const int wl = w > 2 ? 32 : 2, nsub = 32 / wl;   // lanes per set of bins, input split over lanes
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int bin = lane & (wl - 1), sub = lane / wl;
    const int nbg = min(kSegBlocks / kBB, nb > 2 * kBB ? 4 : (nb > kBB ? 2 : 1)), ks = 4 / nbg;
    const int g = warp % nbg, kq = warp / nbg;
    const bool live = bin < w;
    const int col = min(bin, w - 1);
    f32x2 re[kOP][kBB], im[kOP][kBB];   // (output 2 q, output 2 q + 1) of pair q
#pragma unroll
    for (int q = 0; q < kOP; ++q)
#pragma unroll
        for (int j = 0; j < kBB; ++j) {
            re[q][j] = im[q][j] = 0;
            sm.so[warp][(2 * q) * kBB + j][lane] = 0;
            sm.so[warp][(2 * q + 1) * kBB + j][lane] = 0;
        }
    // filter rows of the tile, [input][part][tw]; the pairs after the first one
    // pair_stride further (the last pair again beyond the outputs)
    const size_t pair_elems = (size_t)nI * P * cs;
    const int op0 = e.z >> 1, npair = (nO + 1) >> 1;
    const float4* H0 = l.Hw + op0 * pair_elems + (size_t)t0 * nI * P + (e.y - t0) + col;
    size_t pair_off[kOP];
#pragma unroll
    for (int q = 0; q < kOP; ++q) pair_off[q] = (size_t)(min(op0 + q, npair - 1) - op0) * pair_elems * sizeof(float4);
    int sl0 = (int)(bf % R) + e.w + g * kBB;   // ring row of the group's first block
    sl0 %= R;
    const int step = ks * nsub, wrap = R * cs;
    const int nit = g * kBB < nb ? (nI - kq * nsub + step - 1) / step : 0;
    // The copies run kStages - 1 stages ahead of the sums, through every input:
    // a stage is an input's window under its last part or two parts' filter
    // values with the two spectra that enter the window after them.
    const unsigned ring0 = (unsigned)__cvta_generic_to_shared(sm.ring[warp][0]);
    int p_it = 0, p_part = -1, p_ox = 0;   // the producer: input, part (-1: the window)
    unsigned p_slot = ring0;
    bool p_on = false;
    const float2* p_X = l.X;
    const char* p_H = reinterpret_cast<const char*>(H0);
    auto next_slot = [&](unsigned sl) { return sl == ring0 + (kStages - 1) * kStageBytes ? ring0 : sl + kStageBytes; };
    auto produce = [&]() {
        if (p_it < nit) {
            if (p_part < 0) {
                const int i0 = kq * nsub + p_it * step + sub, i = min(i0, nI - 1);
                p_on = live && i0 < nI;
                p_X = l.X + (size_t)i * R * cs + e.y + col;
                p_H = reinterpret_cast<const char*>(H0 + ((size_t)i * P + P - 1) * tw);
                p_ox = sl0 - (P - 1);   // the window under the last part
                p_ox = (p_ox < 0 ? p_ox + R : p_ox) * cs;
                int o = p_ox;
#pragma unroll
                for (int j = 0; j < kBB; ++j) {
                    cp_async8(p_slot + (j * 32 + lane) * 8, p_X + o, p_on);
                    o += cs;
                    if (o >= wrap) o -= wrap;
                }
                p_ox = o;               // the block that enters next
                p_part = 0;
            } else {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (p_part + u < P) {
#pragma unroll
                        for (int q = 0; q < kOP; ++q)
                            cp_async16(p_slot + ((u * kOP + q) * 32 + lane) * 16, p_H + pair_off[q]);
                        p_H -= tw * sizeof(float4);
                        cp_async8(p_slot + 2 * kOP * 512 + (u * 32 + lane) * 8, p_X + p_ox, p_on);
                        p_ox += cs;
                        if (p_ox >= wrap) p_ox -= wrap;
                    }
                }
                p_part += 2;
                if (p_part >= P) {
                    p_part = -1;
                    ++p_it;
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        p_slot = next_slot(p_slot);
    };
    auto landed = [&]() { asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory"); };
#pragma unroll
    for (int q = 0; q < kStages - 1; ++q) produce();
    int c_slot = 0;
    for (int it = 0; it < nit; ++it) {
        // (re, re) and (im, im) of the window: block (first) + j under the r-th part at [(j + r) mod kBB]
        f32x2 xr[kBB], xi[kBB];
        auto put = [&](int q, f32x2 v) {
            const float2 t = unpack2(v);
            xr[q] = pack2(t.x, t.x);
            xi[q] = pack2(t.y, t.y);
        };
        landed();
        {
            const f32x2* d = reinterpret_cast<const f32x2*>(sm.ring[warp][c_slot]);
#pragma unroll
            for (int j = 0; j < kBB; ++j) put(j, d[j * 32 + lane]);
        }
        c_slot = (c_slot + 1) & (kStages - 1);
        produce();
        for (int p0 = 0; p0 < P; p0 += kBB) {
#pragma unroll
            for (int s = 0; s < kBB / 2; ++s) {
                if (p0 + 2 * s >= P) break;
                landed();
                const char* d = sm.ring[warp][c_slot];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int r = 2 * s + u;   // r-th part from the last, mod kBB
                    if (p0 + r >= P) break;
#pragma unroll
                    for (int q = 0; q < kOP; ++q) {
                        const ulonglong2 h = reinterpret_cast<const ulonglong2*>(d)[(u * kOP + q) * 32 + lane];
                        const f32x2 hr = h.x, hi = h.y, hn = neg2(h.y);
                        // (sixteen independent sums between the two products of one)
#pragma unroll
                        for (int j = 0; j < kBB; ++j) {
                            const int m = (j + r) % kBB;
                            re[q][j] = fma2(xr[m], hr, re[q][j]);
                            im[q][j] = fma2(xr[m], hi, im[q][j]);
                        }
#pragma unroll
                        for (int j = 0; j < kBB; ++j) {
                            const int m = (j + r) % kBB;
                            re[q][j] = fma2(xi[m], hn, re[q][j]);
                            im[q][j] = fma2(xi[m], hr, im[q][j]);
                        }
                    }
                    put(r % kBB,
                        reinterpret_cast<const f32x2*>(d + 2 * kOP * 512)[u * 32 + lane]);   // (unused after the last part)
                }
                c_slot = (c_slot + 1) & (kStages - 1);
                produce();
            }
        }
#pragma unroll
        for (int q = 0; q < kOP; ++q)
#pragma unroll
            for (int j = 0; j < kBB; ++j) {
                f32x2& dr = sm.so[warp][(2 * q) * kBB + j][lane];
                f32x2& di = sm.so[warp][(2 * q + 1) * kBB + j][lane];
                dr = add2(dr, re[q][j]);
                di = add2(di, im[q][j]);
                re[q][j] = im[q][j] = 0;
            }
    }
    __syncthreads();
    // the input ranges in order: lanes, then warps
    const int items = nbg * kOP * kBB * wl;
    for (int x = threadIdx.x; x < items; x += 128) {
        const int bi = x & (wl - 1), r = x / wl, j = r % kBB, q = r / kBB % kOP, gg = r / (kBB * kOP);
        const int o = e.z + 2 * q, b = gg * kBB + j;
        if (bi >= w || o >= nO || b >= nb) continue;
        f32x2 vr = sm.so[gg][(2 * q) * kBB + j][bi], vi = sm.so[gg][(2 * q + 1) * kBB + j][bi];
        for (int p = 1; p < ks * nsub; ++p) {
            const int ww = (p / nsub) * nbg + gg, ll = (p % nsub) * wl + bi;
            vr = add2(vr, sm.so[ww][(2 * q) * kBB + j][ll]);
            vi = add2(vi, sm.so[ww][(2 * q + 1) * kBB + j][ll]);
        }
        const float2 yr = unpack2(vr), yi = unpack2(vi);
        float2* Y = l.Yw + ((size_t)o * l.nbw + e.w + b) * cs + e.y + bi;
        Y[0] = make_float2(yr.x, yi.x);
        if (o + 1 < nO) Y[(size_t)l.nbw * cs] = make_float2(yr.y, yi.y);
    }
}

// ---------------------------------------------------------------------------
// K3: output IFFTs and the step's output
// ---------------------------------------------------------------------------
template <int NT, int MAXB>
__global__ void __launch_bounds__(NT) mimo_yifft_kernel(const MBank* __restrict__ bank_p,
                                                        const MTask* __restrict__ tasks, RunState rs) {
    extern __shared__ float4 dyn_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    const MBank& bank = *bank_p;
    const MTask t = tasks[blockIdx.x];
    const MLevel& l = bank.lv[t.level];
    const int N = l.N, logN = l.logN, tid = threadIdx.x, N0 = bank.N0, o = t.ch;
    float2* s = reinterpret_cast<float2*>(dyn_smem);
    float2* twt = s + N;
    load_twiddles<NT>(twt, logN, bank.W, bank.wlog);
    cudaGridDependencySynchronize();
    __syncthreads();
    const Twiddles tw{twt, logN};
    const float2* Y = l.Yf + (size_t)o * l.cs;
    for (int k = tid; k <= N / 2; k += NT) {
        float2 zk, znk;
        irfft_merge(__ldcg(&Y[k]), __ldcg(&Y[N - k]), k, logN, tw, zk, znk);
        s[k] = zk;
        if (k != 0 && k != N / 2) s[N - k] = znk;
    }
    __syncthreads();
    fft_smem<NT, MAXB>(s, N, logN, tw, true);
    const float* sf = reinterpret_cast<const float*>(s);
    const long long c = rs.step_base;
    if (t.level > 0) {
        const long long t0 = block_of(l, c) * (long long)N;
        float* yr = l.yring + (size_t)o * (l.rmask + 1);
        for (int i = tid; i < N; i += NT) yr[(t0 + i) & l.rmask] = sf[i];
        return;
    }
    const long long t_new = c * (long long)N0;
    float* out = rs.io.out + (c - rs.io.step0) * rs.io.out_step + (long long)o * rs.io.out_ch;
    for (int i = tid; i < N0; i += NT) {
        float v = sf[i];
        for (int L = 1; L < bank.M; ++L) {
            const MLevel& l2 = bank.lv[L];
            v += __ldcg(&l2.yring[(size_t)o * (l2.rmask + 1) + ((t_new + i) & l2.rmask)]);
        }
        out[i * rs.io.out_sample] = v;
    }
}

// where bin k of row ip (input, part) of rows lies in an output's tiles of H
__device__ __forceinline__ size_t tile_elem(const int* __restrict__ tstart, int ntile, int k, int rows, int ip) {
    int lo = 0, hi = ntile;   // tile t with tstart[t] <= k < tstart[t + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tstart[mid] <= k) lo = mid;
        else hi = mid;
    }
    const int k0 = tstart[lo], w = tstart[lo + 1] - k0;
    return (size_t)k0 * rows + (size_t)ip * w + (k - k0);
}

// Hw from H, one row (output pair, input, part) per CTA; an odd last output is
// paired with zeros
__global__ void __launch_bounds__(256) mimo_pair_kernel(const MBank* __restrict__ bank_p, int level) {
    const MBank& bank = *bank_p;
    const MLevel& l = bank.lv[level];
    const int rows = bank.nI * l.P, cs = l.cs, op = blockIdx.x / rows, ip = blockIdx.x - op * rows;
    const bool two = 2 * op + 1 < bank.nO;
    const float2* h = l.H + (size_t)(2 * op) * rows * cs;
    float4* d = l.Hw + (size_t)op * rows * cs;
    for (int k = threadIdx.x; k < cs; k += blockDim.x) {
        const size_t e = tile_elem(l.tstart, l.ntile, k, rows, ip);
        const float2 a = h[e], b = two ? h[(size_t)rows * cs + e] : make_float2(0.f, 0.f);
        const int t0 = tile_start(cs, k);
        d[(size_t)t0 * rows + (size_t)ip * tile_width(cs, t0) + (k - t0)] = make_float4(a.x, b.x, a.y, b.y);
    }
}

// filter spectra of one path row: H[o][i][p] = rfft([0_N, h_{i,o}[start + pN ...]]) / 2N
template <int NT, int MAXB>
__global__ void __launch_bounds__(NT) mimo_spectra_kernel(const float* __restrict__ irs, int ir_len, int nI, int nO,
                                                          int N, int logN, int P, int cs, long long start, float2* H,
                                                          const int* __restrict__ tstart, int ntile,
                                                          const float2* W, int wlog) {
    extern __shared__ float4 dyn_smem[];
    float2* s = reinterpret_cast<float2*>(dyn_smem);
    float2* twt = s + N;
    const int row = blockIdx.x;   // (o * nI + i) * P + p
    const int p = row % P, io = row / P, i = io % nI, o = io / nI;
    const float* h = irs + ((size_t)i * nO + o) * ir_len;
    const long long base = start + (long long)p * N;
    for (int n = threadIdx.x; n < N; n += NT) {
        const int j = 2 * n - N;
        float a = 0.f, b = 0.f;
        if (j >= 0) {
            if (base + j < ir_len) a = h[base + j];
            if (base + j + 1 < ir_len) b = h[base + j + 1];
        }
        s[n] = make_float2(a, b);
    }
    load_twiddles<NT>(twt, logN, W, wlog);
    __syncthreads();
    const Twiddles tw{twt, logN};
    fft_smem<NT, MAXB>(s, N, logN, tw, false);
    const float inv = 1.0f / (float)(2 * N);
    // bin k of path (i, o), part p goes to its tile: H[o][tile][i][p][k - tile start]
    float2* Ho = H + (size_t)o * nI * P * cs;
    const int ip = i * P + p;
    auto put = [&](int kb, float2 v) { Ho[tile_elem(tstart, ntile, kb, nI * P, ip)] = v; };
    for (int k = threadIdx.x; k <= N / 2; k += NT) {
        const int nk = (k == 0) ? 0 : N - k;
        float2 xk, xnk;
        rfft_split(s[k], s[nk], k, logN, tw, xk, xnk);
        put(k, make_float2(xk.x * inv, xk.y * inv));
        if (N - k != k) put(N - k, make_float2(xnk.x * inv, xnk.y * inv));
    }
}

int cls_of(int N) { return N <= 1024 ? 0 : (N <= 4096 ? 1 : 2); }

cudaLaunchConfig_t pdl_cfg(int grid, int nt, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr, bool pdl) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cfg;
}

}  // namespace

struct pcm_handle {
    int verbosity = 0;
    std::string err;
    bool ready = false;
    int device = -1;
    cudaStream_t stream = nullptr;
    cudaEvent_t used = nullptr;   // after the last call on a caller's stream
    int fs = 0, N0 = 0, nI = 0, nO = 0, M = 0, H = 1, maxN = 0, fft_cls = 0;
    std::vector<int> N, P;
    std::vector<void*> allocs;
    MBank hbank{};
    MBank* d_bank = nullptr;
    float* xring = nullptr;
    int rin_mask = 0;
    // per stage and phase: tasks at d_tasks + off, count cnt
    MTask* d_tasks = nullptr;
    std::vector<int> off[3], cnt[3];
    std::vector<double> mac_bytes;   // algorithmic bytes of K2 per phase
    std::vector<std::vector<int>> tiles;   // per level: bin tile starts (last entry cs)
    // block-parallel calls (wide.cu): descriptors of every (level, input) and
    // (output, level), CTA maps in order of their first block's step and the
    // prefix of each that a chunk of n + 1 steps needs
    int C_max = 32;   // most base steps per chunk
    int w_min = kWideMinSteps;   // base steps from which a call runs block-parallel
    int C = 0;        // ... that the workspace in hand holds (0: none yet)
    char* work = nullptr;    // rings and sums of chunks of C steps (before: the rings among `allocs`)
    float4* hw = nullptr;    // the levels' Hw
    size_t work_bytes = 0, hw_bytes = 0;
    bool work_failed = false;   // no room for the size last asked for: not tried again until reset
    bool work_kept = false;     // a graph uses it: no larger one replaces it
    std::vector<WLevel> h_wlv;
    WLevel* d_wlv_of[2] = {};   // d_wlv and the other buffer of it
    const float2* d_tab = nullptr;
    const WLevel* d_wlv = nullptr;
    const int* d_lv0 = nullptr;   // level-0 descriptor of every input
    int n_wlv = 0, w_nt = 0;
    const int2* w_map[3] = {};    // windows, inverse transforms of levels >= 1, output
    const int4* w_mac = nullptr;
    std::vector<int> w_upto[4];
    // spread tasks that rebuild the partial sums after such a call: per level,
    // first task and tasks of the first j slices
    std::vector<int> state_off;
    std::vector<std::vector<int>> state_cnt;
    size_t reset_bytes = 0;   // most of a descriptor's rings that reset clears
    std::vector<std::pair<void*, size_t>> state;   // zeroed by reset
    long long frame_num = 0;
    long long launches = 0;
    long long device_bytes = 0;
};

namespace {

int mfail(pcm_handle* h, int code, const std::string& m) {
    h->err = m;
    return code;
}

#define MCK(call, where)                                                                                   \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return mfail(h, PC_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
cudaError_t malloc_raw(pcm_handle* h, T** p, size_t n) {
    const size_t bytes = sizeof(T) * std::max<size_t>(n, 1);
    cudaError_t e = cudaMalloc((void**)p, bytes);
    if (e != cudaSuccess) return e;
    h->allocs.push_back(*p);
    h->device_bytes += bytes;
    return e;
}
template <class T>
cudaError_t malloc_zero(pcm_handle* h, T** p, size_t n, bool is_state) {
    cudaError_t e = malloc_raw(h, p, n);
    if (e != cudaSuccess) return e;
    const size_t bytes = sizeof(T) * std::max<size_t>(n, 1);
    if (is_state) h->state.push_back({*p, bytes});
    return cudaMemsetAsync(*p, 0, bytes, h->stream);
}

void mfree(pcm_handle* h) {
    if (h->device >= 0) cudaSetDevice(h->device);
    for (void* p : h->allocs) cudaFree(p);
    h->allocs.clear();
    h->state.clear();
    if (h->work) cudaFree(h->work);
    if (h->hw) cudaFree(h->hw);
    h->work = nullptr;
    h->hw = nullptr;
    h->work_bytes = h->hw_bytes = 0;
    h->work_kept = false;
    h->C = 0;
    if (h->used) cudaEventDestroy(h->used);
    h->used = nullptr;
    if (h->stream) cudaStreamDestroy(h->stream);
    h->stream = nullptr;
    h->ready = false;
}

cudaError_t launch_fft_stage(pcm_handle* h, int stage, int grid, const MTask* tasks, const RunState& rs,
                             cudaStream_t st, bool pdl) {
    cudaLaunchAttribute attr[1];
    const int NT = h->fft_cls == 0 ? 256 : 512;
    const size_t smem = (size_t)12 * h->maxN;
    cudaLaunchConfig_t cfg = pdl_cfg(grid, NT, smem, st, attr, pdl);
    if (stage == 0) {
        switch (h->fft_cls) {
            case 0: return cudaLaunchKernelEx(&cfg, mimo_xfft_kernel<256, 1>, (const MBank*)h->d_bank, tasks, rs, h->xring, h->rin_mask);
            case 1: return cudaLaunchKernelEx(&cfg, mimo_xfft_kernel<512, 2>, (const MBank*)h->d_bank, tasks, rs, h->xring, h->rin_mask);
            default: return cudaLaunchKernelEx(&cfg, mimo_xfft_kernel<512, 8>, (const MBank*)h->d_bank, tasks, rs, h->xring, h->rin_mask);
        }
    }
    switch (h->fft_cls) {
        case 0: return cudaLaunchKernelEx(&cfg, mimo_yifft_kernel<256, 1>, (const MBank*)h->d_bank, tasks, rs);
        case 1: return cudaLaunchKernelEx(&cfg, mimo_yifft_kernel<512, 2>, (const MBank*)h->d_bank, tasks, rs);
        default: return cudaLaunchKernelEx(&cfg, mimo_yifft_kernel<512, 8>, (const MBank*)h->d_bank, tasks, rs);
    }
}

cudaError_t launch_mac(pcm_handle* h, int grid, const MTask* tasks, const RunState& rs, cudaStream_t st, bool pdl) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = pdl_cfg(grid, kMacNT, 0, st, attr, pdl);
    return cudaLaunchKernelEx(&cfg, mimo_mac_kernel, (const MBank*)h->d_bank, tasks, rs);
}

// descriptors and CTA maps of the block-parallel kernels, cleared rings
int setup_wide(pcm_handle* h) {
    const MBank& B = h->hbank;
    const int M = h->M, nI = h->nI, nO = h->nO;
    std::vector<WLevel>& wl = h->h_wlv;
    wl.clear();
    std::vector<int> lv0(nI);
    auto common = [&](int L) {
        const MLevel& l = B.lv[L];
        WLevel w{};
        w.N = l.N;
        w.logN = l.logN;
        w.P = 1;
        for (int t = l.T; t > 1; t >>= 1) ++w.logT;
        w.s_blocks = l.s_blocks;
        w.cs = l.cs;
        w.slots = l.slots;
        w.M = M;
        w.scale = 1.0f;
        return w;
    };
    for (int i = 0; i < nI; ++i) {   // inputs: window transforms
        lv0[i] = (int)wl.size();
        for (int L = 0; L < M; ++L) {
            WLevel w = common(L);
            w.P = B.lv[L].P;
            w.in_ch = i;
            w.rin_mask = h->rin_mask;
            w.X = B.lv[L].X + (size_t)i * w.slots * w.cs;
            w.xring = h->xring + (size_t)i * (h->rin_mask + 1);
            wl.push_back(w);
        }
    }
    const int out0 = (int)wl.size();
    for (int o = 0; o < nO; ++o)     // outputs: inverse transforms
        for (int L = 0; L < M; ++L) {
            WLevel w = common(L);
            const MLevel& l = B.lv[L];
            w.out_ch = o;
            w.mix_mode = 1;
            w.lv0 = out0 + o * M;
            w.rmask = l.rmask;
            w.yring = l.yring + (size_t)o * (l.rmask + 1);
            wl.push_back(w);
        }
    h->n_wlv = (int)wl.size();
    h->w_nt = wide_threads(h->maxN);
    std::vector<std::pair<int, int2>> e[3];
    std::vector<std::pair<int, int4>> mac;
    for (int L = 0; L < M; ++L) {
        const MLevel& l = B.lv[L];
        const int nbw = (h->C_max + l.T - 1) / l.T;   // most blocks of a chunk
        for (int b = 0; b < nbw; b += 16 * h->w_nt / l.N) {
            for (int i = 0; i < nI; ++i) e[0].push_back({b * l.T, make_int2(i * M + L, b)});
            for (int o = 0; o < nO && L > 0; ++o) e[1].push_back({b * l.T, make_int2(out0 + o * M + L, b)});
        }
        for (int b = 0; b < nbw && L == 0; b += wide_out_blocks(l.N))
            for (int o = 0; o < nO; ++o) e[2].push_back({b, make_int2(out0 + o * M, b)});
        for (int b = 0; b < nbw; b += kSegBlocks)
            for (int k = 0; k < l.cs; k += kTile)   // (the last two bins by themselves)
                for (int o = 0; o < nO; o += kOB) mac.push_back({b * l.T, make_int4(L, k, o, b)});
    }
    // one allocation and one upload for all the tables
    std::vector<char> blob;
    auto put = [&](const void* src, size_t bytes) {
        const size_t at = blob.size();
        blob.resize(at + ((bytes + 255) & ~(size_t)255));
        if (bytes) std::memcpy(blob.data() + at, src, bytes);
        return at;
    };
    auto put_map = [&](auto& v, std::vector<int>& upto) {
        using E = std::remove_reference_t<decltype(v[0].second)>;
        std::stable_sort(v.begin(), v.end(), [](auto& a, auto& b) { return a.first < b.first; });
        std::vector<E> flat;
        for (auto& x : v) flat.push_back(x.second);
        upto.assign(h->C_max, 0);
        size_t j = 0;
        for (int n = 0; n < h->C_max; ++n) {
            while (j < v.size() && v[j].first <= n) ++j;
            upto[n] = (int)j;
        }
        return put(flat.data(), sizeof(E) * flat.size());
    };
    size_t at[7];
    for (int m = 0; m < 3; ++m) at[m] = put_map(e[m], h->w_upto[m]);
    at[3] = put_map(mac, h->w_upto[3]);
    at[4] = put(wl.data(), sizeof(WLevel) * wl.size());
    at[5] = put(lv0.data(), sizeof(int) * lv0.size());
    at[6] = put(wl.data(), sizeof(WLevel) * wl.size());
    char* d = nullptr;
    MCK(cudaMalloc(&d, blob.size()), "alloc tables");
    h->allocs.push_back(d);
    h->device_bytes += blob.size();
    MCK(cudaMemcpyAsync(d, blob.data(), blob.size(), cudaMemcpyHostToDevice, h->stream), "upload tables");
    MCK(cudaStreamSynchronize(h->stream), "sync");
    for (int m = 0; m < 3; ++m) h->w_map[m] = reinterpret_cast<const int2*>(d + at[m]);
    h->w_mac = reinterpret_cast<const int4*>(d + at[3]);
    h->d_wlv_of[0] = reinterpret_cast<WLevel*>(d + at[4]);
    h->d_wlv_of[1] = reinterpret_cast<WLevel*>(d + at[6]);
    h->d_wlv = h->d_wlv_of[0];
    h->d_lv0 = reinterpret_cast<const int*>(d + at[5]);
    h->reset_bytes = 0;
    for (auto& w : wl) h->reset_bytes = std::max(h->reset_bytes, wide_reset_bytes(w, h->N0));
    MCK(launch_wide_reset(h->d_wlv, h->n_wlv, h->reset_bytes, nullptr, 0, h->stream), "clear rings");
    return PC_OK;
}

// rings of a level for chunks of C steps (0: one-block steps)
int ring_rows(const MLevel& l, int C) { return l.P + (C > 0 ? std::max((C + l.T - 1) / l.T, kBB) : 0); }
long ring_samples(const MLevel& l, int N0, int C) {
    long R = l.N;
    while (R < ((long)l.s_blocks + std::max(C, 1)) * N0) R <<= 1;   // samples in flight
    return R;
}

// A workspace for chunks of up to C steps in place of the present one, its rings
// holding what the present ones do, and Hw if there is none yet.  PC_ERR_NOMEM if
// there is no room: everything stays as it is.
int move_to_work(pcm_handle* h, int C, cudaStream_t st) {
    const MBank old = h->hbank;
    MBank& B = h->hbank;   // (what is uploaded outlives the call; old again on failure)
    const int nI = h->nI, nO = h->nO;
    size_t bytes = 0, hw_elems = 0;
    auto take = [&](size_t n) {
        const size_t o = bytes;
        bytes += (n + 255) & ~(size_t)255;
        return o;
    };
    std::vector<size_t> oX(h->M), oY(h->M), oR(h->M), oH(h->M);
    for (int L = 0; L < h->M; ++L) {
        MLevel& l = B.lv[L];
        l.nbw = (C + l.T - 1) / l.T;
        l.slots = ring_rows(l, C);
        const long R = ring_samples(l, h->N0, C);
        l.rmask = (int)R - 1;
        if ((long long)nI * l.slots * l.cs >= (1LL << 31)) {   // 32-bit offsets
            h->hbank = old;
            return PC_ERR_NOMEM;
        }
        oX[L] = take(sizeof(float2) * (size_t)nI * l.slots * l.cs);
        oY[L] = take(sizeof(float2) * (size_t)nO * l.nbw * l.cs);
        oR[L] = take(sizeof(float) * (size_t)nO * R);
        oH[L] = hw_elems;
        hw_elems += (size_t)((nO + 1) / 2) * nI * l.P * l.cs;
    }
    // (another thread may be capturing a graph meanwhile)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    char* W = nullptr;
    float4* hw = h->hw;
    cudaError_t e = cudaMalloc(&W, bytes);
    if (e == cudaSuccess && !hw) e = cudaMalloc(&hw, sizeof(float4) * hw_elems);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (W) cudaFree(W);
        cudaThreadExchangeStreamCaptureMode(&mode);
        h->hbank = old;
        return PC_ERR_NOMEM;
    }
    for (int L = 0; L < h->M; ++L) {
        MLevel& l = B.lv[L];
        l.X = reinterpret_cast<float2*>(W + oX[L]);
        l.Yw = reinterpret_cast<float2*>(W + oY[L]);
        l.yring = reinterpret_cast<float*>(W + oR[L]);
        l.Hw = hw + oH[L];
    }
    std::vector<WLevel> wl = h->h_wlv;
    for (int j = 0; j < h->n_wlv; ++j) {   // the inputs' levels, then the outputs'
        const int L = j % h->M, ch = j / h->M;
        const MLevel& l = B.lv[L];
        WLevel& w = wl[j];
        w.slots = l.slots;
        if (ch < nI) {
            w.X = l.X + (size_t)ch * l.slots * l.cs;
        } else {
            w.rmask = l.rmask;
            w.Yw = l.Yw + (size_t)(ch - nI) * l.nbw * l.cs;
            w.yring = l.yring + (size_t)(ch - nI) * (l.rmask + 1);
        }
    }
    WLevel* next = h->d_wlv == h->d_wlv_of[0] ? h->d_wlv_of[1] : h->d_wlv_of[0];
    e = cudaMemcpyAsync(next, wl.data(), sizeof(WLevel) * wl.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->d_bank, &B, sizeof(MBank), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = launch_wide_move(h->d_wlv, next, h->n_wlv, h->frame_num, h->N0, st);
    for (int L = 0; L < h->M && !h->hw && e == cudaSuccess; ++L) {
        mimo_pair_kernel<<<(nO + 1) / 2 * nI * B.lv[L].P, 256, 0, st>>>(h->d_bank, L);
        e = cudaGetLastError();
    }
    if (h->work || e != cudaSuccess) {   // nothing may still read what is freed
        const cudaError_t se = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = se;
        cudaFree(e == cudaSuccess ? h->work : W);
        if (e != cudaSuccess && !h->hw) cudaFree(hw);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) h->hbank = old;
    MCK(e, "block-parallel workspace");
    h->launches += 1 + (h->hw ? 0 : h->M);
    h->work = W;
    h->work_bytes = bytes;
    if (!h->hw) {
        h->hw = hw;
        h->hw_bytes = sizeof(float4) * hw_elems;
    }
    h->C = C;
    h->h_wlv.swap(wl);
    h->d_wlv = next;
    return PC_OK;
}

// Whether a call of nsteps base steps on st can run block-parallel: the workspace
// is made for it, in chunks as short as the call, and grows with longer calls up
// to h->C_max steps; where there is no room, a shorter chunk or one-block steps
// serve.  A stream that is being captured takes the workspace as it is, and that
// one then stays, for the graph's launches hold its addresses.
int ensure_wide(pcm_handle* h, long long nsteps, cudaStream_t st, bool* wide) {
    int want = kWideMinChunk;
    while (want < nsteps && want < h->C_max) want <<= 1;
    *wide = h->C > 0;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    MCK(cudaStreamIsCapturing(st, &cs), "capture status");
    if (cs != cudaStreamCaptureStatusNone) h->work_kept = *wide;
    if (h->C >= want || h->work_failed || h->work_kept || cs != cudaStreamCaptureStatusNone) return PC_OK;
    for (; want > h->C && want >= kWideMinChunk; want >>= 1) {
        const int r = move_to_work(h, want, st);
        if (r == PC_OK) {
            *wide = true;
            return PC_OK;
        }
        if (r != PC_ERR_NOMEM) return r;
        h->work_failed = true;   // (of the size asked for: not tried again until reset)
    }
    return PC_OK;
}

// nsteps base steps from h->frame_num, block-parallel
int mimo_wide(pcm_handle* h, const IOView& io, long long nsteps, cudaStream_t st) {
    WArgs a{};
    a.lv = h->d_wlv;
    a.tab = h->d_tab;
    a.N0 = h->N0;
    a.kb = 1;
    a.full = 1;   // as the one-block kernels here
    a.io = io;
    a.vec_in = io.in_sample == 1 && (h->nI == 1 || io.in_ch % 2 == 0) && (reinterpret_cast<uintptr_t>(io.in) & 7) == 0;
    a.vec_out =
        io.out_sample == 1 && (h->nO == 1 || io.out_ch % 2 == 0) && (reinterpret_cast<uintptr_t>(io.out) & 7) == 0;
    while (nsteps > 0) {
        const int n = (int)std::min<long long>(nsteps, h->C);
        a.c0 = h->frame_num;
        a.nsteps = n;
        MCK(launch_wide_fft(false, h->w_nt, h->w_upto[0][n - 1], h->w_map[0], a, st), "MIMO windows");
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = pdl_cfg(h->w_upto[3][n - 1], 128, sizeof(WideMacSmem), st, attr, true);
        MCK(cudaLaunchKernelEx(&cfg, mimo_wide_mac_kernel, (const MBank*)h->d_bank, h->w_mac, a.c0, n),
            "MIMO sums");
        MCK(launch_wide_fft(true, h->w_nt, h->w_upto[1][n - 1], h->w_map[1], a, st), "MIMO inverse");
        MCK(launch_wide_out(h->N0, h->w_upto[2][n - 1], h->w_map[2], a, st), "MIMO output");
        h->launches += 3 + (h->w_upto[1][n - 1] > 0);
        h->frame_num += n;
        nsteps -= n;
    }
    // the input rings and partial sums one-block steps would have left
    a.c0 = h->frame_num;
    a.nsteps = 0;
    MCK(launch_wide_state(256, 64, 0, nullptr, h->d_lv0, h->nI, h->rin_mask + 1, a, st), "MIMO input rings");
    h->launches += 1;
    RunState rs{};
    rs.step_base = h->frame_num - 1;
    rs.io = io;
    for (int L = 0; L < h->M; ++L) {
        const MLevel& l = h->hbank.lv[L];
        const auto& cnt = h->state_cnt[L];
        if (cnt.size() < 2) continue;
        // slices since the level's last block, and those of them built before the call
        const long long q = h->frame_num + l.s_blocks, q0 = io.step0 + l.s_blocks;
        const int have = l.T > 1 && q / l.T == q0 / l.T ? cnt[q0 % l.T] : 0;
        const int n = cnt[l.T == 1 ? 1 : q % l.T] - have;
        if (n <= 0) continue;
        MCK(launch_mac(h, n, h->d_tasks + h->state_off[L] + have, rs, st, true), "MIMO partial sums");
        h->launches += 1;
    }
    return PC_OK;
}

// one base step; kernel k of the step is timed by ev[k] pairs when given
int mimo_step(pcm_handle* h, const RunState& rs, cudaStream_t st, bool first, cudaEvent_t* ev) {
    const int ph = (int)(rs.step_base & (h->H - 1));
    for (int stage = 0; stage < 3; ++stage) {
        const int n = h->cnt[stage][ph];
        if (n <= 0) continue;
        if (ev) cudaEventRecord(ev[2 * stage], st);
        const MTask* tk = h->d_tasks + h->off[stage][ph];
        cudaError_t e = stage == 1 ? launch_mac(h, n, tk, rs, st, !first && !ev)
                                   : launch_fft_stage(h, stage == 0 ? 0 : 1, n, tk, rs, st, !first && !ev);
        if (ev) cudaEventRecord(ev[2 * stage + 1], st);
        if (e != cudaSuccess) return mfail(h, PC_ERR_CUDA, std::string("MIMO step launch: ") + cudaGetErrorString(e));
        h->launches += 1;
        first = false;
    }
    return PC_OK;
}

}  // namespace

extern "C" {

pcm_handle* pcm_create(int verbosity) {
    pcm_handle* h = new (std::nothrow) pcm_handle();
    if (h) h->verbosity = verbosity;
    return h;
}

int pcm_setup(pcm_handle* h, int fs, int buffer_size, int n_in, int n_out, int M, const int* N, int* P,
              const float* irs, int ir_len) {
    if (!h) return PC_ERR_ARG;
    if (h->ready) return mfail(h, PC_ERR_STATE, "setup called twice without cleanup");
    if (!N || !P || !irs || n_in < 1 || n_out < 1 || ir_len < 1 || M < 1)
        return mfail(h, PC_ERR_ARG, "bad MIMO setup arguments");
    if (M > kMaxMimoLevels) return mfail(h, PC_ERR_LIMIT, "too many levels for the MIMO engine");
    if (N[0] != buffer_size || buffer_size < 16) return mfail(h, PC_ERR_LAYOUT, "first block size must equal buffer_size (>= 16)");
    std::vector<int> Nv(N, N + M), Pv(P, P + M);
    char msg[256];
    int r = pc_check_layout(M, Nv.data(), Pv.data(), ir_len, 1, nullptr, msg, sizeof msg);
    if (r) return mfail(h, r, msg);
    if (Nv[M - 1] > kMaxBlockOneCta)
        return mfail(h, PC_ERR_LIMIT, "MIMO levels are limited to blocks of 16384 (larger blocks: pc_* engine)");
    for (int i = 0; i < M; ++i) P[i] = Pv[i];
    MCK(cudaGetDevice(&h->device), "cudaGetDevice");
    MCK(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "stream");
    MCK(cudaEventCreateWithFlags(&h->used, cudaEventDisableTiming), "event");
    h->fs = fs;
    h->N0 = buffer_size;
    h->nI = n_in;
    h->nO = n_out;
    h->M = M;
    h->N = Nv;
    h->P = Pv;
    h->maxN = Nv.back();
    h->H = std::max(1, Nv.back() / buffer_size);
    h->fft_cls = cls_of(h->maxN);
    if (h->fft_cls == 2) {
        MCK(cudaFuncSetAttribute(mimo_xfft_kernel<512, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 12 * 16384), "attr");
        MCK(cudaFuncSetAttribute(mimo_yifft_kernel<512, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 12 * 16384), "attr");
        MCK(cudaFuncSetAttribute(mimo_spectra_kernel<512, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 12 * 16384), "attr");
    }
    {
        const double row = sizeof(float2) * (double)buffer_size * M * std::max(n_in, n_out);   // per base step
        double spectra = 0.0;
        for (int L = 0; L < M; ++L)
            if (Nv[L] / buffer_size > kWideMinSteps)
                spectra += sizeof(float2) * (double)n_in * n_out * Pv[L] * (Nv[L] + 2);
        h->w_min = kWideMinSteps + (int)(spectra / kWideStepBytes + 0.5);
        h->tiles.clear();
        h->work_failed = false;
        h->C = 0;
        h->C_max = kWideMaxChunk;
        while (h->C_max > kWideMinChunk && h->C_max * row > (double)kWideBytes) h->C_max >>= 1;
    }
    // twiddles
    float2* W = nullptr;
    {
        const std::vector<float2>& Wh = host_twiddles(kWlog);
        MCK(malloc_zero(h, &W, Wh.size(), false), "alloc");
        MCK(cudaMemcpyAsync(W, Wh.data(), sizeof(float2) * Wh.size(), cudaMemcpyHostToDevice, h->stream), "upload");
        MCK(cudaStreamSynchronize(h->stream), "sync");
        float2* tab = nullptr;
        MCK(malloc_raw(h, &tab, kFftTabEntries), "alloc");
        MCK(launch_fft_tables(tab, W, kWlog, h->stream), "transform factors");
        h->d_tab = tab;
        MCK(prepare_wide_kernels(), "kernel attributes");
        MCK(cudaFuncSetAttribute(mimo_wide_mac_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(WideMacSmem)),
            "kernel attributes");
    }
    int rin = 1;
    while (rin < 2 * h->maxN) rin <<= 1;
    h->rin_mask = rin - 1;
    MCK(malloc_zero(h, &h->xring, (size_t)n_in * rin, true), "alloc");
    float* d_irs = nullptr;
    MCK(malloc_zero(h, &d_irs, (size_t)n_in * n_out * ir_len, false), "alloc");
    MCK(cudaMemcpyAsync(d_irs, irs, sizeof(float) * (size_t)n_in * n_out * ir_len, cudaMemcpyHostToDevice, h->stream),
        "upload IRs");
    MBank& B = h->hbank;
    B.wlog = kWlog;
    B.N0 = buffer_size;
    B.nI = n_in;
    B.nO = n_out;
    B.M = M;
    B.W = W;
    long s = 0;
    for (int L = 0; L < M; ++L) {
        MLevel& l = B.lv[L];
        l.N = Nv[L];
        l.logN = (int)std::lround(std::log2((double)Nv[L]));
        l.P = Pv[L];
        l.T = Nv[L] / buffer_size;
        l.s_blocks = (int)(s / buffer_size);
        l.cs = Nv[L] + 2;
        const long R = ring_samples(l, buffer_size, 0);
        l.rmask = (int)R - 1;
        // input ranges per spread task (about 8 inputs each, more ranges when
        // a range times the older parts exceeds what one MAC task sums)
        const int p_lo = l.T == 1 ? 2 : 1;
        l.npart = std::max(1, std::min(n_in, 8));
        while (l.npart < n_in && (long)((n_in + l.npart - 1) / l.npart) * std::max(l.P - p_lo, 0) > kMaxMacTerms)
            l.npart *= 2;
        l.npart = std::min(l.npart, n_in);
        if ((long)((n_in + l.npart - 1) / l.npart) * std::max(l.P - p_lo, 0) > kMaxMacTerms ||
            (long)n_in * 2 > kMaxMacTerms || (long)n_in * l.P * l.cs >= (1L << 31))
            return mfail(h, PC_ERR_LIMIT, "MIMO layout too large for one MAC task (inputs x parts)");
        // the level's fixed bin tiles: the slices its MAC tasks take (level 0:
        // the whole row; larger levels: each phase's slice of bins), cut into
        // tiles of at most kMacMaxBins bins
        {
            std::vector<int> ts;
            // a MAC CTA runs floor(kMacNT / columns) term groups over a tile's
            // columns: pick the tile count that keeps most threads busy (a
            // small charge per extra tile for its CTA's fixed work)
            auto tiles_of = [&](int lo, int hi) {
                const int n = hi - lo;
                int best_nt = 0;
                double best = -1e30;
                const int nt0 = (n + kMacMaxBins - 1) / kMacMaxBins;
                for (int nt = nt0; nt <= std::max(nt0, 16); ++nt) {
                    const int per = ((n + nt - 1) / nt + 1) & ~1;
                    if (per < 2 || (nt - 1) * per >= n) continue;
                    double busy = 0.0;
                    for (int k = lo; k < hi; k += per) {
                        const int nc = (std::min(per, hi - k)) >> 1;
                        busy += (double)((kMacNT / nc) * nc) / kMacNT;
                    }
                    const double score = busy / nt - 0.05 * nt;
                    if (score > best) {
                        best = score;
                        best_nt = nt;
                    }
                }
                const int per = ((n + best_nt - 1) / best_nt + 1) & ~1;
                for (int k = lo; k < hi; k += per) ts.push_back(k);
            };
            if (l.T > 1 && l.P >= 2) {
                const int nch = l.T - 1;
                for (int j = 0; j < nch; ++j) {
                    const int lo = (int)(((long)j * l.cs / nch) & ~1L);
                    const int hi = (j == nch - 1) ? l.cs : (int)(((long)(j + 1) * l.cs / nch) & ~1L);
                    if (hi > lo) tiles_of(lo, hi);
                }
            } else {
                tiles_of(0, l.cs);
            }
            ts.push_back(l.cs);
            l.ntile = (int)ts.size() - 1;
            int* d_ts = nullptr;
            MCK(malloc_zero(h, &d_ts, ts.size(), false), "alloc tiles");
            MCK(cudaMemcpyAsync(d_ts, ts.data(), sizeof(int) * ts.size(), cudaMemcpyHostToDevice, h->stream),
                "upload tiles");
            l.tstart = d_ts;
            h->tiles.push_back(ts);
        }
        MCK(malloc_zero(h, &l.H, (size_t)n_out * n_in * l.P * l.cs, false), "alloc H");
        l.Hw = nullptr;
        l.Yw = nullptr;
        l.nbw = 0;
        l.slots = ring_rows(l, 0);
        // (cleared in part by setup_wide)
        MCK(malloc_raw(h, &l.X, (size_t)n_in * l.slots * l.cs), "alloc");
        MCK(malloc_zero(h, &l.Yp, (size_t)n_out * l.npart * 2 * l.cs, true), "alloc");
        MCK(malloc_zero(h, &l.Yf, (size_t)n_out * l.cs, true), "alloc");
        MCK(malloc_raw(h, &l.yring, (size_t)n_out * R), "alloc");
        const size_t smem = (size_t)12 * l.N;
        const int rows = n_out * n_in * l.P;
        switch (cls_of(l.N)) {
            case 0:
                mimo_spectra_kernel<256, 1><<<rows, 256, smem, h->stream>>>(d_irs, ir_len, n_in, n_out, l.N, l.logN, l.P,
                                                                            l.cs, s, l.H, l.tstart, l.ntile, W, kWlog);
                break;
            case 1:
                mimo_spectra_kernel<512, 2><<<rows, 512, smem, h->stream>>>(d_irs, ir_len, n_in, n_out, l.N, l.logN, l.P,
                                                                            l.cs, s, l.H, l.tstart, l.ntile, W, kWlog);
                break;
            default:
                mimo_spectra_kernel<512, 8><<<rows, 512, smem, h->stream>>>(d_irs, ir_len, n_in, n_out, l.N, l.logN, l.P,
                                                                            l.cs, s, l.H, l.tstart, l.ntile, W, kWlog);
                break;
        }
        MCK(cudaGetLastError(), "MIMO spectra");
        h->launches += 1;
        s += (long)Nv[L] * Pv[L];
    }
    MCK(malloc_zero(h, &h->d_bank, 1, false), "alloc");
    MCK(cudaMemcpyAsync(h->d_bank, &B, sizeof(MBank), cudaMemcpyHostToDevice, h->stream), "upload bank");

    // ---- per-phase task lists --------------------------------------------------------
    // spread tasks of slice j of level L's row (level 0: the whole row); returns its bins
    auto spread_tasks = [&](const MLevel& l, int L, int j, std::vector<MTask>& dst) {
        const int nch = l.T == 1 ? 1 : l.T - 1;
        const int lo = (int)(((long)j * l.cs / nch) & ~1L);
        const int hi = (j == nch - 1) ? l.cs : (int)(((long)(j + 1) * l.cs / nch) & ~1L);
        const std::vector<int>& ts = h->tiles[L];
        for (int o = 0; o < n_out; ++o)
            for (size_t t = 0; t + 1 < ts.size(); ++t) {
                if (ts[t] < lo || ts[t + 1] > hi) continue;
                for (int q = 0; q < l.npart; ++q) {
                    const int i0 = (int)((long)q * n_in / l.npart), i1 = (int)((long)(q + 1) * n_in / l.npart);
                    dst.push_back(MTask{2, L, o, ts[t], ts[t + 1], i0, i1, q});
                }
            }
        return hi - lo;
    };
    std::vector<std::vector<MTask>> lists[3];
    for (auto& v : lists) v.assign(h->H, {});
    h->mac_bytes.assign(h->H, 0.0);
    for (int g = 0; g < h->H; ++g) {
        for (int L = 0; L < M; ++L) {
            const MLevel& l = B.lv[L];
            const double C = l.N + 1.0;
            const bool fires = (g + 1 + l.s_blocks) % l.T == 0;
            if (fires) {
                for (int i = 0; i < n_in; ++i) lists[0][g].push_back(MTask{0, L, i, 0, 0, 0, 0, 0});
                const std::vector<int>& ts = h->tiles[L];   // the level's fixed tiles
                for (int o = 0; o < n_out; ++o)
                    for (size_t t = 0; t + 1 < ts.size(); ++t)
                        lists[1][g].push_back(MTask{1, L, o, ts[t], ts[t + 1], 0, n_in, 0});
                for (int o = 0; o < n_out; ++o) lists[2][g].push_back(MTask{3, L, o, 0, 0, 0, 0, 0});
                const int np = (l.T == 1 && l.P >= 2) ? 2 : 1;
                // H rows of parts 0 (and 1) of every path, X rows once per input
                h->mac_bytes[g] += 8.0 * C * ((double)n_out * n_in * np + (double)n_in * np);
            }
            // spread: level 0 every step over parts >= 2; other levels in the
            // T-1 steps after their block, a slice of bins (whole tiles) per step
            const int p_lo = l.T == 1 ? 2 : 1;
            if (l.P <= p_lo) continue;
            const int phi = (g + 1 + l.s_blocks) % l.T;
            if (l.T > 1 && phi == 0) continue;
            const int bins = spread_tasks(l, L, l.T == 1 ? 0 : phi - 1, lists[1][g]);
            h->mac_bytes[g] += 8.0 * bins * ((double)n_out * n_in * (l.P - p_lo) + (double)n_in * (l.P - p_lo));
        }
    }
    // after a block-parallel call: the spread tasks of the steps since each
    // level's last block, in slice order
    std::vector<MTask> state;
    h->state_off.assign(M, 0);
    h->state_cnt.assign(M, {});
    for (int L = 0; L < M; ++L) {
        const MLevel& l = B.lv[L];
        h->state_off[L] = (int)state.size();
        h->state_cnt[L].push_back(0);
        if (l.P <= (l.T == 1 ? 2 : 1)) continue;
        for (int j = 0; j < std::max(1, l.T - 1); ++j) {
            spread_tasks(l, L, j, state);
            h->state_cnt[L].push_back((int)state.size() - h->state_off[L]);
        }
    }
    size_t ntask = 0;
    for (int st = 0; st < 3; ++st) {
        h->off[st].assign(h->H, 0);
        h->cnt[st].assign(h->H, 0);
        for (int g = 0; g < h->H; ++g) {
            h->off[st][g] = (int)ntask;
            h->cnt[st][g] = (int)lists[st][g].size();
            ntask += lists[st][g].size();
        }
    }
    std::vector<MTask> all;
    all.reserve(ntask + state.size());
    for (int st = 0; st < 3; ++st)
        for (int g = 0; g < h->H; ++g) all.insert(all.end(), lists[st][g].begin(), lists[st][g].end());
    for (int& o : h->state_off) o += (int)ntask;
    all.insert(all.end(), state.begin(), state.end());
    MCK(malloc_zero(h, &h->d_tasks, all.size(), false), "alloc tasks");
    MCK(cudaMemcpyAsync(h->d_tasks, all.data(), sizeof(MTask) * all.size(), cudaMemcpyHostToDevice, h->stream),
        "upload tasks");
    {
        int r2 = setup_wide(h);
        if (r2) return r2;
    }
    MCK(cudaStreamSynchronize(h->stream), "setup sync");
    cudaFree(d_irs);
    h->allocs.erase(std::find(h->allocs.begin(), h->allocs.end(), (void*)d_irs));
    h->device_bytes -= (long long)sizeof(float) * n_in * n_out * ir_len;
    h->frame_num = 0;
    h->ready = true;
    return PC_OK;
}

int pcm_process_device(pcm_handle* h, float* d_out, const float* d_in, long long frames, int layout, void* stream) {
    if (!h) return PC_ERR_ARG;
    if (!h->ready) return mfail(h, PC_ERR_STATE, "process before setup");
    if (!d_out || !d_in || frames <= 0 || frames % h->N0)
        return mfail(h, PC_ERR_ARG, "frames must be a positive multiple of buffer_size");
    cudaSetDevice(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    RunState rs{};
    rs.io.in = d_in;
    rs.io.out = d_out;
    rs.io.step0 = h->frame_num;
    if (layout == PC_PLANAR) {
        rs.io.in_step = h->N0;
        rs.io.in_sample = 1;
        rs.io.in_ch = frames;
        rs.io.out_step = h->N0;
        rs.io.out_sample = 1;
        rs.io.out_ch = frames;
    } else {
        rs.io.in_step = (long long)h->N0 * h->nI;
        rs.io.in_sample = h->nI;
        rs.io.in_ch = 1;
        rs.io.out_step = (long long)h->N0 * h->nO;
        rs.io.out_sample = h->nO;
        rs.io.out_ch = 1;
    }
    const long long nsteps = frames / h->N0;
    // in place: one-block steps read a block before they write it, each as a call
    // of its own, which does not look back into its input as chunks do
    const bool in_place = overlap(d_in, frames * h->nI, d_out, frames * h->nO);
    bool wide = nsteps >= h->w_min && !in_place;
    if (wide) {
        const int r = ensure_wide(h, nsteps, st, &wide);
        if (r) return r;
    }
    if (wide) {
        int r = mimo_wide(h, rs.io, nsteps, st);
        if (r) return r;
    } else {
        for (long long s = 0; s < nsteps; ++s) {
            rs.step_base = h->frame_num + s;
            if (in_place) {
                rs.io.step0 = rs.step_base;
                rs.io.in = d_in + s * rs.io.in_step;
                rs.io.out = d_out + s * rs.io.out_step;
            }
            int r = mimo_step(h, rs, st, s == 0, nullptr);
            if (r) return r;
        }
        h->frame_num += nsteps;
    }
    MCK(record_use(h->used, st), "event record");
    return PC_OK;
}

int pcm_reset(pcm_handle* h) {
    if (!h) return PC_ERR_ARG;
    h->frame_num = 0;
    if (!h->ready) return PC_OK;
    h->work_failed = false;
    cudaSetDevice(h->device);
    MCK(cudaStreamWaitEvent(h->stream, h->used, 0), "reset");   // calls still running on a caller's stream
    for (auto& z : h->state) MCK(cudaMemsetAsync(z.first, 0, z.second, h->stream), "reset");
    MCK(launch_wide_reset(h->d_wlv, h->n_wlv, h->reset_bytes, nullptr, 0, h->stream), "reset");
    MCK(cudaStreamSynchronize(h->stream), "reset sync");
    return PC_OK;
}

int pcm_profile_kernels(pcm_handle* h, long long nsteps, pc_kernel_stats* out, int max_kinds, int* n_kinds) {
    if (!h || !h->ready || nsteps < 1 || !out) return PC_ERR_ARG;
    cudaSetDevice(h->device);
    // every step reads and writes the first block of zero-filled scratch I/O
    float* io = nullptr;
    const size_t ion = (size_t)h->N0 * std::max(h->nI, h->nO);
    MCK(cudaMalloc(&io, sizeof(float) * ion * 2), "profile buffer");
    cudaMemsetAsync(io, 0, sizeof(float) * ion * 2, h->stream);
    RunState rs{};
    rs.io.in = io;
    rs.io.out = io + ion;
    rs.io.step0 = 0;
    rs.io.in_sample = h->nI;
    rs.io.in_ch = 1;
    rs.io.out_sample = h->nO;
    rs.io.out_ch = 1;
    double ms[3] = {0, 0, 0}, bytes[3] = {0, 0, 0};
    long long cnt[3] = {0, 0, 0};
    std::vector<cudaEvent_t> evs;
    std::vector<int> phases;
    for (long long s = 0; s < nsteps; ++s) {
        cudaEvent_t e[6];
        for (auto& x : e) {
            cudaEventCreate(&x);
            evs.push_back(x);
        }
        rs.step_base = h->frame_num + s;
        phases.push_back((int)(rs.step_base & (h->H - 1)));
        int r = mimo_step(h, rs, h->stream, true, e);
        if (r) return r;
    }
    h->frame_num += nsteps;
    MCK(cudaStreamSynchronize(h->stream), "profile sync");
    for (long long s = 0; s < nsteps; ++s) {
        for (int k = 0; k < 3; ++k) {
            if (h->cnt[k][phases[s]] <= 0) continue;
            float t = 0;
            cudaEventElapsedTime(&t, evs[6 * s + 2 * k], evs[6 * s + 2 * k + 1]);
            ms[k] += t;
            cnt[k] += 1;
            if (k == 1) bytes[k] += h->mac_bytes[phases[s]];
        }
    }
    for (auto e : evs) cudaEventDestroy(e);
    cudaFree(io);
    static const char* names[3] = {"mimo_xfft", "mimo_mac", "mimo_yifft"};
    int n = 0;
    for (int k = 0; k < 3 && n < max_kinds; ++k) {
        if (!cnt[k]) continue;
        std::snprintf(out[n].name, sizeof out[n].name, "%s", names[k]);
        out[n].launches = cnt[k];
        out[n].total_ms = ms[k];
        out[n].alg_bytes = bytes[k];
        ++n;
    }
    if (n_kinds) *n_kinds = n;
    return PC_OK;
}

long long pcm_device_bytes(const pcm_handle* h) {
    return h ? h->device_bytes + (long long)(h->work_bytes + h->hw_bytes) : 0;
}
long long pcm_kernel_launches(const pcm_handle* h) { return h ? h->launches : 0; }
const char* pcm_last_error(const pcm_handle* h) { return h ? h->err.c_str() : ""; }

void pcm_destroy(pcm_handle* h) {
    if (!h) return;
    mfree(h);
    delete h;
}

}  // extern "C"

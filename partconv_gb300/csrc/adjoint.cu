// adjoint.cu -- differentiable partitioned convolution: block-parallel FDL
// forward pass and hand-written adjoint kernels.
//
// For a batch of signals x_s (length T) and one IR h, y_s = (x_s * h)[0:T].
// The whole signal is known, so nothing calls for the small blocks that a
// layout's first levels keep for latency: the layout given at creation is
// validated (src/partconv.cpp:87-181) and reported, and the computation takes
// one level of N-sample blocks, N the smallest power of two that covers the IR
// with at most 16 parts (256 .. 16384), with every block in parallel (the
// offline form of the streaming FDL of PartConvFilter::runLevel,
// src/partconv.cpp:354-490, run by wide.cu):
//   X_b = rfft(x[(b-1)N, (b+1)N)),  Y_b = sum_p X_{b-p} H_p,
//   H_p = rfft([0_N, h part p]) / 2N,  y block b = irfft(Y_b)[0:N]
// Backward with g = dL/dy:
//   dL/dx (adjoint, anti-causal): dL/dx[i] = sum_j h[j] g[i + j], the same
//     convolution run backwards in time over g, written backwards;
//   dL/dh (partitioned cross-correlation of the input with the gradient):
//     GP_b = rfft([g block b, 0_N]),  D_p = sum_s sum_b conj(GP_b) X_{b-p},
//     dh[pN + q] = irfft(D_p)[N - q] / 2N,  0 <= q < N.
// Sixteen parts: the products of T samples with an IR of L taps take
// (L / N)(T / N) N multiply-adds, so they fall with N while a transform's work
// per sample grows with log N only; below 16 parts the partial sums of D and the
// zero padding of short signals outweigh what is left.  Eight signals of 2^18
// samples, 2^16 taps, forward and backward: 463 us with the layout's own levels
// (512 and 4096: 8 + 15 parts, a walk per level), 222 us so, of which 142 us on
// the device and the rest in autograd's host path; three of 20011 samples,
// 4999 taps: 310 to 236 us, bound by that host path.
// The caller provides the workspace (no allocation here); the input spectra X
// can be kept from the forward pass or recomputed in the backward pass.
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
#include "fft_smem.cuh"
#include "kernels.h"
#include "wide.h"

using namespace pcg;

namespace {

constexpr int kMaxDLevels = 8;
constexpr int kMaxParts = 16;     // parts the block size is chosen for (and of one dL/dh pass)
constexpr int kMinBlock = 256;
constexpr int kRun = 16;          // blocks a thread of the dL/dh correlation sums

__host__ __device__ constexpr int job_threads(int logN) { return logN <= 11 ? 128 : 1 << (logN - 4); }

// Transforms of windows with one zero half: rows of H (h part p in the second
// half, scaled) or of GP (g block b in the first half).
struct WinArgs {
    const float* src;     // h, or dL/dy
    float2* dst;          // rows of cs
    const float2* tab;
    long long len;        // samples per signal
    int rows, per_sig;    // rows in all, per signal
    int cs, second;       // live half of the window
    float scale;
};
template <int LOGN>
__global__ void __launch_bounds__(job_threads(LOGN)) dwin_fft_kernel(WinArgs a) {
    constexpr int NT = job_threads(LOGN);
    using F = RegFft<LOGN, NT>;
    constexpr int N = F::N, TPT = F::TPT;
    extern __shared__ float4 dyn_smem[];
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = reinterpret_cast<float2*>(dyn_smem) + tr * F::SM;
    const int row = blockIdx.x * (NT / TPT) + tr;
    const bool live = row < a.rows;
    if (TPT >= 32 && !live) return;
    const int r = min(row, a.rows - 1), sig = r / a.per_sig, b = r - sig * a.per_sig;
    const float* src = a.src + sig * a.len + (long long)b * N;
    const long long left = a.len - (long long)b * N;   // live samples of the block
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) v[m] = make_float2(0.f, 0.f);
    // window pairs n < N / 2 are the first half, v[0 .. 7]
    float2 u[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int i = 2 * (t + m * TPT);
        u[m] = make_float2(i < left ? src[i] : 0.0f, i + 1 < left ? src[i + 1] : 0.0f);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (a.second) v[m + 8] = u[m];
        else v[m] = u[m];
    }
    fft_reg<LOGN, NT, false, true>(v, t, s, a.tab);
    F::sync();
#pragma unroll
    for (int m = 8; m < 16; ++m) s[rpad(t + m * TPT)] = v[m];
    F::sync();
    if (!live) return;
    float2* d = a.dst + (size_t)r * a.cs;
    const float2* sp = a.tab + ft_sp(LOGN);
    auto put = [&](int k, float2 x) { d[k] = make_float2(x.x * a.scale, x.y * a.scale); };
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int k = t + m * TPT;
        float2 xk, xnk;
        if (m == 0 && t == 0) split_zero(v[0], xk, xnk);
        else split_w(v[m], s[rpad(N - k)], __ldg(sp + k), xk, xnk);
        put(k, xk);
        put(N - k, xnk);
    }
    if (t == 0) {
        float2 xk, xnk;
        split_w(v[8], v[8], __ldg(sp + N / 2), xk, xnk);
        put(N / 2, xk);
    }
}

// dh[p N + q] = irfft(D_p)[N - q] / 2N, q < N, p N + q < len
template <int LOGN>
__global__ void __launch_bounds__(job_threads(LOGN)) dtap_ifft_kernel(const float2* __restrict__ D, int P, int cs,
                                                                      const float2* __restrict__ tab, float* gh, int len) {
    constexpr int NT = job_threads(LOGN);
    using F = RegFft<LOGN, NT>;
    constexpr int N = F::N, TPT = F::TPT;
    extern __shared__ float4 dyn_smem[];
    const int t = threadIdx.x % TPT, tr = threadIdx.x / TPT;
    float2* s = reinterpret_cast<float2*>(dyn_smem) + tr * F::SM;
    const int row = blockIdx.x * (NT / TPT) + tr;
    const bool live = row < P;
    if (TPT >= 32 && !live) return;
    const int p = min(row, P - 1);
    const float2* Y = D + (size_t)p * cs;
    const float2* sp = tab + ft_sp(LOGN);
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
        const int n = t + m * TPT;
        float2 yn = __ldcg(Y + n), yc = __ldcg(Y + N - n), other;
        if (m < 8) {
            if (m == 0 && t == 0) yn.y = yc.y = 0.0f;
            merge_w(yn, yc, __ldg(sp + n), v[m], other);
        } else {
            merge_w(yc, yn, __ldg(sp + N - n), other, v[m]);
        }
    }
    fft_reg<LOGN, NT, true, true>(v, t, s, tab);
    if (!live) return;
    // real samples 2 n, 2 n + 1 in v[m], n = t + m TPT; taps q = N - i, 0 < i <= N
    const float scale = 1.0f / (2.0f * N);
    float* d = gh + (size_t)p * N;
    const int live_taps = min(N, len - p * N);
    auto put = [&](int i, float y) {
        const int q = N - i;
        if (q >= 0 && q < live_taps) d[q] = y * scale;
    };
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        const int i = 2 * (t + m * TPT);
        if (i <= N) {
            put(i, v[m].x);
            put(i + 1, v[m].y);
        }
    }
}

// Dpart[sig * nrun + run][p][k] = sum over the run's blocks b of
// conj(GP[sig][b][k]) X[sig][b-p][k], parts p0 <= p < p0 + 16 (blockIdx.y), the
// bin's last 16 input spectra in registers: each spectrum is loaded once per
// pass instead of once per part, four blocks' loads in flight.  The products
// are rounded before they are added (one rounding of the sum each).
// Bound: latency of two rows per block (63 of 8 x 64 blocks x 4098 bins x 16
// parts are 34 M products, 15 us of packed arithmetic; measured 26 us).
__global__ void __launch_bounds__(128) ddh_slide_kernel(const float2* __restrict__ X, const float2* __restrict__ GP,
                                                        float2* __restrict__ Dpart, int nsig, int nb, int slots, int P,
                                                        int cs) {
    constexpr int U = 4;
    const int nrun = (nb + kRun - 1) / kRun;
    const long long t = blockIdx.x * 128LL + threadIdx.x;
    if (t >= (long long)nsig * nrun * cs) return;
    const int k = (int)(t % cs);
    const int sr = (int)(t / cs), run = sr % nrun, sg = sr / nrun;
    const int p0 = blockIdx.y * kMaxParts;
    const f32x2* Xs = reinterpret_cast<const f32x2*>(X + (size_t)sg * slots * cs + k);
    const float2* Gs = GP + (size_t)sg * nb * cs + k;
    const int b0 = run * kRun, b1 = min(nb, b0 + kRun);
    auto xat = [&](int b) { return b >= 0 ? __ldcg(Xs + (size_t)b * cs) : 0ULL; };
    // w[(p + i) mod 16 from the newest]: block b - p0 - p at step i of the unrolled sixteen
    f32x2 w[kMaxParts], acc[kMaxParts];
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p) {
        acc[p] = 0;
        w[(kMaxParts - 1 - p)] = p < kMaxParts - 1 ? xat(b0 - 1 - p0 - p) : 0;   // slot (15 - p): the block p before b0 - 1
    }
    // at step i the newest block goes to slot i, the block p older to slot (i - p) mod 16
    for (int bb = b0; bb < b1; bb += kMaxParts) {
#pragma unroll
        for (int i0 = 0; i0 < kMaxParts; i0 += U) {
            if (bb + i0 >= b1) break;
            f32x2 xn[U];
            float2 g[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int b = bb + i0 + u;
                if (b < b1) {
                    xn[u] = xat(b - p0);
                    g[u] = __ldcg(Gs + (size_t)b * cs);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (bb + i0 + u >= b1) break;
                const int i = i0 + u;
                w[i] = xn[u];
                // conj(g) x = (g.re x.re + g.im x.im, g.re x.im - g.im x.re)
                const f32x2 gr = pack2(g[u].x, g[u].x), gi = pack2(g[u].y, -g[u].y);
#pragma unroll
                for (int p = 0; p < kMaxParts; ++p)
                    if (p0 + p < P) {
                        const f32x2 x = w[(i - p + kMaxParts) % kMaxParts];
                        acc[p] = add2(acc[p], fma2(x, gr, mul2(swap2(x), gi)));
                    }
            }
        }
    }
    float2* D = Dpart + ((size_t)sr * P + p0) * cs + k;
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p)
        if (p0 + p < P) D[(size_t)p * cs] = unpack2(acc[p]);
}

// D[p][k] = sum of the nchunk partial rows, in order, eight loads in flight
__global__ void ddh_reduce_kernel(const float2* __restrict__ Dpart, float2* __restrict__ D, int total, int nchunk) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    constexpr int U = 8;
    float2 acc = make_float2(0.f, 0.f);
    for (int c0 = 0; c0 < nchunk; c0 += U) {
        float2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + u < nchunk) v[u] = __ldcg(Dpart + (size_t)(c0 + u) * total + t);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + u < nchunk) acc = cadd(acc, v[u]);
    }
    D[t] = acc;
}

// f.template operator()<LOGN>() for block sizes 256 .. 16384
template <class Fn>
cudaError_t by_block(int N, Fn&& f) {
    switch (N) {
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
constexpr size_t job_smem(int nt) { return sizeof(float2) * 17 * (size_t)nt; }

struct WinFft {
    const WinArgs& a;
    cudaStream_t st;
    template <int L>
    cudaError_t operator()() const {
        constexpr int NT = job_threads(L), per = NT * 16 >> L;
        dwin_fft_kernel<L><<<(a.rows + per - 1) / per, NT, job_smem(NT), st>>>(a);
        return cudaGetLastError();
    }
};
struct TapIfft {
    const float2* D;
    int P, cs;
    const float2* tab;
    float* gh;
    int len;
    cudaStream_t st;
    template <int L>
    cudaError_t operator()() const {
        constexpr int NT = job_threads(L), per = NT * 16 >> L;
        dtap_ifft_kernel<L><<<(P + per - 1) / per, NT, job_smem(NT), st>>>(D, P, cs, tab, gh, len);
        return cudaGetLastError();
    }
};
struct Prepare {
    template <int L>
    cudaError_t operator()() const {
        const int b = (int)job_smem(job_threads(L));
        cudaError_t e = cudaFuncSetAttribute(dwin_fft_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(dtap_ifft_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
        return e;
    }
};

}  // namespace

struct pcd_plan {
    int B = 0, ir_len = 0;
    long long T = 0;
    int N = 0, logN = 0, P = 0, cs = 0, nb = 0, slots = 0, nrun = 0;   // P: parts that reach the output
    // workspace offsets (bytes)
    size_t o_H = 0, o_X = 0, o_Y = 0, o_Dp = 0, o_D = 0, total = 0;
    // device tables (built at creation): transform factors, level descriptors of
    // the signals (pointers relative to the workspace), CTA maps
    char* d_tab = nullptr;
    const float2* tab = nullptr;
    const WLevel* lv = nullptr;
    const int2 *m_fft = nullptr, *m_out = nullptr;
    const int4* m_mac = nullptr;
    int n_fft = 0, n_out = 0, n_mac = 0, nt = 0;
    int device = -1;
    std::string err;
    long long launches = 0;
    ~pcd_plan() {
        if (d_tab) {
            int cur = -1;
            cudaGetDevice(&cur);
            if (device >= 0) cudaSetDevice(device);
            cudaFree(d_tab);
            if (cur >= 0) cudaSetDevice(cur);
        }
    }
};

namespace {

size_t take(size_t& off, size_t bytes) {
    size_t o = off;
    off += (bytes + 255) & ~(size_t)255;
    return o;
}

int dfail(pcd_plan* p, int code, const std::string& m) {
    if (p) p->err = m;
    return code;
}

#define DCK(call, where)                                                                                   \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return dfail(p, PC_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
T* at(void* ws, size_t off) {
    return reinterpret_cast<T*>(static_cast<char*>(ws) + off);
}

// in -> in * h over every signal, or with rev both read and written backwards
// in time; spectra of `in` stay in the workspace's X rows
int convolve(pcd_plan* p, const float* in, float* out, void* ws, bool rev, bool windows, cudaStream_t st) {
    WArgs a{};
    a.lv = p->lv;
    a.tab = p->tab;
    a.N0 = p->N;
    a.kb = 1;
    a.full = 1;
    a.nsteps = p->nb;
    a.rel = (long long)reinterpret_cast<unsigned long long>(ws);
    a.len = p->T;
    const long long last = rev ? p->T - 1 : 0;
    a.io.in = in + last;
    a.io.out = out + last;
    a.io.in_sample = a.io.out_sample = rev ? -1 : 1;
    a.io.in_ch = a.io.out_ch = p->T;
    a.vec_in = !rev && (p->B == 1 || p->T % 2 == 0) && (reinterpret_cast<uintptr_t>(in) & 7) == 0;
    a.vec_out = !rev && (p->B == 1 || p->T % 2 == 0) && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    if (windows) {
        DCK(launch_wide_fft(false, p->nt, p->n_fft, p->m_fft, a, st), "window FFT");
        p->launches++;
    }
    if (out) {
        DCK(launch_wide_mac(false, p->n_mac, p->m_mac, a, st), "sum over parts");
        DCK(launch_wide_out(p->N, p->n_out, p->m_out, a, st), "inverse FFT");
        p->launches += 2;
    }
    return PC_OK;
}

int filter_spectra(pcd_plan* p, const float* h, void* ws, cudaStream_t st) {
    WinArgs a{h, at<float2>(ws, p->o_H), p->tab, p->ir_len, p->P, p->P, p->cs, 1, 1.0f / (2.0f * p->N)};
    DCK(by_block(p->N, WinFft{a, st}), "filter spectra");
    p->launches++;
    return PC_OK;
}

// level descriptors, maps and transform factors on the device
int build_tables(pcd_plan* p) {
    std::vector<char> blob;
    auto put = [&](const void* src, size_t bytes) {
        const size_t o = blob.size();
        blob.resize(o + ((bytes + 255) & ~(size_t)255));
        if (bytes) std::memcpy(blob.data() + o, src, bytes);
        return o;
    };
    std::vector<WLevel> lv;
    std::vector<int2> fft, out;
    std::vector<int4> mac;
    auto rel = [](size_t off) { return reinterpret_cast<float2*>(off); };   // completed by WArgs::rel
    const size_t row = sizeof(float2) * (size_t)p->cs;
    p->nt = p->N <= 2048 ? 128 : (p->N <= 4096 ? 256 : 1024);
    for (int s = 0; s < p->B; ++s) {
        WLevel w{};
        w.N = p->N;
        w.logN = p->logN;
        w.P = p->P;
        w.cs = p->cs;
        w.slots = p->slots;
        w.p_lo = 2;
        w.tp = 16;
        w.tpg = 4;
        w.nrows = p->P > 2 ? (p->P - 2 + 15) / 16 : 0;
        w.two = 1;
        w.in_ch = w.out_ch = s;
        w.mix_mode = 1;
        w.M = 1;
        w.lv0 = s;
        w.scale = 1.0f;
        w.H = rel(p->o_H);
        w.X = rel(p->o_X + row * p->slots * s);
        w.Yw = rel(p->o_Y + row * p->nb * s);
        lv.push_back(w);
    }
    // a segment of few enough blocks that there are CTAs for every SM
    int seg = kMacSeg;
    const long long tiles = (p->cs + kMacTile - 1) / kMacTile;
    while (seg > kWideRun && tiles * p->B * ((p->nb + seg - 1) / seg) < 4 * 152) seg >>= 1;
    for (int s = 0; s < p->B; ++s) {
        for (int b = 0; b < p->nb; b += 16 * p->nt / p->N) fft.push_back(make_int2(s, b));
        for (int b = 0; b < p->nb; b += wide_out_blocks(p->N)) out.push_back(make_int2(s, b));
        for (int b = 0; b < p->nb; b += seg)
            for (int k = 0; k < p->cs; k += kMacTile) mac.push_back(make_int4(s, k, b, std::min(p->nb, b + seg)));
    }
    p->n_fft = (int)fft.size();
    p->n_out = (int)out.size();
    p->n_mac = (int)mac.size();
    const auto& t = host_fft_tables();
    const size_t o_t = put(t.data(), sizeof(float2) * t.size());
    const size_t o_lv = put(lv.data(), sizeof(WLevel) * lv.size());
    const size_t o_f = put(fft.data(), sizeof(int2) * fft.size());
    const size_t o_o = put(out.data(), sizeof(int2) * out.size());
    const size_t o_m = put(mac.data(), sizeof(int4) * mac.size());
    DCK(cudaGetDevice(&p->device), "cudaGetDevice");
    DCK(cudaMalloc(&p->d_tab, blob.size()), "table allocation");
    DCK(cudaMemcpy(p->d_tab, blob.data(), blob.size(), cudaMemcpyHostToDevice), "table upload");
    p->tab = reinterpret_cast<const float2*>(p->d_tab + o_t);
    p->lv = reinterpret_cast<const WLevel*>(p->d_tab + o_lv);
    p->m_fft = reinterpret_cast<const int2*>(p->d_tab + o_f);
    p->m_out = reinterpret_cast<const int2*>(p->d_tab + o_o);
    p->m_mac = reinterpret_cast<const int4*>(p->d_tab + o_m);
    DCK(prepare_wide_kernels(), "kernel attributes");
    if (p->N > 2048) DCK(by_block(p->N, Prepare{}), "kernel attributes");
    return PC_OK;
}

}  // namespace

extern "C" {

pcd_plan* pcd_create(int M, const int* N, int* P, int ir_len, int batch, long long length, char* msg, int msglen) {
    auto put = [&](const char* m) {
        if (msg && msglen > 0) snprintf(msg, msglen, "%s", m);
    };
    if (M < 1 || M > kMaxDLevels || !N || !P || ir_len < 1 || batch < 1 || length < 1) {
        put("bad plan arguments");
        return nullptr;
    }
    std::vector<int> Nv(N, N + M), Pv(P, P + M);
    char m2[256];
    if (pc_check_layout(M, Nv.data(), Pv.data(), ir_len, 1, nullptr, m2, sizeof m2)) {
        put(m2);
        return nullptr;
    }
    if (Nv[M - 1] > kMaxBlockOneCta) {
        put("differentiable levels are limited to blocks of 16384 (larger blocks: pc_* engine)");
        return nullptr;
    }
    if (Nv[0] < 16) {
        put("block size of level 0 must be >= 16");
        return nullptr;
    }
    for (int i = 0; i < M; ++i) P[i] = Pv[i];
    pcd_plan* p = new (std::nothrow) pcd_plan();
    if (!p) return nullptr;
    p->B = batch;
    p->ir_len = ir_len;
    p->T = length;
    // the smallest block with at most kMaxParts parts, no larger than the signal needs
    p->N = kMinBlock;
    while (p->N < kMaxBlockOneCta && p->N < length && (long long)p->N * kMaxParts < ir_len) p->N <<= 1;
    while ((1 << p->logN) < p->N) ++p->logN;
    p->cs = p->N + 2;
    p->nb = (int)((length + p->N - 1) / p->N);
    p->P = std::min((ir_len + p->N - 1) / p->N, p->nb);   // later parts reach no output sample
    p->slots = p->P + std::max(p->nb, kWideRun);
    p->nrun = (p->nb + kRun - 1) / kRun;
    const size_t row = sizeof(float2) * (size_t)p->cs;
    size_t off = 0;
    p->o_H = take(off, row * p->P);
    p->o_X = take(off, row * p->slots * batch);
    p->o_Y = take(off, row * p->nb * batch);
    p->o_Dp = take(off, row * p->P * p->nrun * batch);
    p->o_D = take(off, row * p->P);
    p->total = off;
    if (build_tables(p) != PC_OK) {
        put(p->err.c_str());
        delete p;
        return nullptr;
    }
    put("");
    return p;
}

long long pcd_workspace_bytes(const pcd_plan* p) { return p ? (long long)p->total : -1; }

int pcd_forward(pcd_plan* p, const float* d_x, const float* d_h, float* d_y, void* d_ws, void* stream) {
    if (!p || !d_x || !d_h || !d_y || !d_ws) return dfail(p, PC_ERR_ARG, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    int r = filter_spectra(p, d_h, d_ws, st);
    return r ? r : convolve(p, d_x, d_y, d_ws, false, true, st);
}

int pcd_backward(pcd_plan* p, const float* d_x, const float* d_h, const float* d_gy, float* d_gx, float* d_gh,
                 void* d_ws, int recompute, void* stream) {
    if (!p || !d_gy || !d_ws) return dfail(p, PC_ERR_ARG, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    int r;
    if (recompute) {   // rebuild what the forward pass left in the workspace
        if (!d_x || !d_h) return dfail(p, PC_ERR_ARG, "recompute needs x and h");
        if (d_gx && (r = filter_spectra(p, d_h, d_ws, st))) return r;
        if (d_gh && (r = convolve(p, d_x, nullptr, d_ws, false, true, st))) return r;
    }
    // dL/dh first: it needs the input spectra X, which the adjoint pass below
    // overwrites with those of the gradient
    if (d_gh) {
        float2* GP = at<float2>(d_ws, p->o_Y);
        float2 *Dp = at<float2>(d_ws, p->o_Dp), *D = at<float2>(d_ws, p->o_D);
        const WinArgs a{d_gy, GP, p->tab, p->T, p->B * p->nb, p->nb, p->cs, 0, 1.0f};   // GP_b = rfft([g block b, 0_N])
        DCK(by_block(p->N, WinFft{a, st}), "gradient windows");
        const long long tot = (long long)p->B * p->nrun * p->cs;
        const int total = p->P * p->cs;
        ddh_slide_kernel<<<dim3((unsigned)((tot + 127) / 128), (p->P + kMaxParts - 1) / kMaxParts), 128, 0, st>>>(
            at<float2>(d_ws, p->o_X), GP, Dp, p->B, p->nb, p->slots, p->P, p->cs);
        ddh_reduce_kernel<<<(total + 127) / 128, 128, 0, st>>>(Dp, D, total, p->B * p->nrun);
        DCK(cudaGetLastError(), "dL/dh correlation");
        DCK(by_block(p->N, TapIfft{D, p->P, p->cs, p->tab, d_gh, p->ir_len, st}), "dL/dh taps");
        p->launches += 4;
        const long long done = (long long)p->P * p->N;
        if (done < p->ir_len)   // taps beyond the signal's length
            DCK(cudaMemsetAsync(d_gh + done, 0, sizeof(float) * (p->ir_len - done), st), "dL/dh taps");
    }
    return d_gx ? convolve(p, d_gy, d_gx, d_ws, true, true, st) : PC_OK;
}

void pcd_destroy(pcd_plan* p) { delete p; }
const char* pcd_last_error(const pcd_plan* p) { return p ? p->err.c_str() : ""; }
long long pcd_kernel_launches(const pcd_plan* p) { return p ? p->launches : 0; }

}  // extern "C"

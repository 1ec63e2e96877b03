// wide.h -- block-parallel processing of many base steps of a handle
// (wide.cu): the interface the engine uses.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "engine_types.h"

namespace pcg {

// One level of one PC, as the block-parallel kernels read it.
struct WLevel {
    int N, logN, P, logT;
    int s_blocks, cs, slots, rmask;
    int nrows;      // partial-sum rows (groups of parts >= p_lo)
    int p_lo;       // first part of the rows
    int form;       // order of the sum over parts: kFormFire, kFormCluster or kFormMulti
    int two;        // the fire adds X_{b-1} H_1 itself
    int in_ch, out_ch, mix_mode, M;
    int rin_mask, lv0, dfer, pad;
    float scale;
    float pad2;
    const float2* H;
    float2* X;
    float2* Yw;     // [blocks of a chunk][cs]
    float2* Yp;
    float* yring;
    float* xring;
    float* pcw;     // [chunk samples], mixed outputs only
};
enum { kFormFire = 0, kFormCluster = 1, kFormMulti = 2 };

struct WArgs {
    const WLevel* lv;
    const float2* tab;    // build_fft_tables
    const float2* W;      // 2^wlog twiddles (cluster transforms)
    int wlog, N0;
    long long c0;         // first base step of the chunk
    int nsteps, kb;       // base steps of the chunk; base blocks per step of the handle
    int vec_in, vec_out;  // contiguous channels, 8-byte aligned: float2 loads and stores
    IOView io;
};

constexpr int kWideMacNT = 128;
// consecutive blocks a thread of the sum over parts takes together; G is the
// number of running sums per block (fewer blocks where there are more sums,
// so that all stay in registers)
__host__ __device__ constexpr int wide_run(int G = 1) { return G <= 4 ? 8 : 32 / G; }

// CTA maps: (level, first block of the chunk) for the transforms, (level,
// first of kWideMacNT (run, bin) items) for the sum over parts.
int wide_transforms_per_cta(int N);
cudaError_t prepare_wide_kernels();
cudaError_t launch_wide_fft(int N, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// l0: level 0 (writes the output), else a larger level (writes its output ring)
cudaError_t launch_wide_ifft(int N, bool l0, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// G: part groups of the handle's spread tasks, tp: parts per task
cudaError_t launch_wide_mac(int G, int tp, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// outputs fed by several PCs, and outputs without any
cudaError_t launch_wide_mix(const Bank& bank, int n_zero, bool mixed, const WArgs& a, cudaStream_t st);
// the newest samples of a call of `frames` samples appended to every PC's input ring
cudaError_t launch_wide_ring(const WLevel* lv, const int* lv0, int npc, const WArgs& a, long long t_end,
                             long long frames, int max_ring, cudaStream_t st);
// class-3 levels (cluster_fire.cu)
cudaError_t launch_wide_cluster(bool inverse, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// partial sums of the blocks in progress after step c1 - 1 (step_kernels.cu);
// map: (level, first bin, row, end bin) of a tile
cudaError_t launch_wide_partials(int nt, int lanes, int grid, const int4* map, const WLevel* lv, int tp, long long c1,
                                 int kb, cudaStream_t st);

}  // namespace pcg

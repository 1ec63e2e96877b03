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
    int multi;      // level 0 with several base blocks per step: parts < p_lo are one running sum
    int two;        // the fire adds X_{b-1} H_1 itself
    int in_ch, out_ch, mix_mode, M;
    int rin_mask, lv0, dfer;
    int tp, tpg;    // parts per partial-sum row, and per group within one
    float scale;
    const float2* H;
    float2* X;
    float2* Yw;     // [blocks of a chunk][cs]
    float2* Yp;
    float* yring;
    float* xring;   // null: silence before the call
    float* pcw;     // [chunk samples], mixed outputs only
};

struct WArgs {
    const WLevel* lv;
    const float2* tab;    // build_fft_tables
    const float2* W;      // 2^wlog twiddles (cluster transforms)
    int wlog, N0;
    long long c0;         // first base step of the chunk
    int nsteps, kb;       // base steps of the chunk; base blocks per step of the handle
    int vec_in, vec_out;  // contiguous channels, 8-byte aligned: float2 loads and stores
    int full;             // every twiddle factor from the table (fft_reg.cuh)
    long long rel;        // added (bytes) to the descriptors' H, X and Yw: a workspace given per call
    long long len;        // samples of the call's input and output; silence after them (0: whole blocks)
    IOView io;
};
// descriptor pointer p of a launch with a.rel
template <class T>
__host__ __device__ __forceinline__ T* wide_at(T* p, long long rel) {
    return reinterpret_cast<T*>(reinterpret_cast<unsigned long long>(p) + rel);
}

constexpr int kWideRun = 8;       // consecutive blocks a thread of the sum over parts takes together
constexpr int kMacTile = 96;      // bins per CTA of the sum over parts (three warps: 258 bins are tiles of 96, 96 and 66)
constexpr int kMacSeg = 32;       // ... and blocks
constexpr int kMacRes = 18;       // most parts whose filter rows stay in shared memory (16 of a partial-sum row and 2)
constexpr int kMacRows = 59;      // shared rows of a tile (45 KB; registers admit four CTAs per SM)
constexpr int kMacAnyNT = 128;    // threads of the general form

// CTA maps: (level, first block of the chunk) for the transforms; for the sum
// over parts (level, first bin, first block, end block) of a tile and segment,
// or (level, first of kMacAnyNT (run, bin) items) in the general form.
cudaError_t prepare_wide_kernels();
// frames of interleaved samples (at least two channels) to rows pitch apart
cudaError_t launch_wide_planar(const float* in, float* out, int channels, long long pitch, long long frames,
                               cudaStream_t st);
// threads per CTA of the transform kernels for blocks up to max_n (a CTA runs
// 16 threads / N transforms), and blocks per CTA of wide_out
int wide_threads(int max_n);
int wide_out_blocks(int N0);
// (nt = 256: forward transforms of blocks up to 4096; dep = false: tables that the kernel reads are still being written by the stream's last kernel)
cudaError_t launch_wide_fft(bool inverse, int nt, int grid, const int2* map, const WArgs& a, cudaStream_t st,
                            bool dep = true);
// level 0: inverse transforms and the call's output
cudaError_t launch_wide_out(int N0, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// any: tile shapes other than the default, or level 0 with several base blocks per step
cudaError_t launch_wide_mac(bool any, int grid, const int4* map, const WArgs& a, cudaStream_t st);
// outputs fed by several PCs, and outputs without any
cudaError_t launch_wide_mix(const Bank& bank, int n_zero, bool mixed, const WArgs& a, cudaStream_t st);
// clears what a run from the start reads before it writes it: spectrum rows,
// output rings (at most level_bytes of each level), and the state region (16-byte
// aligned)
cudaError_t launch_wide_reset(const WLevel* lv, int nlv, size_t level_bytes, void* state, size_t bytes, cudaStream_t st);
inline size_t wide_reset_bytes(const WLevel& l, int N0) {
    return sizeof(float2) * (size_t)(l.P - 1) * l.cs + sizeof(float) * (size_t)l.s_blocks * N0;
}
// what the rings of lv hold for the steps from `step` on, to the rings of to
cudaError_t launch_wide_move(const WLevel* lv, const WLevel* to, int nlv, long long step, int N0, cudaStream_t st);
// class-3 levels (cluster_fire.cu)
cudaError_t launch_wide_cluster(bool inverse, int grid, const int2* map, const WArgs& a, cudaStream_t st);
// the state one-block steps would have left after step a.c0 - 1
// (step_kernels.cu): the partial sums of the blocks in progress, by n_part
// CTAs of map (level, first bin, row, end bin), and the newest samples of the
// call (which began at step a.io.step0) in the input rings of npc PCs
cudaError_t launch_wide_state(int nt, int lanes, int n_part, const int4* map, const int* lv0, int npc, int max_ring,
                              const WArgs& a, cudaStream_t st);

}  // namespace pcg

// What the host side of the fast path (das_fast.cu) shares with its kernels
// (das_fast_kernel.cuh, instantiated by das_fast_*.cu so that they compile in parallel).
#pragma once

#include "common.cuh"

namespace ustb {

constexpr int kTile = USTB_TILE_PIXELS;
constexpr int kThreads = 256;  // threads of a beamforming CTA
constexpr int kSub = 2;        // sub-tiles (CTAs) per tile

// Interpolation entries of a sample: {x_i, x_{i+1} - x_i} in FP32, or for complex 16-bit
// storage {x_i, x_{i+1}} as they are stored.
enum EntryKind { kEntReal = 0, kEntComplex = 1, kEntHalf = 2, kEntBf16 = 3 };
constexpr int entry_size(int ent) { return ent == kEntComplex ? 16 : 8; }

struct Params {
    const void* entries;  // [F][W][N][Lp] interpolation entries of kind `ent`
    int ent;
    int64_t L, Lp, N, W, F, P;
    const float* el;
    const float* px;
    const int32_t* tiles;
    int64_t n_tiles;
    const ustb_wave* waves;
    const float* tx_delay_tab;
    const float* tx_apo_tab;
    const float* rx_apo_tab;
    const float2* pix_phase;
    float fs, t0, fd, c, inv_c, lens;
    double fd_fs;  // fd / fs
    double fs_c;   // fs / c
    int64_t wave_step, frame_step;  // entries from a wave (a frame) to the next
    int rx_window;
    float win_r1, win_a, win_e, win_b, win_c, win_d;  // see window_coeffs()
    float fnx, fny, minx, miny, maxx, maxy;
    int rx_origin;
    float ox, oy, oz;
    float cf_thr;
    void* cube;
    float2* o_das;
    float* o_cf;
    float2* o_cfimg;
    float* o_sdmas;
    int64_t rx_f, w_f, f_f;
    uint32_t* flags;
    bool after_entries; // grid kernel: the entries pre-pass is the launch before it
    int split;          // grid kernel: CTAs (parts) per sub-tile
    float2* partial;    // sums of the parts [F * sub-tiles][split][1, or 3 for the epilogue][kThreads]
    unsigned* tickets;  // parts that have finished, per frame and sub-tile (zeroed)
    int shape;  // stage shape (Shape<> index)
    int fpi;    // persistent kernel: frames per work item (one tile, consecutive frames)
};

// Kernel variant of (dimension, epilogue, stage shape) for one request kind: one grid
// launch of reqs[0] (BATCH false) or one persistent launch of n requests.
template <int ENT, bool BATCH>
int das_dispatch(int dim, int epi, int shape, const Params* reqs, const int64_t* frames, int n,
                 unsigned long long* counter, int64_t nt, int64_t F, cudaStream_t s, int max_ctas);

constexpr int kMaxBatch = 40;  // requests per persistent launch

}  // namespace ustb

// What the host side of the fast path (das_fast.cu) shares with its kernels
// (das_fast_kernel.cuh, instantiated by das_fast_*.cu so that they compile in parallel).
#pragma once

#include "common.cuh"

namespace ustb {

constexpr int kTile = USTB_TILE_PIXELS;

// Stage shapes: a stage is cg channels x kw waves (channel, wave) slots.
//   shape 0: waves outer (2 channels x 16 waves); per-wave accumulators, the
//            receive geometry of a channel is formed once per 16-wave chunk
//   shape 1: channels outer (8 channels x 4 waves); per-channel accumulators,
//            the receive geometry is formed once per (pixel, channel) and the
//            transmit geometry once per stage
//   shape 2: channels outer (16 channels x 2 waves)
//   shapes 3, 4, 5: waves outer (8 x 4, 16 x 2, 4 x 8), dimension.receive
// dimension.receive needs waves outer, dimension.transmit/none channels outer;
// dimension.both runs with any of the first three.  A sub-tile of complex data whose windows
// do not fit 80-entry slots runs half-size stages with 160-entry slots (half the
// channels of a waves-outer stage, half the waves of a channels-outer one) in the same
// buffers; real entries are half as large and always have 160-entry slots.
struct StageShape {
    int cg, kw;
    bool waves_outer;
};
constexpr StageShape kShapes[6] = {{2, 16, true}, {8, 4, false}, {16, 2, false}, {8, 4, true}, {16, 2, true}, {4, 8, true}};

constexpr int kBufBytes = 40960;  // a stage buffer: 32 slots x 80 or 16 x 160 complex entries, 32 x 160 real
constexpr int kRing = 2;          // stage buffers: stage s + kRing - 1 is copied during stage s
constexpr size_t kBuffers = (size_t)kRing * kBufBytes;

// Shared memory of one CTA: kRing stage buffers, then the per-tile tables (their size
// depends on N, W and the stage shape): byte offsets, 16-byte records first.
struct TileTables {
    size_t el4, txc, txp, win_w, rxp, base_w, len_n, olist, kind_w, total;
};

// Per-channel tables hold NP and per-wave tables WP records, the counts rounded up to
// whole stages: the channels / waves past N / W are padding with zero weight, so a
// stage never needs bounds checks.
__host__ __device__ __forceinline__ TileTables tile_tables(StageShape s, int64_t NP, int64_t WP) {
    // counts of channel groups and wave chunks, of the smaller stages where there are two
    const int64_t NG = NP / (s.waves_outer ? s.cg / 2 : s.cg), NC = WP / (s.waves_outer ? s.kw : s.kw / 2);
    TileTables t;
    size_t o = 0;
    t.el4 = o;    o += 16 * NP;        // float4 per channel: x, y, z, delay base
    t.txc = o;    o += 16 * WP;        // float4 per wave: delay coefficients
    t.txp = o;    o += 16 * WP;        // float4 per wave: phase offset, apodization, fs/c, window offset
    t.win_w = o;  o += 8 * WP;         // {window start, its largest position as a float (sign bit: inactive)} per wave
    t.rxp = o;    o += 8 * NP;         // float2 per channel: phase (cycles) of the delay base, window offset
    t.base_w = o; o += 4 * WP;         // delay base of each wave
    t.len_n = o;  o += 4 * NP;         // largest window position of each channel (< 0: inactive)
    t.olist = o;  o += 2 * (NG + NC);  // active outer indices, then active inner indices (16 bits)
    t.kind_w = o; o += WP;
    t.total = (o + 15) & ~size_t(15);
    return t;
}
inline size_t smem_bytes(int shape, int64_t N, int64_t W) {
    const StageShape s = kShapes[shape];
    return kBuffers + tile_tables(s, (N + s.cg - 1) / s.cg * s.cg, (W + s.kw - 1) / s.kw * s.kw).total;
}

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
    int subs;   // sub-tiles (CTAs) per tile: 2, or 1 (see subs_for)
};

// Kernel variant of (dimension, epilogue, stage shape) for one request kind and number of
// sub-tiles: one grid launch of reqs[0] (BATCH false) or one persistent launch of n requests.
template <int ENT, bool BATCH, int SUBS>
int das_dispatch(int dim, int epi, int shape, const Params* reqs, const int64_t* frames, int n,
                 unsigned long long* counter, int64_t nt, int64_t F, cudaStream_t s, int max_ctas);

// CTAs of a beamforming kernel with `smem` bytes of dynamic shared memory that an SM has
// room for: 2, or 1.
int ctas_per_sm(size_t smem, int& n);

constexpr int kMaxBatch = 40;  // requests per persistent launch

}  // namespace ustb

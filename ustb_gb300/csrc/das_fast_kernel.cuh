// Fast delay-and-sum: reduced-precision channel storage, geometry formed on the
// fly, factored phase, sample windows staged in shared memory.
//
// Same formula as the reference's das_c (+mex/source/das_c.cpp:355-409), with
// the tables das.m builds in MATLAB (+midprocess/das.m:91-209) computed per
// pixel-channel and pixel-wave in registers:
//
//   y = sum_w sum_n  A_w(p) * B_n(p) * lerp(x_{n,w}, s_tx(p,w) + s_rx(p,n))
//   A_w = apo_tx * exp(i 2 pi fd tau_tx),  B_n = apo_rx * exp(i 2 pi fd tau_rx)
//
// One CTA of 256 threads beamforms half of a 512-pixel tile (one pixel per thread) for
// one frame; two CTAs share an SM, so that one computes while the other waits at a stage
// barrier or sets a tile up.  (Tables of about 1180 channels or more leave room for one: then
// a CTA of 512 threads may take the whole tile, see subs_for in das_fast.cu.)  The (channel, wave) pairs are processed in stages of 32
// slots; for each pair the CTA needs a short window of samples whose start and length
// follow from bounding boxes: the delay bases base_n / base_w are integer lower bounds of
// the whole tile's receive / transmit delays (in samples), the windows cover the CTA's
// half of it.
//
// A pre-pass (build_entries_kernel) rewrites the channel data, whatever its
// storage type, as FP32 interpolation entries {x_i, x_{i+1} - x_i} with das_c's
// validity rule (0 < i < L-1) folded in as zero entries; complex 16-bit data keeps pairs
// {x_i, x_{i+1}} as stored (entries_for in das_fast.cu).  A stage's windows are then plain
// runs of 16-byte (complex FP32) or 8-byte entries that the CTA
// copies with cp.async into one of two shared-memory buffers while it computes
// the stage before; no per-sample work is left in the staging.  A unit costs:
//   s = s_tx_loc + s_rx_loc; j = floor(s); b = s - j; e = slot[j];
//   v = e.x + b*e.d;  acc += weight * v,
// in packed FP32 pairs: two units share their position, fraction and accumulation
// instructions.  Delays relative to the tile bases stay below 80 samples, so j and b
// keep full sub-sample precision in FP32.
//
// What bounds it (75-wave IQ compounding, 400 x 400 pixels, 0.49 ms a launch on a GB300;
// 0.594 ms with one 512-thread CTA per SM and scalar units): the units' 16-byte
// shared-memory loads alone take 0.24 ms; the stages' copies, barriers and transmit
// set-ups overlap them only in part.  Measured with parts taken out of a copy: no
// barriers 0.43 ms, no copies 0.42 ms, no units 0.32 ms.  Not kept, same workload: TMA
// bulk copies of the windows (0.60 ms: about 50 clocks a copy), three 80-register CTAs
// per SM with 16-slot stages (0.58 ms), two pixels per thread (0.59 ms: spills).
// A small launch is bound by setting tiles up, 15,000 clocks of dependent loads and long
// arithmetic before the first stage (a stage takes about 3,500): the loads are issued
// together at the start, channels and waves go to different warps, the stage buffers are
// zeroed meanwhile (32 channels x 1 wave on 135 x 96 pixels: 30 to 26 us a call, with the
// launch that overlaps the pre-pass's end).
//
// Loop orders: waves outer / channels inner for dimension.both and .receive
// (rx weight per unit, tx weight once per wave chunk); channels outer / waves
// inner for .transmit and .none (tx weight per unit).
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "das_fast.cuh"
#include "f32x2.cuh"
#include "phasor.cuh"

namespace ustb {
namespace {

// Sub-tiles (CTAs) per tile, set by the including file: 2, or 1 for requests whose tables
// leave no room for two CTAs on an SM.
#ifndef USTB_SUBS
#define USTB_SUBS 2
#endif
constexpr int kSub = USTB_SUBS;
constexpr int kThreads = kTile / kSub;          // a CTA takes one sub-tile, one pixel per thread
constexpr int kItemFrames = 8;                  // frames of a persistent work item at most
constexpr float kHalf = 79.f;                   // max relative delay of each component (160-entry slots)
constexpr float kMagic = 8388608.0f;            // 2^23: floor via round-toward-zero add
constexpr int kMagicBits = 0x4B000000;

// ---------------------------------------------------------------------------
// apodization windows, +uff/apodization.m:172-223 (0 beyond ratio 1/2)
//
// Every window has the form
//   w(r) = 1                                  for r <= r1
//        = a + e*r + b*cos(c*(r - d))          for r1 < r <= 1/2
//        = 0                                   beyond
// with per-window constants (window_coeffs() in das_fast.cu), so the kernel evaluates it without
// branching on the window type:
//   boxcar    r1 = 1/2
//   hanning   r1 = -1, a = b = 1/2, c = 2*pi, d = 0
//   hamming   r1 = -1, a = 0.53836, b = 0.46164, c = 2*pi, d = 0
//   tukey(R)  r1 = (1-R)/2, a = b = 1/2, c = 2*pi/R, d = R/2 + 1/2
//   triangle  r1 = -1, a = 1, e = -2
// (Tukey's strict r < 1/2 edge gives the same value, 0, at r = 1/2.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float window(const Params& A, float r) {
    const float taper = fmaf(A.win_e, r, A.win_a) + A.win_b * __cosf(A.win_c * (r - A.win_d));
    const float w = r <= 0.5f ? taper : 0.f;
    return r <= A.win_r1 ? 1.f : w;  // NaN ratios (0/0) give 0
}

__device__ __forceinline__ float msign(float v) { return (float)((v > 0.f) - (v < 0.f)); }

// min/max aperture clamps of apodization.m:452-462 (MATLAB sign(0) = 0)
__device__ __forceinline__ float clamp_ap(float z, float fnum, float minap, float maxap) {
    const float a = fminf(fmaxf(fabsf(z), minap * fnum), maxap * fnum);
    return copysignf(a, z) * (z != 0.f ? 1.f : 0.f);
}

__device__ __forceinline__ float rx_apodization(const Params& A, float ex, float ey, float ez, float px,
                                                float py, float pz) {
    if (A.rx_window == USTB_WIN_NONE) return 1.f;
    float xd, yd, zd;
    if (A.rx_origin) {
        xd = ex - A.ox;
        yd = ey - A.oy;
        const float qx = px - A.ox, qy = py - A.oy, qz = pz - A.oz;
        zd = sqrtf(qx * qx + qy * qy + qz * qz);
    } else {
        xd = px - ex;
        yd = py - ey;
        zd = pz - ez;
    }
    const float zx = clamp_ap(zd, A.fnx, A.minx, A.maxx);
    const float rt = fabsf(A.fnx * __fdividef(xd, zx));
    const float wx = window(A, rt);
    if (yd == 0.f) return wx;  // elevation ratio 0: every window is 1 there
    const float zy = clamp_ap(zd, A.fny, A.miny, A.maxy);
    const float rp = fabsf(A.fny * __fdividef(yd, zy));
    return wx * window(A, rp);
}

// exp(i 2 pi fd tau) from the phase in cycles
__device__ __forceinline__ float2 phasor_cycles(float cyc) {
    const float k = rintf(cyc);
    const float fr = cyc - k;  // exact for |cyc| < 2^22
    float s, c;
    __sincosf(6.283185307179586f * fr, &s, &c);
    return make_float2(c, s);
}

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ void dist_range(const Box& b, float x, float y, float z, float& dmin, float& dmax) {
    const float q[3] = {x, y, z};
    float n2 = 0.f, f2 = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float dl = b.lo[i] - q[i], dh = q[i] - b.hi[i];
        const float dn = fmaxf(0.f, fmaxf(dl, dh));
        const float df = fmaxf(fabsf(q[i] - b.lo[i]), fabsf(q[i] - b.hi[i]));
        n2 += dn * dn;
        f2 += df * df;
    }
    dmin = sqrtf(n2);
    dmax = sqrtf(f2);
}

// lower / upper bound of a wave's transmit delay (s) over the tile box
__device__ __forceinline__ void tx_tau_range(const ustb_wave& wv, const Box& b, float& lo, float& hi) {
    switch (wv.kind) {
        case USTB_WAVE_PLANE: {
            float mn = 0.f, mx = 0.f;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float u = wv.dir[i] * b.lo[i], v = wv.dir[i] * b.hi[i];
                mn += fminf(u, v);
                mx += fmaxf(u, v);
            }
            lo = mn / wv.sound_speed - wv.delay;
            hi = mx / wv.sound_speed - wv.delay;
            return;
        }
        case USTB_WAVE_SPHERICAL: {
            float dmin, dmax;
            dist_range(b, wv.src[0], wv.src[1], wv.src[2], dmin, dmax);
            float vlo, vhi;
            if (b.lo[2] >= wv.src[2]) { vlo = dmin; vhi = dmax; }
            else if (b.hi[2] < wv.src[2]) { vlo = -dmax; vhi = -dmin; }
            else { vlo = -dmax; vhi = dmax; }
            lo = (vlo + wv.offset) / wv.sound_speed - wv.delay;
            hi = (vhi + wv.offset) / wv.sound_speed - wv.delay;
            return;
        }
        default:
            lo = hi = -wv.delay;
            return;
    }
}

// Block-wide minimum of NV floats per thread (all threads call; results broadcast).
// Floats are compared as integers in an order-preserving form; a maximum is the minimum
// of the negated value.  ``red``: NV words per warp; reused by the next call, which
// starts with a barrier.
__device__ __forceinline__ int float_order(float v) {
    const int i = __float_as_int(v);
    return i ^ ((i >> 31) & 0x7fffffff);
}
template <int NV>
__device__ __forceinline__ void block_min(float (&v)[NV], int* red) {
    static_assert(NV <= 32, "one lane per value");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int mine = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int m = __reduce_min_sync(0xffffffffu, float_order(v[i]));
        if (lane == i) mine = m;
    }
    __syncthreads();
    if (lane < NV) red[warp * NV + lane] = mine;
    __syncthreads();
    if (lane < NV) {
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) mine = min(mine, red[w * NV + lane]);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int m = __shfl_sync(0xffffffffu, mine, i);
        v[i] = __int_as_float(m ^ ((m >> 31) & 0x7fffffff));
    }
}

// {x_i, x_{i+1} - x_i} in FP32, or {x_i, x_{i+1}} as stored, whose difference the unit forms
template <int ENT>
struct EntryT { using type = uint2; };
template <>
struct EntryT<kEntReal> { using type = float2; };
template <>
struct EntryT<kEntComplex> { using type = float4; };

// a stored 16-bit pair in FP32 (exact)
template <int ENT>
__device__ __forceinline__ float2 unpack16(unsigned v) {
    if constexpr (ENT == kEntHalf) {
        __half2 h;
        memcpy(&h, &v, 4);
        return __half22float2(h);
    } else {
        return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
}

// a stored pair less x, in FP32 roundings: mixed-precision subtractions, without the two
// conversions of the pair (matrix volume in FP16 7.64 -> 7.22 ms)
template <int ENT>
__device__ __forceinline__ float2 minus16(unsigned v, float2 x) {
    float2 d;
    if constexpr (ENT == kEntHalf)
        asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nsub.rn.f32.f16 %0, lo, %3;\nsub.rn.f32.f16 %1, hi, %4;\n}\n"
            : "=f"(d.x), "=f"(d.y) : "r"(v), "f"(x.x), "f"(x.y));
    else
        asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nsub.rn.f32.bf16 %0, lo, %3;\nsub.rn.f32.bf16 %1, hi, %4;\n}\n"
            : "=f"(d.x), "=f"(d.y) : "r"(v), "f"(x.x), "f"(x.y));
    return d;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ---- asynchronous global -> shared copies (cp.async, 16 or 8 bytes per thread) -----
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
// The grid may start while the kernel before it in the stream (the entries pre-pass) ends
// (see launch_dependent): nothing of that kernel is read, and no output written, before
// this returns.  Every CTA calls it, also one without work.
__device__ __forceinline__ void wait_for_entries() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Conservative test that channel `n`'s receive window is zero over the whole tile
// box: every window is 0 for ratio > 1/2 (apodization.m:172-186), and the ratio
// F#*|x_dist|/|z| is bounded below by the box.
__device__ __forceinline__ bool rx_active(const Params& A, const Box& b, float ex, float ey, float ez) {
    if (A.rx_apo_tab || A.rx_window == USTB_WIN_NONE) return true;
    float xd, yd, zmax;
    if (A.rx_origin) {
        xd = fabsf(ex - A.ox);
        yd = fabsf(ey - A.oy);
        float dmin, dmax;
        dist_range(b, A.ox, A.oy, A.oz, dmin, dmax);
        zmax = dmax;
    } else {
        xd = fmaxf(0.f, fmaxf(b.lo[0] - ex, ex - b.hi[0]));
        yd = fmaxf(0.f, fmaxf(b.lo[1] - ey, ey - b.hi[1]));
        zmax = fmaxf(fabsf(b.lo[2] - ez), fabsf(b.hi[2] - ez));
    }
    const float zx = fminf(fmaxf(zmax, A.minx * A.fnx), A.maxx * A.fnx);
    const float zy = fminf(fmaxf(zmax, A.miny * A.fny), A.maxy * A.fny);
    if (!(zx > 0.f) || !(zy > 0.f)) return true;
    const float lim = 0.5f * (1.f + 1e-4f);
    return !(A.fnx * xd / zx > lim || A.fny * yd / zy > lim);
}

template <int SHAPE>
struct Shape {
    static constexpr bool WAVES_OUTER = kShapes[SHAPE].waves_outer;
    static constexpr int CG = kShapes[SHAPE].cg, KW = kShapes[SHAPE].kw;
};
template <int SHAPE, bool BIG, bool WIDE>
struct Stage {
    static constexpr int CG = (WIDE && Shape<SHAPE>::WAVES_OUTER) ? Shape<SHAPE>::CG / 2 : Shape<SHAPE>::CG;
    static constexpr int KW = (WIDE && !Shape<SHAPE>::WAVES_OUTER) ? Shape<SHAPE>::KW / 2 : Shape<SHAPE>::KW;
    static constexpr int SLOT = (WIDE || !BIG) ? 160 : 80;  // entries per (channel, wave) window
    static_assert(CG * KW * SLOT * (BIG ? 16 : 8) == kBufBytes, "a stage fills one buffer");
};

// Once per CTA: zero the stage buffers, so that units whose sums nothing takes (idle lanes,
// inactive channels), which may read past a window's end, never read uninitialised words.
// The caller's barriers follow.
__device__ __forceinline__ void zero_slots() {
    extern __shared__ __align__(16) unsigned char smem[];
    float4* z = reinterpret_cast<float4*>(smem);
    for (int i = threadIdx.x; i < (int)(kBuffers / 16); i += kThreads) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float frac_cycles(double v) { return (float)(v - floor(v)); }

// Beamform one sub-tile of one frame (the whole CTA participates).
//
// Delays are kept relative to integer delay bases of the whole tile: for pixel p,
//   s_tx(p, w) = (tau_tx - t0) fs - base_w,   s_rx(p, n) = tau_rx fs - base_n,
// both in [0, kHalf], and the unit's sample position is base_n + base_w + s_tx + s_rx.
// The phase factors exp(i 2 pi fd tau) are formed from these relative delays and a
// per-tile offset of each base (computed in double):
//   fd tau_tx = (fd/fs) s_tx + frac(fd (base_w/fs + t0)),  fd tau_rx = (fd/fs) s_rx + frac(fd base_n / fs).
// A plane or photoacoustic wave's s_tx is affine in the pixel position and a
// spherical wave's is sigma |p - src| fs/c + const; the per-tile coefficients
// sit in shared memory (txc, txp).
//
// The windows cover the CTA's sub-tile only: window (n, w) starts j_n + j_w samples
// after base_n + base_w, with j the floor of the sub-tile's own lower delay bound, and a
// unit reads its slot at (s_tx - j_w) + (s_rx - j_n) (the subtractions are exact).
//
// FRAMES (persistent kernel): frames f_first .. f_first + nfr - 1 of the tile in turn,
// after one build of the tile's tables and stage lists (the geometry is the same for
// every frame of a request).
template <int MODE, int ENT, bool EPI, int SHAPE, bool FRAMES = false>
__device__ __forceinline__ void das_tile(const Params& A, int tile, int sub, int64_t f_first, int part = -1,
                                         int nfr = 1, bool first = true) {
    constexpr bool ORDER_A = Shape<SHAPE>::WAVES_OUTER;
    static_assert(MODE != USTB_DIM_RECEIVE || ORDER_A, "dimension.receive keeps waves outer");
    static_assert((MODE != USTB_DIM_TRANSMIT && MODE != USTB_DIM_NONE) || !ORDER_A,
                  "dimension.transmit / none keep channels outer");
    constexpr bool CPLX = ENT != kEntReal, BIG = ENT == kEntComplex;
    using Entry = typename EntryT<ENT>::type;
    constexpr int ES = (int)sizeof(Entry);

    const int64_t N = A.N, W = A.W, P = A.P;
    extern __shared__ __align__(16) unsigned char smem[];
    Entry* slots = reinterpret_cast<Entry*>(smem);
    constexpr int CGM = Shape<SHAPE>::CG, KWM = Shape<SHAPE>::KW;
    const int NP = ((int)N + CGM - 1) / CGM * CGM, WP = ((int)W + KWM - 1) / KWM * KWM;
    const TileTables tt = tile_tables(kShapes[SHAPE], NP, WP);
    unsigned char* tb = smem + kBuffers;
    float4* el4 = reinterpret_cast<float4*>(tb + tt.el4);
    float4* txc = reinterpret_cast<float4*>(tb + tt.txc);
    float4* txp = reinterpret_cast<float4*>(tb + tt.txp);
    int2* win_w = reinterpret_cast<int2*>(tb + tt.win_w);
    float2* rxp = reinterpret_cast<float2*>(tb + tt.rxp);
    float* base_w = reinterpret_cast<float*>(tb + tt.base_w);
    uint16_t* olist = reinterpret_cast<uint16_t*>(tb + tt.olist);
    float* len_n = reinterpret_cast<float*>(tb + tt.len_n);
    unsigned char* kind_w = tb + tt.kind_w;
    __shared__ int s_red[kThreads / 32 * 12];
    __shared__ int s_tx_general;  // a spherical or tabulated wave, or tabulated tx apodization
    __shared__ int s_tx_sph;      // every active wave spherical, and no tx tables
    __shared__ int s_maxn, s_maxw;  // largest active window positions (bits of floats >= 0)
    __shared__ int s_nout, s_nin;
    __shared__ int s_where[3];      // tile, sub-tile, part: read again after the stages (fewer live registers)
    __shared__ bool s_last;             // this part is the last of its sub-tile to finish
    __shared__ int s_flat, s_in_plane;  // every element at one z; no elevation offset in the tile

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int32_t* tl = A.tiles + (int64_t)tile * kTile;
    // Setting a tile up is a chain of dependent loads and long-latency arithmetic: what the
    // tables below read is loaded first, beside the pixel indices and positions, channels
    // by the first threads and waves by the last ones, so that different warps work on both.
    const int wtid = kThreads - 1 - tid;
    float3 next_el = make_float3(0.f, 0.f, 0.f);
    ustb_wave next_wv = {};
    auto load_el = [&](int n) {
        if (n < (int)N) next_el = make_float3(__ldg(A.el + 3 * n), __ldg(A.el + 3 * n + 1), __ldg(A.el + 3 * n + 2));
    };
    auto load_wave = [&](int w) {
        if (w < (int)W) next_wv = A.waves[w];
    };
    load_el(tid);
    load_wave(wtid);
    const float el0_z = N > 0 ? __ldg(A.el + 2) : 0.f;
    // tile entries outside [0, P) are idle lanes; lane 0 names the tile's anchor pixel
    auto in_image = [&](int32_t q) { return q >= 0 && (int64_t)q < A.P; };
    const int32_t p_own = __ldg(tl + sub * kThreads + tid);
    const int32_t p_anchor = __ldg(tl);
    // this thread's pixel of the other sub-tile: the delay bases are the whole tile's
    static_assert(kSub <= 2, "one other sub-tile");
    const int32_t p_other = kSub == 2 ? __ldg(tl + (sub ^ 1) * kThreads + tid) : -1;
    const bool live = in_image(p_own), live_o = in_image(p_other);
    if (tid == 0) {
        s_tx_general = A.tx_apo_tab != nullptr || A.tx_delay_tab != nullptr;
        s_tx_sph = !s_tx_general;
        s_maxn = s_maxw = 0;
        s_flat = 1;
        s_in_plane = 1;
        s_where[0] = tile;
        s_where[1] = sub;
        s_where[2] = part;
    }
    if (first) zero_slots();
    if (!__syncthreads_or(live)) {  // an idle sub-tile
        wait_for_entries();
        return;
    }
    const int p = live ? p_own : (in_image(p_anchor) ? p_anchor : 0);
    const float* const pxyz = A.px + 3 * (int64_t)p;
    const float px = __ldg(pxyz), py = __ldg(pxyz + 1), pz = __ldg(pxyz + 2);
    if (live && py != py) s_in_plane = 0;  // the box does not hold it: its window is 0, not 1

    Box box, tbox;  // sub-tile, whole tile
    {
        const float big = 3.4e38f;
        const int64_t po = live_o ? p_other : p;
        const float own[3] = {px, py, pz};
        float v[12];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float a = own[i], b = __ldg(A.px + 3 * po + i);
            const bool ua = live && a == a, ub = live_o && b == b;  // NaN coordinates bound nothing
            v[i] = ua ? a : big;
            v[3 + i] = ua ? -a : big;
            v[6 + i] = fminf(v[i], ub ? b : big);
            v[9 + i] = fminf(v[3 + i], ub ? -b : big);
        }
        block_min(v, s_red);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            box.lo[i] = v[i]; box.hi[i] = -v[3 + i];
            tbox.lo[i] = v[6 + i]; tbox.hi[i] = -v[9 + i];
        }
    }

    // ---- per-tile delay bases, window parts, activity and delay/phase coefficients ----
    const double fd_fs = A.fd_fs;
    // Padding waves have no window.  The units of a wave without a weight are evaluated, so
    // it has one that lies before every trace and zeros are stored for it: what an earlier
    // stage left in its slots may not be finite.  Either length has its sign bit set.
    const int2 inactive = make_int2(0, __float_as_int(-1e9f)), zeros = make_int2(-(1 << 30), __float_as_int(-0.f));
    auto act_n = [&](int n) { return len_n[n] >= 0.f; };
    auto act_w = [&](int w) { return win_w[w].y >= 0; };  // the sign bit
    // sub-tile delays [lo, hi] -> window start j after `base` and largest position after
    // that, both in [0, kHalf]; the margin covers the rounding of the bounds
    auto window_part = [&](float base, float lo, float hi, float& j, float& len) {
        constexpr float kMargin = 0.0625f;
        j = fminf(fmaxf(floorf(lo - kMargin) - base, 0.f), kHalf);
        len = fminf(fmaxf(hi + kMargin - base - j, 0.f), kHalf);
    };
    auto pack_part = [&](float base, float j, float len) { return make_int2((int)base + (int)j, __float_as_int(len)); };
    // the largest window position of a warp's channels or waves into m
    auto longest = [&](int& m, float len) {
        const int v = __reduce_max_sync(0xffffffffu, __float_as_int(len));
        if (lane == 0 && v > 0) atomicMax(&m, v);
    };
    float longest_n = 0.f, longest_w = 0.f;
    for (int n = tid; n < NP; n += kThreads) {
        const float ex = next_el.x, ey = next_el.y, ez = next_el.z;
        load_el(n + kThreads);
        if (n >= (int)N) {  // padding channels: never active
            el4[n] = make_float4(0.f, 0.f, 0.f, 0.f);
            rxp[n] = make_float2(0.f, 0.f);
            len_n[n] = -1e9f;
            continue;
        }
        float dmin, dmax;
        dist_range(tbox, ex, ey, ez, dmin, dmax);
        float lo = (dmin * A.inv_c + A.lens) * A.fs, hi = (dmax * A.inv_c + A.lens) * A.fs;
        const float fbase = floorf(lo) - 1.f;
        const bool ok = (hi - fbase <= kHalf - 2.f) && fabsf(fbase) < 1.0e9f;
        if (!ok && rx_active(A, tbox, ex, ey, ez)) atomicOr(A.flags, USTB_FLAG_WINDOW_OVERFLOW);
        const float base = fminf(fmaxf(fbase, -1.0e9f), 1.0e9f);
        dist_range(box, ex, ey, ez, dmin, dmax);
        lo = (dmin * A.inv_c + A.lens) * A.fs;
        hi = (dmax * A.inv_c + A.lens) * A.fs;
        float j, len;
        window_part(base, lo, hi, j, len);
        const bool act = rx_active(A, box, ex, ey, ez);
        if (ez != el0_z) s_flat = 0;
        if (A.rx_origin ? ey != A.oy : (box.lo[1] != ey || box.hi[1] != ey)) s_in_plane = 0;
        el4[n] = make_float4(ex, ey, ez, base);
        rxp[n] = make_float2(frac_cycles(fd_fs * (double)base), j);
        len_n[n] = act ? len : -1e9f;
        if (act) longest_n = fmaxf(longest_n, len);
    }
    for (int w = wtid; w < WP; w += kThreads) {
        const ustb_wave wv = next_wv;
        load_wave(w + kThreads);
        if (w >= (int)W) {  // padding waves: zero weight
            txc[w] = make_float4(0.f, 0.f, 0.f, 0.f);
            txp[w] = make_float4(0.f, 0.f, 0.f, 0.f);
            base_w[w] = 0.f;
            kind_w[w] = USTB_WAVE_ZERO;
            win_w[w] = inactive;
            continue;
        }
        // a table wave without a table has the constant delay -delay
        const bool table = wv.kind == USTB_WAVE_TABLE;
        kind_w[w] = (unsigned char)(table && !A.tx_delay_tab ? USTB_WAVE_ZERO : wv.kind);
        if (table && A.tx_delay_tab) continue;  // bases from the table below
        float lo, hi;
        tx_tau_range(wv, tbox, lo, hi);
        lo = (lo - A.t0) * A.fs;
        hi = (hi - A.t0) * A.fs;
        const float fbase = floorf(lo) - 1.f;
        const bool ok = (hi - fbase <= kHalf - 2.f) && fabsf(fbase) < 1.0e9f;
        const bool act = A.tx_apo_tab != nullptr || wv.apodization != 0.f;
        if (!ok && act && !table) atomicOr(A.flags, USTB_FLAG_WINDOW_OVERFLOW);
        if (wv.kind == USTB_WAVE_SPHERICAL && act) s_tx_general = 1;
        if (wv.kind != USTB_WAVE_SPHERICAL && act && !table) s_tx_sph = 0;
        const float bw = fminf(fmaxf(fbase, -1.0e9f), 1.0e9f);
        base_w[w] = bw;
        tx_tau_range(wv, box, lo, hi);
        lo = (lo - A.t0) * A.fs;
        hi = (hi - A.t0) * A.fs;
        float j, len;
        window_part(bw, lo, hi, j, len);
        win_w[w] = act ? pack_part(bw, j, len) : zeros;
        if (!act) {  // at position 0 of the window of zeros
            txc[w] = txp[w] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        longest_w = fmaxf(longest_w, len);
        // s_tx(p) = (tau(p) - t0) fs - base_w; constant part in double
        const double fs_c = wv.sound_speed == A.c ? A.fs_c : (double)A.fs / (double)wv.sound_speed;
        const double c0 = -((double)wv.delay + (double)A.t0) * (double)A.fs - (double)bw;
        if (wv.kind == USTB_WAVE_PLANE)
            txc[w] = make_float4((float)(wv.dir[0] * fs_c), (float)(wv.dir[1] * fs_c), (float)(wv.dir[2] * fs_c),
                                 (float)c0);
        else if (wv.kind == USTB_WAVE_SPHERICAL)
            txc[w] = make_float4(wv.src[0], wv.src[1], wv.src[2], (float)(c0 + (double)wv.offset * fs_c));
        else
            txc[w] = make_float4(0.f, 0.f, 0.f, (float)c0);
        txp[w] = make_float4(frac_cycles(fd_fs * ((double)bw + (double)A.t0 * (double)A.fs)), wv.apodization,
                             table ? 0.f : (float)fs_c, j);
    }
    longest(s_maxn, longest_n);
    longest(s_maxw, longest_w);
    if (A.tx_delay_tab) {  // tabulated transmit delays: the tile's actual range
        for (int64_t w = 0; w < W; ++w) {
            const ustb_wave wv = A.waves[w];
            if (wv.kind != USTB_WAVE_TABLE) continue;
            const float* tab = A.tx_delay_tab + w * P;
            const float big = 3.4e38f;
            const float s = (__ldg(tab + p) - A.t0) * A.fs;
            const float so = live_o ? (__ldg(tab + p_other) - A.t0) * A.fs : big;
            const bool us = live && s == s, uo = live_o && so == so;
            float v[4];
            v[0] = us ? s : big;
            v[1] = us ? -s : big;
            v[2] = fminf(v[0], uo ? so : big);
            v[3] = fminf(v[1], uo ? -so : big);
            block_min(v, s_red);
            if (tid == 0) {
                const float fbase = floorf(v[2]) - 1.f;
                const bool ok = (-v[3] - fbase <= kHalf - 2.f) && fabsf(fbase) < 1.0e9f;
                if (!ok) atomicOr(A.flags, USTB_FLAG_WINDOW_OVERFLOW);
                const float bw = fminf(fmaxf(fbase, -1.0e9f), 1.0e9f);
                base_w[w] = bw;
                float j, len;
                window_part(bw, v[0], -v[1], j, len);
                win_w[w] = pack_part(bw, j, len);
                atomicMax(&s_maxw, __float_as_int(len));
                txc[w] = make_float4(0.f, 0.f, 0.f, 0.f);
                txp[w] = make_float4(frac_cycles(fd_fs * ((double)bw + (double)A.t0 * (double)A.fs)),
                                     wv.apodization, 0.f, j);
            }
        }
    }
    __syncthreads();

    // Complex data: narrow slots (80 entries) when every window fits one; the clamps keep
    // any unit inside its slot: receive parts in [0, hn], transmit parts in [0, hw],
    // hn + hw + 1 at most the entries per slot.
    const float maxn = __int_as_float(s_maxn), maxw = __int_as_float(s_maxw);
    constexpr float kNarrowEnd = (float)Stage<SHAPE, BIG, false>::SLOT - 1.125f;
    const bool narrow = BIG && maxn + maxw <= kNarrowEnd;
    const float hn = narrow ? maxn : kHalf, hw = narrow ? kNarrowEnd - maxn : kHalf;

    // The stages are every (active outer, active inner) pair of channel groups and wave
    // chunks in loop order: warp 0 compacts the active outer indices, warp 1 the inner
    // ones (ballots).
    auto build_lists = [&](auto stage) {
        using ST = decltype(stage);
        const int NG = NP / ST::CG, NC = WP / ST::KW;
        const int NO = ORDER_A ? NC : NG, NI = ORDER_A ? NG : NC;
        if (warp < 2) {
            const bool chan = (warp == 0) != ORDER_A;  // this warp compacts channel groups
            const int cnt = warp == 0 ? NO : NI, per = chan ? ST::CG : ST::KW;
            uint16_t* list = warp == 0 ? olist : olist + NO;
            int got = 0;
            for (int b = 0; b < cnt; b += 32) {
                bool a = false;
                if (b + lane < cnt)
                    for (int c = 0; c < per; ++c) a |= chan ? act_n((b + lane) * per + c) : act_w((b + lane) * per + c);
                const unsigned m = __ballot_sync(0xffffffffu, a);
                if (a) list[got + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(b + lane);
                got += __popc(m);
            }
            if (lane == 0) (warp == 0 ? s_nout : s_nin) = got;
        }
        __syncthreads();
    };

    // frames f0 .. f0 + nf - 1: outer index, then frames, then inner index, so that the
    // outer geometry is formed once for all of them
    auto run = [&](auto stage, const int64_t f0, const int nf) {
    using ST = decltype(stage);
    constexpr int CG = ST::CG, KW = ST::KW, SLOT = ST::SLOT, NS = CG * KW;  // NS slots per stage
    const float2 ph = MODE != USTB_DIM_BOTH && A.pix_phase ? __ldg(A.pix_phase + p) : make_float2(1.f, 0.f);
    const float fdfs = (float)fd_fs;
    const int Lc = (int)A.L;             // entries per trace
    const uint32_t slots_s = (uint32_t)__cvta_generic_to_shared(slots);
    const int NG = NP / CG, NC = WP / KW;
    const uint16_t* ilist = olist + (ORDER_A ? NC : NG);
    const int no = s_nout, ni = s_nin, nstages = no * ni * nf;

    // A stage's windows into buffer `buf`, for channel group / wave chunk at n0 / w0.
    // LPS lanes copy one slot's window [i0, i0 + len) entry by entry with cp.async; the
    // entries outside the trace, in windows that cross one of its ends, are stored as
    // zeros.  i0 and len come from the per-tile {start, length} of the slot's channel and
    // wave.  A thread always serves the same slot (c, k), so what depends on the outer
    // index is formed when it changes.  Slots of inactive channels and of padding are left
    // as they are: nothing that is stored has read them.
    constexpr int NWARPS = kThreads / 32, PER = NS / NWARPS, LPS = 32 / PER;  // slots per warp, lanes per slot
    const int my_sl = warp * PER + lane / LPS, my_c = my_sl / KW, my_k = my_sl - my_c * KW, hl = lane % LPS;
    const Entry* const ent_f = reinterpret_cast<const Entry*>(A.entries) + f0 * A.frame_step;
    const uint32_t my_dst = slots_s + (uint32_t)(my_sl * SLOT + hl) * ES;
    int part_start = 0;                       // the outer index's part of my slot's window
    float part_len = 0.f;                     // (-1e9: no work)
    const Entry* part_src = ent_f;            // entry 0 of the channel's first wave (waves outer: of channel 0's wave)
    auto chan_part = [&](int n, int& start, float& len, const Entry*& src) {
        len = len_n[n];
        start = (int)el4[n].w + (int)rxp[n].y;
        src += (int64_t)n * A.Lp;
    };
    auto wave_part = [&](int w, int& start, float& len, const Entry*& src) {
        const int2 b = win_w[w];
        start = b.x;
        len = __int_as_float(b.y);
        src += w * A.wave_step;
    };
    auto issue_outer = [&](int n0, int w0) {
        part_src = ent_f;
        if (ORDER_A) wave_part(w0 + my_k, part_start, part_len, part_src);
        else chan_part(n0 + my_c, part_start, part_len, part_src);
    };
    // Where my slot's window of a stage lies; located ahead of the stage barrier, so that
    // only the copies follow it.
    const Entry* win_src = ent_f;  // my first entry
    int win_len = 0, win_i0 = 0;   // entries from my first one on (<= 0: none), its index in the trace
    auto locate = [&](int n0, int w0, int fr) {
        int start;
        float ln;
        const Entry* src = part_src;
        if (FRAMES) src += fr * A.frame_step;
        if (ORDER_A) chan_part(n0 + my_c, start, ln, src);
        else wave_part(w0 + my_k, start, ln, src);
        // entries 0 .. floor(largest position), and one for the rounding of the units' sums
        win_len = min(SLOT, (int)(part_len + ln) + 2) - hl;
        win_i0 = part_start + start + hl;
        win_src = src + win_i0;
    };
    auto issue = [&](int buf) {
        const uint32_t dst = my_dst + (uint32_t)(buf * kBufBytes);
        if (win_i0 >= hl && win_i0 + win_len <= Lc) {
#pragma unroll
            for (int j = 0; j < SLOT; j += LPS) {
                if (j >= win_len) break;
                cp_async<ES>(dst + (uint32_t)(j * ES), win_src + j);
            }
        } else {
            for (int j = 0; j < win_len; j += LPS) {
                if ((unsigned)(win_i0 + j) < (unsigned)Lc) {
                    cp_async<ES>(dst + (uint32_t)(j * ES), win_src + j);
                } else {
                    if constexpr (BIG)
                        asm volatile("st.shared.v4.f32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst + (uint32_t)(j * ES)), "f"(0.f) : "memory");
                    else
                        asm volatile("st.shared.v2.f32 [%0], {%1, %1};\n" ::"r"(dst + (uint32_t)(j * ES)), "f"(0.f) : "memory");
                }
            }
        }
    };

    // per-thread geometry
    float srx[CG];
    float2 B[CG];
    float stx[KW];
    float2 Aw[KW];
    // partial sums per wave (waves outer) or channel, in pairs
    constexpr int NACC = ORDER_A ? KW : CG;
    static_assert(NACC % 2 == 0, "partial sums are kept in pairs");
    f32x2 accr[NACC / 2], acci[NACC / 2];
    auto sum_of = [&](int i) {
        const float2 re = unpack2(accr[i / 2]), im = unpack2(acci[i / 2]);
        return (i & 1) ? make_float2(re.y, im.y) : make_float2(re.x, im.x);
    };
    float2 Y[FRAMES ? kItemFrames : 1];  // dimension.both: the pixel's sum of each frame
    for (int i = 0; i < (FRAMES ? nf : 1); ++i) Y[i] = make_float2(0.f, 0.f);
    float2 eS = make_float2(0.f, 0.f);
    float eI = 0.f, eM = 0.f, eR = 0.f, eQ = 0.f;

    // a channel's receive part: its place in the slot and its weight (times the phasor)
    auto put_rx = [&](int c, int n, float s, float2 rp, float apo) {
        if (CPLX) {
            const float2 e = phasor_cycles(fmaf(s, fdfs, rp.x));
            B[c] = make_float2(apo * e.x, apo * e.y);
        } else {
            B[c] = make_float2(apo, 0.f);
        }
        srx[c] = fminf(fmaxf(s - rp.y, 0.f), hn);  // NaN -> 0: stays inside the slot
        if constexpr (EPI) eM += (n < (int)N && apo > A.cf_thr) ? 1.f : 0.f;  // (weight 0 counts below a negative threshold)
    };
    // Closed-form window (no table): the same arithmetic as rx_apodization without its
    // per-channel branches; padding channels are inactive, so their weight is 0.
    const bool rx_plain = !A.rx_apo_tab && A.rx_window != USTB_WIN_NONE;
    // The distance the aperture is measured at is one per pixel for sector scans and for
    // flat probes (every element at one z): its clamped reciprocals are formed once, in the
    // roundings of __fdividef(x, z) = x * rcp(z).
    const bool rx_flat = rx_plain && (A.rx_origin || s_flat);
    const bool rx_in_plane = s_in_plane != 0;  // no elevation offsets: every window is 1 there
    float rcx = 0.f, rcy = 0.f;
    if (rx_flat) {
        float zd = pz - el4[0].z;
        if (A.rx_origin) {
            const float qx = px - A.ox, qy = py - A.oy, qz = pz - A.oz;
            zd = sqrtf(qx * qx + qy * qy + qz * qz);
        }
        rcx = __fdividef(1.f, clamp_ap(zd, A.fnx, A.minx, A.maxx));
        rcy = __fdividef(1.f, clamp_ap(zd, A.fny, A.miny, A.maxy));
    }
    auto setup_rx_flat = [&](int n0) {
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            const int n = n0 + c;
            const float4 e4 = el4[n];
            const float dx = px - e4.x, dy = py - e4.y, dz = pz - e4.z;
            const float r2 = fmaxf(dx * dx + dy * dy + dz * dz, 1e-30f);
            const float r = r2 * rsqrtf(r2);
            const float s = (r * A.inv_c + A.lens) * A.fs - e4.w;
            float apo = window(A, fabsf(A.fnx * ((A.rx_origin ? e4.x - A.ox : -dx) * rcx)));
            if (!rx_in_plane) {
                const float yd = A.rx_origin ? e4.y - A.oy : -dy;
                if (yd != 0.f) apo *= window(A, fabsf(A.fny * (yd * rcy)));
            }
            if (!live || !act_n(n)) apo = 0.f;
            put_rx(c, n, s, rxp[n], apo);
        }
    };
    auto setup_rx = [&](int n0) {
        if (rx_flat) {
            setup_rx_flat(n0);
            return;
        }
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            const int n = n0 + c;
            if (act_n(n)) {
                const float4 e4 = el4[n];
                const float ex = e4.x, ey = e4.y, ez = e4.z;
                const float dx = px - ex, dy = py - ey, dz = pz - ez;
                const float r2 = fmaxf(dx * dx + dy * dy + dz * dz, 1e-30f);
                const float r = r2 * rsqrtf(r2);
                const float s = (r * A.inv_c + A.lens) * A.fs - e4.w;
                float apo = A.rx_apo_tab ? __ldg(A.rx_apo_tab + (int64_t)n * P + p) : rx_apodization(A, ex, ey, ez, px, py, pz);
                if (!live) apo = 0.f;
                put_rx(c, n, s, rxp[n], apo);
            } else {
                srx[c] = 0.f;
                B[c] = make_float2(0.f, 0.f);
                if constexpr (EPI) eM += (n < (int)N && 0.f > A.cf_thr) ? 1.f : 0.f;
            }
        }
    };
    // Plane and photoacoustic waves (every tile without spherical or tabulated waves
    // and without a tx apodization table): s_tx is affine in the pixel position and
    // the weight is the wave's constant apodization times the phasor; padding and
    // inactive waves carry apodization 0.  No branches.
    const bool tx_affine = !s_tx_general;
    // Diverging and focused waves (every active wave spherical, no tables): the same
    // arithmetic as the general setup below without its per-wave branches; padding and
    // inactive waves carry apodization 0, and a table wave without a table has fs/c = 0
    // there, so its s_tx is the constant term as in the general setup.
    const bool tx_sph = s_tx_sph != 0;
    auto put_tx = [&](int k, float s, float4 q, float apo) {
        stx[k] = fminf(fmaxf(s - q.w, 0.f), hw);
        if (CPLX) {
            const float2 e = phasor_cycles(fmaf(s, fdfs, q.x));
            Aw[k] = make_float2(apo * e.x, apo * e.y);
        } else {
            Aw[k] = make_float2(apo, 0.f);
        }
    };
    auto setup_tx = [&](int w0) {
        if (tx_affine) {
#pragma unroll
            for (int k = 0; k < KW; ++k) {
                const float4 cw = txc[w0 + k];
                const float4 q = txp[w0 + k];
                put_tx(k, fmaf(cw.x, px, fmaf(cw.y, py, fmaf(cw.z, pz, cw.w))), q, q.y);
            }
            return;
        }
        if (tx_sph) {
#pragma unroll
            for (int k = 0; k < KW; ++k) {
                const float4 cw = txc[w0 + k];
                const float4 q = txp[w0 + k];
                const float dx = px - cw.x, dy = py - cw.y, dz = pz - cw.z;
                const float d = sqrtf(dx * dx + dy * dy + dz * dz);
                put_tx(k, fmaf(pz < cw.z ? -d : d, q.z, cw.w), q, q.y);
            }
            return;
        }
#pragma unroll
        for (int k = 0; k < KW; ++k) {
            const int w = w0 + k;
            if (act_w(w)) {
                const float4 cw = txc[w];
                const float4 q = txp[w];
                const int kind = kind_w[w];
                float s;
                if (kind == USTB_WAVE_SPHERICAL) {
                    const float dx = px - cw.x, dy = py - cw.y, dz = pz - cw.z;
                    const float d = sqrtf(dx * dx + dy * dy + dz * dz);
                    s = fmaf(pz < cw.z ? -d : d, q.z, cw.w);
                } else if (kind == USTB_WAVE_TABLE) {
                    s = (__ldg(A.tx_delay_tab + w * P + p) - A.t0) * A.fs - base_w[w];
                } else {  // plane; photoacoustic (zero coefficients)
                    s = fmaf(cw.x, px, fmaf(cw.y, py, fmaf(cw.z, pz, cw.w)));
                }
                float apo = A.tx_apo_tab ? __ldg(A.tx_apo_tab + (int64_t)w * P + p) : q.y;
                if (!live) apo = 0.f;
                put_tx(k, s, q, apo);
            } else {
                stx[k] = 0.f;
                Aw[k] = make_float2(0.f, 0.f);
            }
        }
    };

    // shared address of entry 0 of slot 0 in the current stage's buffer, minus the bias of
    // the 2^23 floor trick
    const unsigned slot0 = slots_s - (unsigned)kMagicBits * (unsigned)sizeof(Entry);
    unsigned slot_base = slot0;
    const f32x2 magic2 = pack2(kMagic, kMagic);
    // the entry of slot (c, k) that t = floor(s) + 2^23 names, interpolated at fraction b
    auto interp = [&](int c, int k, float t, float b) -> float2 {
        const unsigned addr = (unsigned)__float_as_int(t) * (unsigned)sizeof(Entry) + slot_base +
                              (unsigned)((c * KW + k) * SLOT * (int)sizeof(Entry));
        if constexpr (ENT == kEntHalf || ENT == kEntBf16) {
            unsigned a, d;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(a), "=r"(d) : "r"(addr));
            const float2 x = unpack16<ENT>(a), df = minus16<ENT>(d, x);
            return make_float2(fmaf(b, df.x, x.x), fmaf(b, df.y, x.y));
        } else if constexpr (CPLX) {
            float4 e;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                         : "=f"(e.x), "=f"(e.y), "=f"(e.z), "=f"(e.w) : "r"(addr));
            return make_float2(fmaf(b, e.z, e.x), fmaf(b, e.w, e.y));
        } else {
            float2 e;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(e.x), "=f"(e.y) : "r"(addr));
            return make_float2(fmaf(b, e.y, e.x), 0.f);
        }
    };
    // Two units at a time, at positions s: slots (c0, k0) and (c1, k1), values added into
    // the pair of sums i with the weights (wx, wy) of both.  Packed arithmetic: per unit
    // 2 instructions for position and fraction, 1 address, 1 load, 2 interpolation and 2
    // to accumulate, in the roundings of the scalar form.
    auto unit_pair = [&](int i, f32x2 s, int c0, int k0, int c1, int k1, f32x2 wx, f32x2 wy, f32x2 nwy) {
        const f32x2 t = add2_rz(s, magic2);
        const float2 b = unpack2(sub2(s, sub2(t, magic2)));
        const float2 tt = unpack2(t);
        const float2 v0 = interp(c0, k0, tt.x, b.x), v1 = interp(c1, k1, tt.y, b.y);
        const f32x2 vx = pack2(v0.x, v1.x);
        if constexpr (CPLX) {
            const f32x2 vy = pack2(v0.y, v1.y);
            accr[i] = fma2(wx, vx, fma2(nwy, vy, accr[i]));
            acci[i] = fma2(wx, vy, fma2(wy, vx, acci[i]));
        } else {
            accr[i] = fma2(wx, vx, accr[i]);
        }
    };

    auto store_cube = [&](int64_t o, float2 y) {
        if (!live || !A.cube) return;
        if constexpr (CPLX) reinterpret_cast<float2*>(A.cube)[o] = y;
        else reinterpret_cast<float*>(A.cube)[o] = y.x;
    };

    // Double-buffered pipeline over the active stages: the next stage's windows are
    // copied while a stage is computed.  One barrier per stage: it makes the stage's
    // entries visible to every warp and frees the other buffer (read by the stage
    // before) for the next stage's copies.
    // part = k >= 0: this CTA takes part k of A.split equal parts of the work; -1: all of it.
    // dimension.both: of the stages, whose partial sums are added (store_both).  transmit
    // and receive: of the outer list (channel groups, wave chunks), whose outputs are
    // disjoint; gaps in the list, inactive and so zero, belong to the part before them.
    const int parts = part < 0 ? 1 : A.split, me = part < 0 ? 0 : part;
    constexpr bool kByOuter = MODE != USTB_DIM_BOTH;
    const int n_split = kByOuter ? no : nstages;
    const int u_lo = (int)((int64_t)n_split * me / parts), u_hi = (int)((int64_t)n_split * (me + 1) / parts);
    const int s_lo = kByOuter ? u_lo * ni * nf : u_lo, s_hi = kByOuter ? u_hi * ni * nf : u_hi;
    const int out_lo = (kByOuter && me > 0) ? (u_lo < no ? olist[u_lo] : (ORDER_A ? NC : NG)) : 0;
    const int out_hi = (kByOuter && me + 1 < parts) ? (u_hi < no ? olist[u_hi] : (ORDER_A ? NC : NG)) : (ORDER_A ? NC : NG);
    // list positions (outer, inner), frame, first channel and first wave of a stage
    struct Pos { int o, i, f, n0, w0; };
    auto place_outer = [&](Pos& q) { (ORDER_A ? q.w0 : q.n0) = olist[q.o] * (ORDER_A ? KW : CG); };
    auto place_inner = [&](Pos& q) { (ORDER_A ? q.n0 : q.w0) = ilist[q.i] * (ORDER_A ? CG : KW); };
    Pos next = {ni > 0 ? s_lo / ni : 0, ni > 0 ? s_lo % ni : 0, 0, 0, 0};  // (parts: nf = 1)
    static_assert(kRing == 2, "the next stage is copied one ahead");
    if (s_lo < s_hi) {
        place_outer(next);
        place_inner(next);
        issue_outer(next.n0, next.w0);
        locate(next.n0, next.w0, 0);
        issue(0);
    }
    Pos cur_pos = next;
    int buf = 1;  // the current stage's buffer
    auto begin_stage = [&](int si) {
        const bool more = si + 1 < s_hi;
        if (more) {
            if (++next.i == ni) {
                next.i = 0;
                if (!FRAMES || ++next.f == nf) {
                    next.f = 0;
                    ++next.o;
                    place_outer(next);
                    issue_outer(next.n0, next.w0);
                }
            }
            place_inner(next);
            locate(next.n0, next.w0, next.f);
        }
        cp_async_wait_all();
        __syncthreads();
        buf ^= 1;
        if (more) issue(buf ^ 1);
        slot_base = slot0 + (unsigned)(buf * kBufBytes);
    };
    const float2 zero2 = make_float2(0.f, 0.f);
    // Every part of a sub-tile leaves its sums in its slab; the last one to come (true)
    // adds them in order.
    auto sum_of_parts = [&](auto& v, int tile, int sub, int part, int64_t f) {
        constexpr int NV = (int)(sizeof(v) / sizeof(v[0]));
        const int parts = A.split;
        const int64_t u = f * A.n_tiles * kSub + (int64_t)tile * kSub + sub;
        float2* slab = A.partial + u * parts * NV * kThreads + tid;
#pragma unroll
        for (int i = 0; i < NV; ++i) slab[(int64_t)(part * NV + i) * kThreads] = v[i];
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(A.tickets + u, 1u) == (unsigned)(parts - 1);
        __syncthreads();
        if (!s_last) return false;
        __threadfence();
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = make_float2(0.f, 0.f);
        for (int k = 0; k < parts; ++k)
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const float2 a = __ldcg(slab + (int64_t)(k * NV + i) * kThreads);
                v[i].x += a.x;
                v[i].y += a.y;
            }
        return true;
    };
    // dimension.both: the pixel's sum (of all parts)
    auto store_both = [&](int fr) {
        const int tile = s_where[0], sub = s_where[1], part = s_where[2];
        const int p = __ldg(A.tiles + (int64_t)tile * kTile + sub * kThreads + tid);
        const int64_t f = f0 + fr;
        float2 y[1] = {Y[fr]};
        if (part >= 0 && !sum_of_parts(y, tile, sub, part, f)) return;
        if (!in_image(p) || !A.cube) return;
        if (CPLX && A.pix_phase) y[0] = cmul(y[0], __ldg(A.pix_phase + p));
        const int64_t o = p + A.f_f * f;
        if constexpr (CPLX) reinterpret_cast<float2*>(A.cube)[o] = y[0];
        else reinterpret_cast<float*>(A.cube)[o] = y[0].x;
    };

    if constexpr (ORDER_A) {
        int cur = -1, cur_f = 0;  // current wave chunk and frame
        auto zero_chunks = [&](int from, int to) {  // receive mode: skipped chunks are zero
            if constexpr (MODE == USTB_DIM_RECEIVE)
                for (int w = from * KW; w < min(to * KW, (int)W); ++w)
                    for (int64_t f = f0; f < f0 + nf; ++f) store_cube(p + A.w_f * w + A.f_f * f, zero2);
        };
        auto finish_chunk = [&]() {
            const int64_t f = f0 + cur_f;
            const int w0 = cur * KW;
            const int kw = min(KW, (int)W - w0);
#pragma unroll
            for (int k = 0; k < KW; ++k) {
                if (k >= kw) continue;
                float2 y;
                if constexpr (CPLX) y = cmul(Aw[k], sum_of(k));
                else y = make_float2(Aw[k].x * sum_of(k).x, 0.f);
                if (MODE == USTB_DIM_BOTH) {
                    Y[FRAMES ? cur_f : 0].x += y.x;
                    Y[FRAMES ? cur_f : 0].y += y.y;
                } else {
                    store_cube(p + A.w_f * (w0 + k) + A.f_f * f, CPLX ? cmul(y, ph) : y);
                }
            }
        };
        for (int si = s_lo; si < s_hi; ++si, cur_pos = next) {
            const int w0 = cur_pos.w0, n0 = cur_pos.n0;
            const int oc = w0 / KW;
            if (oc != cur || (FRAMES && cur_pos.f != cur_f)) {
                if (cur >= 0) finish_chunk();
                if (oc != cur) {
                    zero_chunks(cur < 0 ? out_lo : cur + 1, oc);
                    setup_tx(w0);
                }
                cur = oc;
                cur_f = cur_pos.f;
#pragma unroll
                for (int k = 0; k < NACC / 2; ++k) accr[k] = acci[k] = 0ull;
            }
            setup_rx(n0);
            begin_stage(si);
            const int kw = min(KW, (int)W - w0);
            auto units = [&](auto full) {
#pragma unroll
                for (int c = 0; c < CG; ++c) {
                    const float2 b = B[c];
                    // a channel whose receive weight is zero for the whole warp adds
                    // nothing (das_c skips zero-apodization units too)
                    if (!__any_sync(0xffffffffu, b.x != 0.f || b.y != 0.f)) continue;
                    const f32x2 bx = pack2(b.x, b.x), by = pack2(b.y, b.y), nby = pack2(-b.y, -b.y);
                    const f32x2 sr = pack2(srx[c], srx[c]);
#pragma unroll
                    for (int k = 0; k < KW; k += 2) {
                        if (!decltype(full)::value && k >= kw) continue;  // last, partial wave chunk
                        unit_pair(k / 2, add2(pack2(stx[k], stx[k + 1]), sr), c, k, c, k + 1, bx, by, nby);
                    }
                }
            };
            if (kw == KW) units(std::true_type{});
            else units(std::false_type{});
        }
        if (cur >= 0) finish_chunk();
        zero_chunks(cur < 0 ? out_lo : cur + 1, out_hi);
        if (MODE == USTB_DIM_BOTH)
            for (int fr = 0; fr < (FRAMES ? nf : 1); ++fr) store_both(fr);
    } else {
        if (MODE == USTB_DIM_NONE) {  // units outside the active stages are zero
            for (int n = 0; n < N; ++n)
                for (int w = 0; w < W; ++w)
                    for (int64_t f = f0; f < f0 + nf; ++f) store_cube(p + A.rx_f * n + A.w_f * w + A.f_f * f, zero2);
        }
        int cur = -1, cur_f = 0;  // current channel group and frame
        unsigned gmask = 0;  // its channels with a nonzero weight in this warp
        auto zero_groups = [&](int from, int to) {
            if constexpr (MODE == USTB_DIM_TRANSMIT)
                for (int n = from * CG; n < min(to * CG, (int)N); ++n)
                    for (int64_t f = f0; f < f0 + nf; ++f) store_cube(p + A.rx_f * n + A.f_f * f, zero2);
        };
        auto finish_group = [&]() {
            if constexpr (MODE == USTB_DIM_NONE) return;
            const int64_t f = f0 + cur_f;
            const int n0 = cur * CG;
            const int cg = min(CG, (int)N - n0);
#pragma unroll
            for (int c = 0; c < CG; ++c) {
                if (c >= cg) continue;
                float2 y;
                // a channel without a weight in this warp may have summed stale windows
                // beside its pair's: it adds nothing
                const float2 a = ((gmask >> c) & 1u) ? sum_of(c) : zero2;
                if constexpr (CPLX) y = cmul(B[c], a);
                else y = make_float2(B[c].x * a.x, 0.f);
                if constexpr (MODE == USTB_DIM_BOTH) {
                    Y[FRAMES ? cur_f : 0].x += y.x;
                    Y[FRAMES ? cur_f : 0].y += y.y;
                } else {
                    if constexpr (CPLX) y = cmul(y, ph);
                    store_cube(p + A.rx_f * (n0 + c) + A.f_f * f, y);
                    if constexpr (EPI) {
                        eS.x += y.x;
                        eS.y += y.y;
                        eI += y.x * y.x + y.y * y.y;
                        const float re = y.x;
                        eR += msign(re) * sqrtf(fabsf(re));
                        eQ += fabsf(re);
                    }
                }
            }
        };
        constexpr unsigned kAll = (1u << CG) - 1u;
        constexpr int kWhole = 0, kMasked = 1, kPart = 2;
        static_assert(KW <= 4, "only the last wave of a chunk that is more than half full can be padding");
        auto units = [&](int n0, int w0, auto all) {
            if constexpr (MODE == USTB_DIM_NONE) {
#pragma unroll
                for (int c = 0; c < CG; ++c) {
#pragma unroll
                    for (int k = 0; k < KW; ++k) {
                        const float s = stx[k] + srx[c], t = __fadd_rz(s, kMagic);
                        const float2 v = interp(c, k, t, s - (t - kMagic));
                        if (n0 + c < N && w0 + k < W && act_n(n0 + c) && act_w(w0 + k)) {
                            const float2 y = CPLX ? cmul(cmul(cmul(Aw[k], B[c]), v), ph)
                                                  : make_float2(Aw[k].x * B[c].x * v.x, 0.f);
                            store_cube(p + A.rx_f * (n0 + c) + A.w_f * (w0 + k) + A.f_f * (f0 + cur_f), y);
                        }
                    }
                }
            } else if constexpr (decltype(all)::value == kWhole) {
#pragma unroll
                for (int k = 0; k < KW; ++k) {
                    if (KW > 2 && k + 1 == KW && w0 + k >= W) continue;  // padding
                    const f32x2 ax = pack2(Aw[k].x, Aw[k].x), ay = pack2(Aw[k].y, Aw[k].y);
                    const f32x2 nay = pack2(-Aw[k].y, -Aw[k].y), st = pack2(stx[k], stx[k]);
#pragma unroll
                    for (int c = 0; c < CG; c += 2)
                        unit_pair(c / 2, add2(st, pack2(srx[c], srx[c + 1])), c, k, c + 1, k, ax, ay, nay);
                }
            } else {
#pragma unroll
                for (int c = 0; c < CG; c += 2) {
                    if (!((gmask >> c) & 3u)) continue;
                    const f32x2 sr = pack2(srx[c], srx[c + 1]);
#pragma unroll
                    for (int k = 0; k < KW; ++k) {
                        if ((decltype(all)::value == kPart || (KW > 2 && k + 1 == KW)) && w0 + k >= W) continue;  // padding
                        unit_pair(c / 2, add2(pack2(stx[k], stx[k]), sr), c, k, c + 1, k, pack2(Aw[k].x, Aw[k].x),
                                  pack2(Aw[k].y, Aw[k].y), pack2(-Aw[k].y, -Aw[k].y));
                    }
                }
            }
        };
        for (int si = s_lo; si < s_hi; ++si, cur_pos = next) {
            const int n0 = cur_pos.n0, w0 = cur_pos.w0;
            const int og = n0 / CG;
            if (og != cur || (FRAMES && cur_pos.f != cur_f)) {
                if (cur >= 0) finish_group();
                if (og != cur) {
                    zero_groups(cur < 0 ? out_lo : cur + 1, og);
                    setup_rx(n0);
                    gmask = 0;
#pragma unroll
                    for (int c = 0; c < CG; ++c)
                        if (MODE == USTB_DIM_NONE || __any_sync(0xffffffffu, B[c].x != 0.f || B[c].y != 0.f)) gmask |= 1u << c;
                }
                cur = og;
                cur_f = cur_pos.f;
#pragma unroll
                for (int c = 0; c < NACC / 2; ++c) accr[c] = acci[c] = 0ull;
            }
            setup_tx(w0);
            begin_stage(si);
            if (w0 + KW / 2 >= W) units(n0, w0, std::integral_constant<int, kPart>{});  // mostly padding
            else if (gmask == kAll) units(n0, w0, std::integral_constant<int, kWhole>{});
            else units(n0, w0, std::integral_constant<int, kMasked>{});
        }
        if (cur >= 0) finish_group();
        zero_groups(cur < 0 ? out_lo : cur + 1, out_hi);
        if constexpr (MODE == USTB_DIM_BOTH)
            for (int fr = 0; fr < (FRAMES ? nf : 1); ++fr) store_both(fr);
        if constexpr (EPI) {
            bool whole = true;  // this CTA has the sums over every channel
            if (!FRAMES && A.split > 1) {
                float2 v[3] = {eS, make_float2(eI, eM), make_float2(eR, eQ)};
                whole = sum_of_parts(v, s_where[0], s_where[1], s_where[2], f0);
                eS = v[0];
                eI = v[1].x;
                eM = v[1].y;
                eR = v[2].x;
                eQ = v[2].y;
            }
            if (live && whole) {
                const int64_t o = p + P * f0;
                float cf = (eS.x * eS.x + eS.y * eS.y) / eI * (1.f / eM);
                if (cf != cf) cf = 0.f;  // NaN -> 0 (coherence_factor.m:132)
                if (A.o_das) A.o_das[o] = eS;
                if (A.o_cf) A.o_cf[o] = cf;
                if (A.o_cfimg) A.o_cfimg[o] = make_float2(cf * eS.x, cf * eS.y);
                if (A.o_sdmas) A.o_sdmas[o] = 0.5f * (eR * eR - eQ);
            }
        }
    }
    __syncthreads();  // the buffers are reused by the next frame, the tables by the next tile
    };
    auto frames = [&](auto stage) {
        build_lists(stage);
        wait_for_entries();
        if constexpr (FRAMES && EPI) {  // the epilogue's sums are one frame's
            for (int64_t f = f_first; f < f_first + nfr; ++f) run(stage, f, 1);
        } else {
            run(stage, f_first, FRAMES ? nfr : 1);
        }
    };
    if constexpr (BIG) {
        if (narrow) frames(Stage<SHAPE, true, false>{});
        else frames(Stage<SHAPE, true, true>{});
    } else {
        frames(Stage<SHAPE, false, false>{});
    }
}

// One launch per request: grid = (tiles x sub-tiles x CTAs per sub-tile, frames).
template <int MODE, int ENT, bool EPI, int SHAPE>
__global__ void __launch_bounds__(kThreads, kSub) das_fast_kernel(const Params A) {
    const int b = (int)(blockIdx.x / A.split), part = A.split >= 2 ? (int)(blockIdx.x % A.split) : -1;
    das_tile<MODE, ENT, EPI, SHAPE>(A, b / kSub, b % kSub, (int64_t)blockIdx.y, part);
}

// Persistent form: the CTAs that fit the SMs pull (request, half tile, frames) work items from a
// queue counter until the batch is done, so requests of different scans, channel
// counts and frame counts share one launch and balance across SMs.  An item is half a
// tile over up to 8 consecutive frames of a request (fewer while that leaves each CTA
// under 8 items), so the tile's tables and receive geometry are built once for those
// frames.
struct BatchParams {
    Params req[kMaxBatch];
    int64_t first_item[kMaxBatch + 1];  // prefix sums of half tiles * frame groups
    int n;
    unsigned long long* counter;        // queue head (device scratch, zeroed per launch)
};

template <int MODE, int ENT, bool EPI, int SHAPE>
__global__ void __launch_bounds__(kThreads, kSub) das_fast_persistent(const __grid_constant__ BatchParams B) {
    __shared__ long long s_item;
    bool first = true;
    const int64_t total = B.first_item[B.n];
    for (;;) {
        if (threadIdx.x == 0) s_item = (long long)atomicAdd(B.counter, 1ull);
        __syncthreads();
        const int64_t item = s_item;
        __syncthreads();
        if (item >= total) break;
        int r = 0;
        while (r + 1 < B.n && B.first_item[r + 1] <= item) ++r;
        const Params& A = B.req[r];
        const int64_t local = item - B.first_item[r];
        const int64_t subs = A.n_tiles * kSub;
        const int64_t f0 = (local / subs) * A.fpi;
        const int b = (int)(local % subs);
        das_tile<MODE, ENT, EPI, SHAPE, true>(A, b / kSub, b % kSub, f0, -1, (int)min((int64_t)A.fpi, A.F - f0), first);
        first = false;
    }
}

// Launch with leave to start while the kernel before it in the stream ends: the CTAs set
// their tile up (8 to 10 us of dependent loads and long arithmetic) beside the end of the
// entries pre-pass.  After anything but a kernel the launch is an ordinary one.
template <typename K, typename P>
cudaError_t launch_dependent(K* kern, dim3 grid, size_t smem, cudaStream_t s, const P& params) {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, params);
}

template <int MODE, int ENT, bool EPI, int SHAPE>
int launch(const Params& A, int64_t n_tiles, int64_t F, cudaStream_t s) {
    const size_t smem = smem_bytes(SHAPE, A.N, A.W);
    auto kern = das_fast_kernel<MODE, ENT, EPI, SHAPE>;
    size_t limit = 0;
    const int rc = shared_limit((const void*)kern, limit);
    if (rc) return rc;
    USTB_REQUIRE(smem <= limit, USTB_E_SHAPE,
                 "%lld channels / %lld waves need %zu bytes of shared memory per tile (limit %zu)",
                 (long long)A.N, (long long)A.W, smem, limit);
    dim3 grid((unsigned)(n_tiles * kSub * A.split), (unsigned)F);
    // only the pre-pass is known to leave the outputs and the geometry alone
    if (A.after_entries) {
        USTB_CUDA(launch_dependent(kern, grid, smem, s, A));
    } else {
        kern<<<grid, kThreads, smem, s>>>(A);
    }
    USTB_CUDA(cudaGetLastError());
    return USTB_OK;
}

template <int MODE, int ENT, bool EPI, int SHAPE>
int launch_batch(const Params* reqs, const int64_t* frames, int n, unsigned long long* counter, int max_ctas,
                 cudaStream_t s) {
    BatchParams B;
    B.n = n;
    B.counter = counter;
    B.first_item[0] = 0;
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    size_t smem = 0;
    for (int i = 0; i < n; ++i) smem = std::max(smem, smem_bytes(SHAPE, reqs[i].N, reqs[i].W));
    int fit = 0;
    int rc = ctas_per_sm(smem, fit);
    if (rc) return rc;
    const int64_t nct = (max_ctas > 0 ? std::min(max_ctas, sms) : sms) * (int64_t)std::min(fit, kSub);
    for (int i = 0; i < n; ++i) {
        B.req[i] = reqs[i];
        // frames per work item: up to kItemFrames, while every CTA keeps at least 8 items of the request
        const int64_t subs = reqs[i].n_tiles * kSub;
        const int64_t fpi = std::max<int64_t>(1, std::min<int64_t>(kItemFrames, subs * frames[i] / (8 * nct)));
        B.req[i].fpi = (int)fpi;
        B.first_item[i + 1] = B.first_item[i] + subs * ((frames[i] + fpi - 1) / fpi);
    }
    if (B.first_item[n] == 0) return USTB_OK;
    auto kern = das_fast_persistent<MODE, ENT, EPI, SHAPE>;
    size_t limit = 0;
    rc = shared_limit((const void*)kern, limit);
    if (rc) return rc;
    USTB_REQUIRE(smem <= limit, USTB_E_SHAPE, "a request needs %zu bytes of shared memory per tile (limit %zu)", smem,
                 limit);
    USTB_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s));
    // as many CTAs as the SMs hold, or fewer (max_ctas SMs) to leave room to launches on other streams
    const unsigned grid = (unsigned)std::min<int64_t>(B.first_item[n], nct);
    kern<<<grid, kThreads, smem, s>>>(B);
    USTB_CUDA(cudaGetLastError());
    return USTB_OK;
}

}  // namespace

// Kernel variant of (dimension, epilogue, stage shape) for one request kind.
template <int ENT, bool BATCH, int SUBS>
int das_dispatch(int dim, int epi, int shape, const Params* reqs, const int64_t* frames, int n,
             unsigned long long* counter, int64_t nt, int64_t F, cudaStream_t s, int max_ctas) {
    static_assert(SUBS == kSub, "the including file sets the number");
    auto run = [&](auto m, auto e, auto sh) {
        constexpr int M = decltype(m)::value, S = decltype(sh)::value;
        constexpr bool E = decltype(e)::value;
        if constexpr (BATCH) return launch_batch<M, ENT, E, S>(reqs, frames, n, counter, max_ctas, s);
        else return launch<M, ENT, E, S>(reqs[0], nt, F, s);
    };
#define USTB_RUN(M, E, S) \
    return run(std::integral_constant<int, M>{}, std::integral_constant<bool, E>{}, std::integral_constant<int, S>{})
    constexpr bool k16 = ENT == kEntHalf || ENT == kEntBf16;        // (entries_for: the library's shapes only)
    constexpr bool kOwn = k16 || (BATCH && ENT == kEntComplex);     // (as das_fast_batch_impl sets them)
    if constexpr (SUBS == 2) {  // (subs_for: whole tiles for dimension.both only)
        if constexpr (!k16)
            if (dim == USTB_DIM_NONE) {
                if constexpr (!kOwn)
                    if (shape == 2) USTB_RUN(USTB_DIM_NONE, false, 2);
                USTB_RUN(USTB_DIM_NONE, false, 1);
            }
        if (dim == USTB_DIM_RECEIVE) {
            if constexpr (!k16) {
                if (shape == 4) USTB_RUN(USTB_DIM_RECEIVE, false, 4);
                if (shape == 5) USTB_RUN(USTB_DIM_RECEIVE, false, 5);
            }
            if constexpr (!kOwn)
                if (shape == 0) USTB_RUN(USTB_DIM_RECEIVE, false, 0);
            USTB_RUN(USTB_DIM_RECEIVE, false, 3);
        }
        if (dim == USTB_DIM_TRANSMIT) {
            if constexpr (ENT != kEntReal)
                if (epi) {
                    if constexpr (!kOwn)
                        if (shape == 2) USTB_RUN(USTB_DIM_TRANSMIT, true, 2);
                    USTB_RUN(USTB_DIM_TRANSMIT, true, 1);
                }
            if constexpr (!kOwn)
                if (shape == 2) USTB_RUN(USTB_DIM_TRANSMIT, false, 2);
            USTB_RUN(USTB_DIM_TRANSMIT, false, 1);
        }
    }
    if constexpr (!kOwn) {
        if (shape == 0) USTB_RUN(USTB_DIM_BOTH, false, 0);
        if (shape == 2) USTB_RUN(USTB_DIM_BOTH, false, 2);
    }
    USTB_RUN(USTB_DIM_BOTH, false, 1);
#undef USTB_RUN
}

}  // namespace ustb

// RF -> IQ demodulation fused with the conversion into the fast path's storage type:
// down-mix, low-pass FIR and decimation in one pass over the RF samples
// (+preprocess/fast_demodulation.m:121-167 and :286-293 for the filter):
//
//   mix[j] = scale * x[j] * exp(-i 2 pi fc t_j),   t_j = t0 + j / fs
//   y[m]   = sum_k b[k] * mix[m*D - k]              (causal FIR, zero before j = 0)
//
// for m = 0 .. ceil(L/D) - 1 (MATLAB's data(1:D:end,...)).  The caller shifts the
// output's initial time by the filter delay (ntaps - 1) / 2 / fs.
//
// The mixer's phase is moved from the samples into the taps and the outputs,
//   y[m] = exp(-i 2 pi fc t_(mD)) * sum_k (scale b[k] exp(i 2 pi fc k / fs)) * x[m*D - k],
// so the FIR runs over the real samples as they are (one word of shared memory each, no
// sine and cosine per sample) with complex taps, at the same 2 FMA per tap and output.
//
// One CTA computes kout (<= 1024) consecutive outputs of tp traces (as many as fill its
// threads, fewer where that leaves SMs without a CTA) and loops over trace groups, so the complex taps are formed once per CTA.  It
// stages the samples that the outputs need in shared memory in polyphase order
// (phase-major): output o reads, for tap k, position o + (last - k)/D of row (last - k) % D,
// so the taps of one row step one position at a time.  Each thread forms two runs of 4
// consecutive outputs; per block of 4 taps of a row it loads 4 new samples of each run (a
// 16-byte load, neighbouring threads neighbouring addresses; the other 3 it spans are in
// registers) and the 4 taps (two broadcast loads) for 64 FMA.  While a group is computed,
// the next group's samples are copied into shared memory as they are.  The output phase
// is formed in cycles as c0 + j*step with step split into two floats and the product's
// rounding error recovered by an FMA, so it stays exact to ~1e-7 cycles over any trace
// length.  The outputs leave through shared memory, so that the stores are contiguous.
//
// Instruction-bound (75 % issue; HBM would take 51 us).  GB300, a call on 56320 int16 traces
// of 1536 samples, 31 taps, decimation 2, half-precision output: 284 us (515 us with a
// mixed complex sample staged per input sample); zero phase, 14080 float traces of 1536,
// 129 taps, decimation 4: 164 us (246 us).
//
// The zero-phase variant (ustb_demodulate_filtfilt, the reference's Python port,
// python/src/ustb/preprocess/fast_demodulation.py:47-76) is the same pass with the
// taps replaced by the autocorrelation of b (2 ntaps - 1 of them, formed per CTA),
// the sequence shifted by ntaps - 1 samples so the filter is centred, and the
// trace odd-extended about its end samples (scipy filtfilt's padding) instead of
// zero-extended.  The extension 2 X_e - X_r of the mixed trace is not a real sequence at
// the mixer's phase, so the few outputs within ntaps samples of an end add its terms
// separately, one thread per output.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int kThreads = 256;            // threads per CTA at most
constexpr int kRun = 4;                  // consecutive outputs of a run
constexpr int kOPT = 2 * kRun;           // outputs per thread: two runs, half of the trace's outputs apart
constexpr int kTB = 4;                   // taps per register block
constexpr int kOutMax = 1024;            // outputs per CTA and trace at most
// output o of a trace in shared memory, one float2 of padding after every run (distinct banks)
__host__ __device__ __forceinline__ int out_pad(int o) { return o + (o >> 2); }
constexpr int kStage = 16384;            // staged samples per CTA at most (64 KB), when kout allows

template <typename S>
__device__ __forceinline__ float rf_sample(const S* p, int64_t i);
template <>
__device__ __forceinline__ float rf_sample<float>(const float* p, int64_t i) { return __ldg(p + i); }
template <>
__device__ __forceinline__ float rf_sample<int16_t>(const int16_t* p, int64_t i) { return (float)__ldg(p + i); }
template <>
__device__ __forceinline__ float rf_sample<__half>(const __half* p, int64_t i) { return __half2float(__ldg(p + i)); }

// 4 consecutive samples as floats, from an address aligned to 4 samples
__device__ __forceinline__ float4 vec4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 vec4(const int16_t* p) {
    // exact: x + 32768 put into the mantissa of 2^23, then 2^23 + 32768 taken off (the
    // conversion instruction runs at a quarter of the rate)
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    auto lo = [](uint32_t w) { return __uint_as_float((w & 0xFFFFu) ^ 0x4B008000u) - 8421376.0f; };
    auto hi = [](uint32_t w) { return __uint_as_float((w >> 16) ^ 0x4B008000u) - 8421376.0f; };
    return make_float4(lo(u.x), hi(u.x), lo(u.y), hi(u.y));
}
__device__ __forceinline__ float4 vec4(const __half* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
// asynchronous copy of 4 samples (both addresses aligned to 4 samples)
template <typename S>
__device__ __forceinline__ void copy4_async(S* dst, const S* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(S) == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
template <typename S>
__device__ __forceinline__ S zero_sample() { return S(0); }
template <>
__device__ __forceinline__ __half zero_sample<__half>() { return __float2half_rn(0.f); }

template <typename D>
__device__ __forceinline__ void store_iq(D* out, int64_t i, float2 v);
template <>
__device__ __forceinline__ void store_iq<float>(float* out, int64_t i, float2 v) {
    reinterpret_cast<float2*>(out)[i] = v;
}
template <>
__device__ __forceinline__ void store_iq<__half>(__half* out, int64_t i, float2 v) {
    reinterpret_cast<__half2*>(out)[i] = __floats2half2_rn(v.x, v.y);
}
template <>
__device__ __forceinline__ void store_iq<__nv_bfloat16>(__nv_bfloat16* out, int64_t i, float2 v) {
    reinterpret_cast<__nv_bfloat162*>(out)[i] = __floats2bfloat162_rn(v.x, v.y);
}

struct DemodArgs {
    int64_t L, Ld, n_traces, chunks, groups;  // chunks of kout outputs per trace, groups of (chunk, tp traces)
    int D, ntaps, kout;
    int tp, tpt, threads;  // traces per CTA, threads per trace and of a CTA
    int mb, shift;         // zero-phase: taps of the reference filter, and mb - 1
    int Qp, Cap;           // padded row stride (words); taps per polyphase row (a multiple of kTB)
    int raw;               // samples copied ahead per trace (a multiple of 4)
    int edges;             // zero-phase: outputs near one end that read the extension, at most
    int vec;               // the RF pointer is aligned to 4 samples
    uint32_t inv_d;        // ceil(2^32 / D): s / D = high word of s * inv_d for s < 2^20
    float c0;              // fractional part of fc * t0 (cycles)
    float step_hi, step_lo;  // fc / fs split into two floats
    float scale;
};

// nearest integer of |v| < 2^22
__device__ __forceinline__ float nearest(float v) { return __fsub_rn(__fadd_rn(v, 12582912.0f), 12582912.0f); }
// cycles (within a few periods of 0) of the mixer at sample j, |j| < 2^24, from sample 0: frac(j fc / fs)
__device__ __forceinline__ float cycles_at(int j, const DemodArgs& a) {
    const float jf = (float)j;  // exact: |j| < 2^24
    const float p = jf * a.step_hi;
    const float e = fmaf(jf, a.step_hi, -p);  // rounding error of the product
    return (p - rintf(p)) + fmaf(jf, a.step_lo, e);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// exp(-i 2 pi (c0 + j fc / fs))
__device__ __forceinline__ float2 phasor_at(int j, const DemodArgs& a) {
    const float cyc = a.c0 + cycles_at(j, a);
    float sn, cs;
    __sincosf(-6.283185307179586f * (cyc - nearest(cyc)), &sn, &cs);
    return make_float2(cs, sn);
}

// Shared memory (words): complex taps by polyphase row [D * Cap] x 2, staged samples
// [tp][D * Qp], the next group's samples as they are [tp][raw], outputs [tp][kout] x 2, then, zero-phase, the real taps [ntaps], the
// extension [tp][2][mb - 1] x 2 and the edge outputs' extension sums [tp][2][edges] x 2.
struct DemodLayout {
    size_t taps, raw, x, out, real, ext, esum, total;
};
__host__ __device__ __forceinline__ DemodLayout demod_layout(const DemodArgs& a, bool zp) {
    DemodLayout l;
    auto up = [](size_t v) { return (v + 3) & ~(size_t)3; };
    l.taps = 0;
    l.x = up(2 * (size_t)a.D * a.Cap);
    l.raw = l.x + up((size_t)a.tp * a.D * a.Qp);
    l.out = l.raw + up((size_t)a.tp * a.raw);  // (room for 4-byte samples)
    l.real = l.out + up(2 * (size_t)a.tp * out_pad(a.kout) + 2);
    l.ext = l.real + (zp ? up((size_t)a.ntaps) : 0);
    l.esum = l.ext + (zp ? up(4 * (size_t)a.tp * a.mb) : 0);
    l.total = l.esum + (zp ? up(4 * (size_t)a.tp * a.edges) : 0);
    return l;
}

template <typename S, typename D, bool ZP>
__global__ void __launch_bounds__(kThreads, 4) demod_kernel(const S* __restrict__ rf, D* __restrict__ iq,
                                                         const float* __restrict__ taps, const DemodArgs a) {
    extern __shared__ __align__(16) float sm[];
    const DemodLayout lay = demod_layout(a, ZP);
    float2* g = reinterpret_cast<float2*>(sm + lay.taps);
    float* xs = sm + lay.x;
    float2* outs = reinterpret_cast<float2*>(sm + lay.out);
    float2* ext = reinterpret_cast<float2*>(sm + lay.ext);
    float2* esum = reinterpret_cast<float2*>(sm + lay.esum);
    S* raws = reinterpret_cast<S*>(sm + lay.raw);
    __shared__ float2 step[kRun];  // exp(-i 2 pi q D fc / fs): the mixer from a thread's first output to its q-th
    const int nthr = blockDim.x, tid = threadIdx.x;
    const int last = a.ntaps - 1;
    float* htap = sm + lay.real;
    if constexpr (ZP) {
        // the single FIR equal to filtfilt at the kept samples: the autocorrelation
        // h[t] = sum_j b[j] b[j - t], |t| < mb (b staged in the extension's space)
        float* bt = sm + lay.ext;
        for (int k = tid; k < a.mb; k += nthr) bt[k] = __ldg(taps + k);
        __syncthreads();
        // two neighbouring threads per tap, each summing half of the products
        for (int i0 = 0; i0 < 2 * a.ntaps; i0 += nthr) {  // bounds uniform across the CTA
            const int i = i0 + tid, k = i >> 1;
            float h = 0.f;
            if (k < a.ntaps) {
                const int t = k - (a.mb - 1);
                const int lo = max(0, t), hi = min(a.mb, a.mb + t), mid = (lo + hi) >> 1;
                for (int j = (i & 1) ? mid : lo; j < ((i & 1) ? hi : mid); ++j) h = fmaf(bt[j], bt[j - t], h);
            }
            h += __shfl_xor_sync(0xffffffffu, h, 1);
            if (k < a.ntaps && !(i & 1)) htap[k] = a.scale * h;
        }
        __syncthreads();
    }
    // complex taps g[k] = scale b[k] exp(i 2 pi fc (k - shift) / fs), tap k in row
    // (last - k) % D at (last - k) / D; zeros pad the rows
    for (int i = tid; i < a.D * a.Cap; i += nthr) {
        const int ph = i / a.Cap, m = i - ph * a.Cap;
        const int k = last - ph - m * a.D;
        float2 v = make_float2(0.f, 0.f);
        if (k >= 0 && k < a.ntaps) {
            const float b = ZP ? htap[k] : a.scale * __ldg(taps + k);
            const float cyc = cycles_at(k - a.shift, a);
            float sn, cs;
            sincospif(2.f * (cyc - rintf(cyc)), &sn, &cs);
            v = make_float2(b * cs, b * sn);
        }
        g[i] = v;
    }
    if (tid < kRun) {
        const float cyc = cycles_at(tid * a.D, a);
        float sn, cs;
        sincospif(-2.f * (cyc - rintf(cyc)), &sn, &cs);
        step[tid] = make_float2(cs, sn);
    }
    // the rows' tails, read by the last outputs' padded tap blocks, stay zero
    for (int i = tid; i < a.tp * a.D * a.Qp; i += nthr) xs[i] = 0.f;
    const int nstage = a.kout * a.D + a.ntaps - 1;  // staged samples per trace
    const int my_tr = tid / a.tpt, half = kRun * a.tpt, o0 = (tid - my_tr * a.tpt) * kRun;  // runs o0.., half + o0..
    const int L = (int)a.L, Ld = (int)a.Ld;
    const int t0 = 4 * (tid - my_tr * a.tpt);  // this thread stages samples t0 + 4 tpt i .. + 3 of its trace
    S* const raw = raws + my_tr * a.raw;
    struct Group { int64_t first; int m0, j0, off, ntr; };
    auto group_at = [&](uint32_t gid) {
        const uint32_t tg = a.chunks == 1 ? gid : gid / (uint32_t)a.chunks;
        Group q;
        const int64_t trace0 = (int64_t)tg * a.tp;
        q.first = (trace0 + my_tr) * a.L;  // first sample of this thread's trace
        q.m0 = (int)(gid - tg * (uint32_t)a.chunks) * a.kout;
        q.ntr = (int)min((int64_t)a.tp, a.n_traces - trace0);
        q.j0 = q.m0 * a.D - last + a.shift;  // trace index of staged sample 0
        q.off = (int)((uint32_t)(q.first + q.j0) & 3u);
        return q;
    };
    // copies a group's samples as they are, from where the address is 4-sample aligned,
    // while the group before is computed; zeros outside the trace
    auto fetch = [&](const Group& q) {
        if (my_tr >= q.ntr) return;
        const S* x = rf + q.first;
        for (int s = t0; s < nstage + q.off; s += 4 * a.tpt) {
            const int jv = q.j0 + s - q.off;
            if (a.vec && jv >= 0 && jv + 3 < L) {
                copy4_async<S>(raw + s, x + jv);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) raw[s + u] = (jv + u >= 0 && jv + u < L) ? __ldg(x + jv + u) : zero_sample<S>();
            }
        }
    };
    // this thread's copied samples into the polyphase rows
    auto place = [&](const Group& q, float* rows, auto dec) {
        constexpr int DEC = decltype(dec)::value;  // the decimation 1, 2 or 4, or 0: any
        for (int s = t0; s < nstage + q.off; s += 4 * a.tpt) {
            const int s0 = s - q.off;
            const float4 w = vec4(raw + s);
            const float v[4] = {w.x, w.y, w.z, w.w};
            if (DEC > 0 && s0 >= 0 && s0 + 3 < nstage) {
                // sample s0's row is the same for every thread (s0 = -off mod 4)
                constexpr int SH = DEC == 4 ? 2 : DEC == 2 ? 1 : 0;
                float* dst = rows + (s0 >> SH);
                const int ph0 = -q.off & (DEC - 1);
#pragma unroll
                for (int u = 0; u < 4; ++u) dst[((ph0 + u) & (DEC - 1)) * a.Qp + ((ph0 + u) >> SH)] = v[u];
                continue;
            }
            // row and position of sample s0 (of sample 0 where s0 < 0)
            int p = a.D == 1 ? max(s0, 0) : (int)__umulhi((uint32_t)max(s0, 0), a.inv_d);
            int ph = max(s0, 0) - p * a.D;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (s0 + u < 0 || s0 + u >= nstage) continue;
                rows[ph * a.Qp + p] = v[u];
                if (++ph == a.D) {
                    ph = 0;
                    ++p;
                }
            }
        }
    };
    Group cur = group_at(blockIdx.x);
    fetch(cur);
    for (uint32_t gid = blockIdx.x; gid < (uint32_t)a.groups; gid += gridDim.x) {
        const int64_t trace0 = (int64_t)(a.chunks == 1 ? gid : gid / (uint32_t)a.chunks) * a.tp;
        const int m0 = cur.m0, ntr = cur.ntr;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // the previous group's samples and outputs are read
        if (my_tr < ntr) {  // a trace is staged by the threads that form its outputs
            float* rows = xs + my_tr * a.D * a.Qp;
            if (a.D == 1) place(cur, rows, std::integral_constant<int, 1>{});
            else if (a.D == 2) place(cur, rows, std::integral_constant<int, 2>{});
            else if (a.D == 4) place(cur, rows, std::integral_constant<int, 4>{});
            else place(cur, rows, std::integral_constant<int, 0>{});
        }
        if (gid + gridDim.x < (uint32_t)a.groups) {
            cur = group_at(gid + gridDim.x);
            fetch(cur);
        }
        if constexpr (ZP) {
            // the odd extension of the mixed trace past its ends: 2 X_e - X_r, r = 1 .. mb - 1
            const int ne = a.mb - 1;
            const bool left = m0 * a.D < ne, right = (m0 + a.kout - 1) * a.D > L - a.mb;
            if (left || right) {
                for (int i = tid; i < ntr * 2 * ne; i += nthr) {
                    const int tr = i / (2 * ne), e = i - tr * 2 * ne, side = e >= ne, r = e - side * ne + 1;
                    const S* x = rf + (trace0 + tr) * a.L;
                    const int je = side ? L - 1 : 0, jr = side ? L - 1 - r : r;
                    const float2 te = phasor_at(je, a), tr2 = phasor_at(jr, a);
                    const float ve = 2.f * rf_sample<S>(x, je), vr = rf_sample<S>(x, jr);
                    ext[i] = make_float2(ve * te.x - vr * tr2.x, ve * te.y - vr * tr2.y);
                }
                __syncthreads();
                // edge output (trace, side, i): left m = i, right m = Ld - 1 - i; the taps reach
                // the extension's entries r at h[mb - 1 + dist + r] (h is symmetric), dist the
                // output's distance from the end sample
                for (int u = tid; u < ntr * 2 * a.edges; u += nthr) {
                    const int tr = u / (2 * a.edges), e = u - tr * 2 * a.edges, side = e >= a.edges, i = e - side * a.edges;
                    const int m = side ? Ld - 1 - i : i;
                    const int dist = side ? L - 1 - m * a.D : m * a.D;
                    const int nr = (m >= 0 && m < Ld) ? a.mb - 1 - dist : 0;  // entries r = 1 .. nr
                    const float2* er = ext + (tr * 2 + side) * ne;
                    const float* h = htap + a.mb + dist;
                    float2 v = make_float2(0.f, 0.f);
                    for (int r = 0; r < nr; ++r) {
                        v.x = fmaf(h[r], er[r].x, v.x);
                        v.y = fmaf(h[r], er[r].y, v.y);
                    }
                    esum[u] = v;
                }
            }
        }
        __syncthreads();
        // Two runs of kRun consecutive outputs per thread.  Output o at tap k reads staged
        // sample o*D + last - k, i.e. row (last - k) % D at o + (last - k) / D: the taps of
        // one row, k = last - ph - m*D, step the read position by one.  (Scalar FMAs: a
        // packed pair takes as long as four of them and needs each sample twice.)
        if (my_tr < ntr) {
            float ar[2][kRun], ai[2][kRun];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < kRun; ++q) ar[h][q] = ai[h][q] = 0.f;
            for (int ph = 0; ph < a.D && ph <= last; ++ph) {
                const int nb = (last - ph) / a.D / kTB + 1;  // blocks of kTB taps of this row
                const float4* xa = reinterpret_cast<const float4*>(xs + (my_tr * a.D + ph) * a.Qp + o0);
                const float4* xb = reinterpret_cast<const float4*>(xs + (my_tr * a.D + ph) * a.Qp + half + o0);
                const float4* tr4 = reinterpret_cast<const float4*>(g + ph * a.Cap);
                float4 wa0 = xa[0], wb0 = xb[0], wa1, wb1;
                // taps 4b .. 4b + 3 over the 7 samples from position 4b on, in x and the new y
                auto run = [&](int h, const float4& t0, const float4& t1, const float4& x, const float4& y) {
                    const float re[kTB] = {t0.x, t0.z, t1.x, t1.z}, im[kTB] = {t0.y, t0.w, t1.y, t1.w};
                    const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                    for (int mm = 0; mm < kTB; ++mm)
#pragma unroll
                        for (int q = 0; q < kRun; ++q) {
                            ar[h][q] = fmaf(re[mm], w[q + mm], ar[h][q]);
                            ai[h][q] = fmaf(im[mm], w[q + mm], ai[h][q]);
                        }
                };
                auto block = [&](int b, const float4& pa, float4& na, const float4& pb, float4& nbb) {
                    na = xa[b + 1];
                    nbb = xb[b + 1];
                    const float4 t0 = tr4[2 * b], t1 = tr4[2 * b + 1];
                    run(0, t0, t1, pa, na);
                    run(1, t0, t1, pb, nbb);
                };
                int b = 0;
                for (; b + 2 <= nb; b += 2) {
                    block(b, wa0, wa1, wb0, wb1);
                    block(b + 1, wa1, wa0, wb1, wb0);
                }
                if (b < nb) block(b, wa0, wa1, wb0, wb1);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int oh = o0 + h * half;
                float2* my_out = outs + my_tr * out_pad(a.kout) + out_pad(oh);
                const int no = min(kRun, min(a.kout - oh, Ld - m0 - oh));
                const float2 mix0 = phasor_at((m0 + oh) * a.D, a);
#pragma unroll
                for (int q = 0; q < kRun; ++q) {
                    if (q >= no) continue;
                    const int m = m0 + oh + q;
                    float2 y = cmul(cmul(mix0, step[q]), make_float2(ar[h][q], ai[h][q]));
                    if constexpr (ZP) {
                        float2 e = make_float2(0.f, 0.f);
                        if (m * a.D < a.mb - 1) e = esum[my_tr * 2 * a.edges + m];
                        else if (L - 1 - m * a.D < a.mb - 1) e = esum[(my_tr * 2 + 1) * a.edges + Ld - 1 - m];
                        y.x += e.x;
                        y.y += e.y;
                    }
                    my_out[q] = y;
                }
            }
        }
        __syncthreads();
        const int nout = min(a.kout, Ld - m0);
        for (int tr = 0; tr < ntr; ++tr) {
            D* dst = iq + 2 * ((trace0 + tr) * a.Ld + m0);
            for (int o = tid; o < nout; o += nthr) store_iq<D>(dst, o, outs[tr * out_pad(a.kout) + out_pad(o)]);
        }
    }
}

// The split of the work: outputs per trace and CTA (the trace's Ld outputs in the fewest
// equal chunks: a last, short chunk would leave most of its CTA idle), threads per trace
// and as many traces as fill the CTA's threads and its shared memory, or few enough that
// every SM has a group (128 traces of 645 samples, in a graph: 31 taps, decimation 2, 5.8 us
// with full CTAs, 4.8; zero phase 11.9, 8.5; 256 of 1536, zero phase, 10.0, 9.6; with 64
// threads to such a CTA 4.9, 10.6 and 10.0).
void plan_demod(DemodArgs& a, bool zp, bool vec, int sms) {
    const int64_t kmax = std::max<int64_t>(32, std::min<int64_t>(kOutMax, (kStage - a.ntaps) / a.D));
    a.chunks = (a.Ld + kmax - 1) / kmax;
    a.kout = (int)((a.Ld + a.chunks - 1) / a.chunks);
    a.tpt = (a.kout + kOPT - 1) / kOPT;
    a.inv_d = a.D > 1 ? (uint32_t)(((uint64_t(1) << 32) + a.D - 1) / a.D) : 0;
    a.Cap = ((a.ntaps - 1) / a.D / kTB + 1) * kTB;
    // the farthest position a thread's last tap block loads is below 8 tpt + Cap + 4
    a.Qp = (a.tpt * kOPT + a.Cap + 4 + 3) & ~3;
    a.raw = (a.kout * a.D + a.ntaps - 1 + 3 + 3) & ~3;
    a.edges = zp ? std::max(1, (a.mb - 2) / a.D + 1) : 0;
    a.vec = vec ? 1 : 0;
    const int64_t per_trace = (int64_t)a.D * a.Qp + a.raw + 2 * a.kout + (zp ? 4 * (a.mb - 1) + 4 * a.edges : 0);
    const int64_t fill = std::max<int64_t>(1, std::min<int64_t>((int64_t)kThreads / a.tpt, 12288 / per_trace));
    const int64_t each = (a.n_traces * a.chunks + sms - 1) / sms;  // a group for every SM
    a.tp = (int)std::min(fill, each);
    // a CTA of fewer traces keeps the threads: they form its taps and leave its outputs
    a.threads = each < fill ? kThreads : (a.tp * a.tpt + 31) / 32 * 32;
    a.groups = (a.n_traces + a.tp - 1) / a.tp * a.chunks;
}


template <typename S, bool ZP>
int launch_demod(const S* rf, void* iq, int32_t dst_type, const float* taps, DemodArgs a, cudaStream_t s) {
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    plan_demod(a, ZP, ((uintptr_t)rf & (4 * sizeof(S) - 1)) == 0, sms);
    USTB_REQUIRE(a.groups <= INT32_MAX, USTB_E_SHAPE, "too many traces x output chunks");
    const size_t smem = sizeof(float) * demod_layout(a, ZP).total;
    const unsigned blocks = (unsigned)std::min<int64_t>(a.groups, (int64_t)sms * 16);
    auto start = [&](auto kern, auto* dst) -> int {
        size_t limit = 0;
        const int rc = ustb::shared_limit((const void*)kern, limit);
        if (rc) return rc;
        USTB_REQUIRE(smem <= limit, USTB_E_SHAPE, "decimation %d with %d taps needs %zu bytes of shared memory", a.D,
                     a.ntaps, smem);
        kern<<<blocks, a.threads, smem, s>>>(rf, dst, taps, a);
        USTB_CUDA(cudaGetLastError());
        return USTB_OK;
    };
    switch (dst_type) {
        case USTB_STORE_F32: return start(demod_kernel<S, float, ZP>, (float*)iq);
        case USTB_STORE_F16: return start(demod_kernel<S, __half, ZP>, (__half*)iq);
        default: return start(demod_kernel<S, __nv_bfloat16, ZP>, (__nv_bfloat16*)iq);
    }
}

}  // namespace

extern "C" int ustb_demodulate(const void* rf, int32_t src_type, void* iq, int32_t dst_type, int64_t L,
                               int64_t n_traces, double fs, double t0, double fc, int32_t decimation,
                               const float* taps, int32_t ntaps, float scale, void* stream) {
    ustb::clear_error();
    USTB_REQUIRE(src_type >= 0 && src_type <= 2, USTB_E_DTYPE, "unknown source type %d", (int)src_type);
    USTB_REQUIRE(dst_type >= 0 && dst_type <= 2, USTB_E_DTYPE, "unknown storage type %d", (int)dst_type);
    USTB_REQUIRE(L >= 0 && n_traces >= 0, USTB_E_SHAPE, "negative size");
    USTB_REQUIRE(L < (1 << 24), USTB_E_SHAPE, "at most 2^24 samples per trace");
    USTB_REQUIRE(decimation >= 1 && decimation <= 64, USTB_E_ARG, "decimation must be in [1, 64], got %d",
                 (int)decimation);
    USTB_REQUIRE(ntaps >= 1 && ntaps <= 4096, USTB_E_ARG, "ntaps must be in [1, 4096], got %d", (int)ntaps);
    USTB_REQUIRE(fs > 0.0, USTB_E_ARG, "sampling frequency must be > 0");
    if (L == 0 || n_traces == 0) return USTB_OK;
    USTB_REQUIRE(rf && iq && taps, USTB_E_ARG, "NULL pointer");
    DemodArgs a;
    a.L = L;
    a.Ld = (L + decimation - 1) / decimation;
    a.n_traces = n_traces;
    a.D = decimation;
    a.ntaps = ntaps;
    const double c0 = fc * t0;
    a.c0 = (float)(c0 - std::floor(c0));
    const double step = fc / fs;
    a.step_hi = (float)step;
    a.step_lo = (float)(step - (double)a.step_hi);
    a.scale = scale;
    a.mb = ntaps;
    a.shift = 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (src_type) {
        case USTB_SRC_F32: return launch_demod<float, false>((const float*)rf, iq, dst_type, taps, a, s);
        case USTB_SRC_I16: return launch_demod<int16_t, false>((const int16_t*)rf, iq, dst_type, taps, a, s);
        default: return launch_demod<__half, false>((const __half*)rf, iq, dst_type, taps, a, s);
    }
}

extern "C" int ustb_demodulate_filtfilt(const void* rf, int32_t src_type, void* iq, int32_t dst_type, int64_t L,
                                        int64_t n_traces, double fs, double t0, double fc, int32_t decimation,
                                        const float* taps, int32_t ntaps, float scale, void* stream) {
    ustb::clear_error();
    USTB_REQUIRE(src_type >= 0 && src_type <= 2, USTB_E_DTYPE, "unknown source type %d", (int)src_type);
    USTB_REQUIRE(dst_type >= 0 && dst_type <= 2, USTB_E_DTYPE, "unknown storage type %d", (int)dst_type);
    USTB_REQUIRE(L >= 0 && n_traces >= 0, USTB_E_SHAPE, "negative size");
    USTB_REQUIRE(L < (1 << 24), USTB_E_SHAPE, "at most 2^24 samples per trace");
    USTB_REQUIRE(decimation >= 1 && decimation <= 64, USTB_E_ARG, "decimation must be in [1, 64], got %d",
                 (int)decimation);
    USTB_REQUIRE(ntaps >= 1 && ntaps <= 1024, USTB_E_ARG, "ntaps must be in [1, 1024], got %d", (int)ntaps);
    USTB_REQUIRE(fs > 0.0, USTB_E_ARG, "sampling frequency must be > 0");
    if (n_traces == 0) return USTB_OK;
    // scipy filtfilt: the trace must be longer than the padding
    USTB_REQUIRE(L > 3 * (int64_t)ntaps, USTB_E_SHAPE,
                 "the trace (%lld samples) must be longer than the padding 3 * ntaps = %d", (long long)L,
                 3 * (int)ntaps);
    USTB_REQUIRE(rf && iq && taps, USTB_E_ARG, "NULL pointer");
    // At every kept sample, filtfilt equals one FIR with the 2 ntaps - 1 taps of b's
    // autocorrelation applied to the odd-extended mixed trace: the kept outputs only
    // use forward values at least 2 ntaps + 1 samples into the extension and backward
    // sums that end at least 2 ntaps samples before its end, so neither pass's
    // steady-state start is reached.
    DemodArgs a;
    a.L = L;
    a.Ld = (L + decimation - 1) / decimation;
    a.n_traces = n_traces;
    a.D = decimation;
    a.ntaps = 2 * ntaps - 1;
    a.mb = ntaps;
    a.shift = ntaps - 1;
    const double c0 = fc * t0;
    a.c0 = (float)(c0 - std::floor(c0));
    const double step = fc / fs;
    a.step_hi = (float)step;
    a.step_lo = (float)(step - (double)a.step_hi);
    a.scale = scale;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (src_type) {
        case USTB_SRC_F32: return launch_demod<float, true>((const float*)rf, iq, dst_type, taps, a, s);
        case USTB_SRC_I16: return launch_demod<int16_t, true>((const int16_t*)rf, iq, dst_type, taps, a, s);
        default: return launch_demod<__half, true>((const __half*)rf, iq, dst_type, taps, a, s);
    }
}

// Plain single-precision DAS on precomputed delay/apodization tables — the
// drop-in for the reference's das_c (+mex/source/das_c.cpp:355-409).
//
// One thread per pixel, or with few pixels four warps of a CTA that share the channels of
// 32 pixels (in_parts()).  For the summing modes each thread keeps FC frame
// accumulators in registers and writes every output element exactly once, so
// the output needs no clearing.  Per unit the arithmetic follows das_c step by
// step in single precision, with the same roundings where they decide the
// result: delay = fl(tx + rx), s = fl(fl(delay - t0) * fs), n0 = trunc(s),
// b = s - floor(s), phase = fl(wd * delay).  Only the order of the final sums
// and FMA contraction in the interpolation/rotation differ (a few ulp).
//
// Loop order: for dimension.both/.receive, chunks of WC waves outer (their tx
// values in registers) and channels inner (rx values re-read once per chunk);
// for .transmit/.none, channels outer and wave chunks inner.
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "f32x2.cuh"
#include "phasor.cuh"

namespace {

constexpr int kThreads = 128;
constexpr double kRefPi = 3.14159265359;  // the PI das_c uses for wd (das_c.cpp:33,243)

struct TableArgs {
    const void* ch;
    int64_t L, N, W, F, P, LN, LNW;
    float fs, t0, wd;
    const float* apo_tx;
    const float* apo_rx;
    const float* d_tx;
    const float* d_rx;
    void* out;
    int64_t rx_f, w_f, f_f;
};

// Threads of a CTA that share a pixel's channels (its parts, whole warps) and this thread's
// pixel and part.  A CTA takes kThreads / PARTS pixels; with parts, threads beyond the last
// pixel follow it without storing.
template <int PARTS>
struct Place {
    static constexpr int kPixels = kThreads / PARTS;
    static_assert(kPixels % 32 == 0, "a part is made of whole warps");
    const int part = PARTS > 1 ? threadIdx.x / kPixels : 0, px = threadIdx.x - part * kPixels;
    int64_t p = (int64_t)blockIdx.x * kPixels + px;
    const bool live;
    __device__ explicit Place(const TableArgs& A) : live(p < A.P) {
        if (PARTS > 1 && !live) p = A.P - 1;
    }
};

template <bool CPLX, int FC>
struct Acc {
    float re[FC];
    float im[FC];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int f = 0; f < FC; ++f) re[f] = im[f] = 0.f;
    }
};

template <bool CPLX, int FC>
__device__ __forceinline__ void store(const TableArgs& A, int64_t idx, int64_t f0, int nf,
                                      const Acc<CPLX, FC>& acc) {
#pragma unroll
    for (int f = 0; f < FC; ++f) {
        if (f < nf) {
            const int64_t o = idx + (f0 + f) * A.f_f;
            if (CPLX)
                reinterpret_cast<float2*>(A.out)[o] = make_float2(acc.re[f], acc.im[f]);
            else
                reinterpret_cast<float*>(A.out)[o] = acc.re[f];
        }
    }
}

// Waves are processed in chunks of WC whose tx delay/apodization sit in
// registers; for each channel the WC units of the chunk are independent.  They
// are evaluated branch-free: every unit loads from a safe sample index and an
// invalid or zero-apodization unit's contribution is selected away (not
// multiplied by zero, so non-finite samples behave as in das_c, which skips
// those units).  All WC sample loads are then in flight together.
constexpr int WC = 8;
// At most this many waves run in chunks of channels (das_table_few_waves), where those were
// the faster ones (128 channels, 200 x 200 pixels, chunks of waves against chunks of
// channels, us; real data crosses at the same counts):
//   both      1 wave 75 / 42, 2 waves 71 / 61, 3 waves 72 / 87
//   receive   1 wave 65 / 27, 3 waves 73 / 69, 4 waves 75 / 91
//   transmit  1 wave 99 / 35, 5 waves 116 / 96, 8 waves 133 / 141
constexpr int few_waves(int mode) { return mode == USTB_DIM_BOTH ? 2 : mode == USTB_DIM_RECEIVE ? 3 : 5; }

// A table value that is read once per wave chunk: kept out of L1 so that it does not
// evict the channel-data lines the sample gathers reuse.
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
    return v;
}

// das_c's n0 = (int)s and floor(s) (das_c.cpp:381-383).  For traces of at most 2^23
// samples the integer part comes from adding 2^23 with round-toward-zero: it equals
// (int)s for 0 <= s < 2^23, and negative, too large, NaN or infinite s give indices
// outside (0, L - 1), so those units stay invalid as in das_c; for the valid units
// (s >= 1) floor(s) = (int)s and the fraction s - floor(s) is the same float.
// Longer traces use the conversion instructions.
template <bool MAGIC>
__device__ __forceinline__ int trunc_floor(float s, float& fl) {
    if constexpr (MAGIC) {
        const float t = __fadd_rz(s, 8388608.0f);
        fl = __fsub_rn(t, 8388608.0f);
        return __float_as_int(t) - 0x4B000000;
    } else {
        fl = floorf(s);
        return __float2int_rz(s);
    }
}

// Prefetch into L1 the sample lines of one channel's WC units, so that their loads a
// channel later hit L1 instead of waiting on L2 (same index arithmetic as chunk_units).
template <bool CPLX, typename IDX, bool MAGIC>
__device__ __forceinline__ void prefetch_units(const TableArgs& A, IDX nL, const IDX* wbase, int wc, const float* txd,
                                               float rxd, float rxa) {
    if (rxa == 0.0f) return;
    const int Lm1 = (int)(A.L - 1);
#pragma unroll
    for (int k = 0; k < WC; ++k) {
        const float denay = __fmul_rn(__fsub_rn(__fadd_rn(txd[k], rxd), A.t0), A.fs);
        float fl;
        const int n0 = trunc_floor<MAGIC>(denay, fl);
        if (k < wc && n0 > 0 && n0 < Lm1) {
            const char* x = reinterpret_cast<const char*>(A.ch) + (size_t)(nL + wbase[k] + (IDX)n0) * (CPLX ? 8 : 4);
            asm volatile("prefetch.global.L1 [%0];\n" ::"l"(x));
        }
    }
}

// IDX: int32_t when every sample index of the call fits 31 bits, else int64_t.
// pf: also prefetch into L1 the next channel's sample line of each unit, at this unit's
// sample index shifted by dn, the receive-delay step to the next channel in samples
// (clamped into the trace; only where the lines are, not which units are valid).
// PACK: the position and phase arithmetic of two units per instruction.  2 % faster for
// complex chunks of waves (IQ compounding 1.240 -> 1.197 ms) and chunks of channels (one
// wave, receive kept: 32 -> 26 us); slower where chunks of waves are inner (real RF, 16
// waves, channels kept: 185 -> 205 us), so not used there.
template <bool CPLX, int FC, bool PER_WAVE, int NACC, typename IDX, bool MAGIC, bool PACK>
__device__ __forceinline__ void chunk_units(const TableArgs& A, IDX nL, const IDX* wbase, int wc, int64_t f0,
                                            int nf, const float* txd, const float* txa, float rxd, float rxa,
                                            Acc<CPLX, FC>* acc, bool pf = false, int dn = 0, IDX ahead = 0) {
    float a[WC], b[WC], wr[WC], wi[WC];
    IDX base[WC];
    bool ok[WC];
    const int Lm1 = (int)(A.L - 1);
    auto place = [&](int k, int n0) {  // validity, prefetch and sample offset of unit k
        ok[k] = k < wc && txa[k] != 0.0f && rxa != 0.0f && n0 > 0 && n0 < Lm1;
        if (pf && k < wc) {
            const int m = min(max(n0 + dn, 1), Lm1 - 1);
            const char* x = reinterpret_cast<const char*>(A.ch) +
                            (size_t)(nL + ahead + wbase[k] + (IDX)m) * (CPLX ? 8 : 4);
            asm volatile("prefetch.global.L1 [%0];\n" ::"l"(x));
        }
        base[k] = nL + wbase[k] + (IDX)(ok[k] ? n0 : 1);
    };
    if constexpr (PACK && MAGIC) {
        using namespace ustb;
        const f32x2 rxd2 = pack2(rxd, rxd), rxa2 = pack2(rxa, rxa), magic = pack2(8388608.0f, 8388608.0f);
#pragma unroll
        for (int k = 0; k < WC; k += 2) {
            const f32x2 delay = add2(pack2(txd[k], txd[k + 1]), rxd2);
            const f32x2 apo = mul2(pack2(txa[k], txa[k + 1]), rxa2);
            const f32x2 denay = mul2(sub2(delay, pack2(A.t0, A.t0)), pack2(A.fs, A.fs));
            const f32x2 t = add2_rz(denay, magic);  // trunc_floor
            const f32x2 bb = sub2(denay, sub2(t, magic));
            const float2 tt = unpack2(t), b2 = unpack2(bb), a2 = unpack2(sub2(pack2(1.0f, 1.0f), bb));
            place(k, __float_as_int(tt.x) - 0x4B000000);
            place(k + 1, __float_as_int(tt.y) - 0x4B000000);
            b[k] = b2.x; b[k + 1] = b2.y;
            a[k] = a2.x; a[k + 1] = a2.y;
            float2 w0 = unpack2(apo), w1 = make_float2(0.f, 0.f);
            if (CPLX) {
                float2 c, sn;
                expi_reduced2(mul2(pack2(A.wd, A.wd), delay), c, sn);
                w1 = unpack2(mul2(pack2(sn.x, sn.y), apo));
                w0 = unpack2(mul2(pack2(c.x, c.y), apo));
            }
            wr[k] = w0.x; wr[k + 1] = w0.y;
            wi[k] = w1.x; wi[k + 1] = w1.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < WC; ++k) {
            const float delay = __fadd_rn(txd[k], rxd);
            const float apo = __fmul_rn(txa[k], rxa);
            const float denay = __fmul_rn(__fsub_rn(delay, A.t0), A.fs);
            float fl;
            place(k, trunc_floor<MAGIC>(denay, fl));
            b[k] = __fsub_rn(denay, fl);
            a[k] = __fsub_rn(1.0f, b[k]);
            if (CPLX) {
                float c, s;
                ustb::expi_reduced(__fmul_rn(A.wd, delay), c, s);
                wr[k] = c * apo;
                wi[k] = s * apo;
            } else {
                wr[k] = apo;
                wi[k] = 0.f;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < FC; ++f) {
        if (f >= nf) continue;
#pragma unroll
        for (int k = 0; k < WC; ++k) {
            Acc<CPLX, FC>& ac = acc[PER_WAVE ? k : 0];
            if (CPLX) {
                const float2* x = reinterpret_cast<const float2*>(A.ch) + base[k] + f * A.LNW;
                const float2 x0 = __ldg(x), x1 = __ldg(x + 1);
                const float vr = fmaf(b[k], x1.x, a[k] * x0.x);
                const float vi = fmaf(b[k], x1.y, a[k] * x0.y);
                const float nr = fmaf(wr[k], vr, fmaf(-wi[k], vi, ac.re[f]));
                const float ni = fmaf(wr[k], vi, fmaf(wi[k], vr, ac.im[f]));
                ac.re[f] = ok[k] ? nr : ac.re[f];
                ac.im[f] = ok[k] ? ni : ac.im[f];
            } else {
                const float* x = reinterpret_cast<const float*>(A.ch) + base[k] + f * A.LNW;
                const float x0 = __ldg(x), x1 = __ldg(x + 1);
                const float nr = fmaf(wr[k], fmaf(b[k], x1, a[k] * x0), ac.re[f]);
                ac.re[f] = ok[k] ? nr : ac.re[f];
            }
        }
    }
}

// The index half of one channel's WC units (dimension both / receive): das_c's delay,
// the sample index and fraction, and which units are valid.  Formed one channel
// ahead, so that the same arithmetic also prefetches the channel's sample lines into
// L1, and carried to the next iteration, where unit_sum adds the units.
template <typename IDX>
struct UnitIdx {
    float delay[WC], b[WC];
    IDX base[WC];
    unsigned ok;  // bit k: unit k valid (k < wc, nonzero weights, 0 < n0 < L - 1)
};

template <bool CPLX, typename IDX, bool MAGIC>
__device__ __forceinline__ void unit_index(const TableArgs& A, IDX nL, const IDX* wbase, int wc, const float* txd,
                                           const float* txa, float rxd, float rxa, bool prefetch, UnitIdx<IDX>& u) {
    const unsigned Lm2 = (unsigned)(A.L - 2);  // L >= 3 here (the host zero-fills shorter traces)
    u.ok = 0u;
#pragma unroll
    for (int k = 0; k < WC; ++k) {
        const float delay = __fadd_rn(txd[k], rxd);
        const float denay = __fmul_rn(__fsub_rn(delay, A.t0), A.fs);
        float fl;
        const int n0 = trunc_floor<MAGIC>(denay, fl);
        const bool ok = k < wc && txa[k] != 0.0f && rxa != 0.0f && (unsigned)(n0 - 1) < Lm2;
        u.delay[k] = delay;
        u.b[k] = __fsub_rn(denay, fl);
        u.base[k] = nL + wbase[k] + (IDX)(ok ? n0 : 1);
        u.ok |= ok ? (1u << k) : 0u;
        if (prefetch && ok) {
            const char* x = reinterpret_cast<const char*>(A.ch) + (size_t)u.base[k] * (CPLX ? 8 : 4);
            asm volatile("prefetch.global.L1 [%0];\n" ::"l"(x));
        }
    }
}

template <bool CPLX, int FC, bool PER_WAVE, typename IDX>
__device__ __forceinline__ void unit_sum(const TableArgs& A, const UnitIdx<IDX>& u, const float* txa, float rxa,
                                         int nf, Acc<CPLX, FC>* acc) {
#pragma unroll
    for (int k = 0; k < WC; ++k) {
        const bool ok = (u.ok >> k) & 1u;
        const float apo = __fmul_rn(txa[k], rxa);
        const float b = u.b[k], a = __fsub_rn(1.0f, b);
        float wr = apo, wi = 0.f;
        if (CPLX) {
            float c, sn;
            ustb::expi_reduced(__fmul_rn(A.wd, u.delay[k]), c, sn);
            wr = c * apo;
            wi = sn * apo;
        }
#pragma unroll
        for (int f = 0; f < FC; ++f) {
            if (f >= nf) continue;
            Acc<CPLX, FC>& ac = acc[PER_WAVE ? k : 0];
            if (CPLX) {
                const float2* x = reinterpret_cast<const float2*>(A.ch) + u.base[k] + f * A.LNW;
                const float2 x0 = __ldg(x), x1 = __ldg(x + 1);
                const float vr = fmaf(b, x1.x, a * x0.x);
                const float vi = fmaf(b, x1.y, a * x0.y);
                const float nr = fmaf(wr, vr, fmaf(-wi, vi, ac.re[f]));
                const float ni = fmaf(wr, vi, fmaf(wi, vr, ac.im[f]));
                ac.re[f] = ok ? nr : ac.re[f];
                ac.im[f] = ok ? ni : ac.im[f];
            } else {
                const float* x = reinterpret_cast<const float*>(A.ch) + u.base[k] + f * A.LNW;
                const float x0 = __ldg(x), x1 = __ldg(x + 1);
                const float nr = fmaf(wr, fmaf(b, x1, a * x0), ac.re[f]);
                ac.re[f] = ok ? nr : ac.re[f];
            }
        }
    }
}

// The parts' sums, added in order in part 0 (every thread of the CTA calls).
template <bool CPLX, int FC, int PARTS>
__device__ __forceinline__ void sum_parts(const Place<PARTS>& q, Acc<CPLX, FC>& acc) {
    if constexpr (PARTS > 1) {
        __shared__ float2 sums[FC][kThreads];
        __syncthreads();
#pragma unroll
        for (int f = 0; f < FC; ++f) sums[f][threadIdx.x] = make_float2(acc.re[f], acc.im[f]);
        __syncthreads();
        if (q.part != 0) return;
#pragma unroll
        for (int k = 1; k < PARTS; ++k)
#pragma unroll
            for (int f = 0; f < FC; ++f) {
                const float2 v = sums[f][k * Place<PARTS>::kPixels + q.px];
                acc.re[f] += v.x;
                acc.im[f] += v.y;
            }
    }
}

// Real data: at most 80 registers (6 CTAs of 128 threads per SM), with the carried unit
// indices; complex data: the phase of every unit needs more registers.
template <int MODE, bool CPLX, int FC, typename IDX, bool MAGIC, int PARTS>
__global__ void __launch_bounds__(kThreads, (CPLX ? 1 : 6)) das_table_kernel(const TableArgs A) {
    const Place<PARTS> q(A);
    if (PARTS == 1 && !q.live) return;
    const int64_t p = q.p, P = A.P;
    const bool stores = PARTS == 1 || (q.live && q.part == 0);
    constexpr bool PER_WAVE = (MODE == USTB_DIM_RECEIVE || MODE == USTB_DIM_NONE);
    constexpr int NACC = PER_WAVE ? WC : 1;
    Acc<CPLX, FC> acc[NACC];
    float txd[WC], txa[WC];
    auto load_tx = [&](int64_t w0, int wc) {
#pragma unroll
        for (int k = 0; k < WC; ++k) {
            txa[k] = k < wc ? __ldg(A.apo_tx + P * (w0 + k) + p) : 0.f;
            txd[k] = k < wc ? __ldg(A.d_tx + P * (w0 + k) + p) : 0.f;
        }
    };
    for (int64_t f0 = 0; f0 < A.F; f0 += FC) {
        const int nf = (int)min((int64_t)FC, A.F - f0);
        if (MODE == USTB_DIM_RECEIVE || MODE == USTB_DIM_BOTH) {
            if (MODE == USTB_DIM_BOTH) acc[0].zero();
            // the warp's channels with a nonzero receive weight lie in [nlo, nhi]: one scan
            // of the apodization column, so that every wave chunk reads the receive tables
            // of those channels only (the others are skipped per unit anyway)
            int nlo = (int)A.N, nhi = -1;
            if constexpr (PARTS == 1) {
                for (int n = 0; n < (int)A.N; ++n)
                    if (ld_stream(A.apo_rx + P * n + p) != 0.0f) {
                        nlo = min(nlo, n);
                        nhi = n;
                    }
                const unsigned live = __activemask();
                nlo = __reduce_min_sync(live, nlo);
                nhi = __reduce_max_sync(live, nhi);
            } else {  // a part scans its share of the column, eight loads in flight
                const int per = ((int)A.N + PARTS - 1) / PARTS, end = min((q.part + 1) * per, (int)A.N);
                for (int n0 = q.part * per; n0 < end; n0 += 8) {
                    float a[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i] = n0 + i < end ? ld_stream(A.apo_rx + P * (n0 + i) + p) : 0.f;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (a[i] != 0.0f) {
                            nlo = min(nlo, n0 + i);
                            nhi = n0 + i;
                        }
                }
                nlo = __reduce_min_sync(0xffffffffu, nlo);
                nhi = __reduce_max_sync(0xffffffffu, nhi);
                __shared__ int lo[kThreads / 32], hi[kThreads / 32];
                __syncthreads();
                if ((threadIdx.x & 31) == 0) {
                    lo[threadIdx.x / 32] = nlo;
                    hi[threadIdx.x / 32] = nhi;
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < kThreads / 32; ++i) {
                    nlo = min(nlo, lo[i]);
                    nhi = max(nhi, hi[i]);
                }
                // every PARTS-th channel: the weights of a part's channels end alike, and
                // two-dimensional apertures have gaps (equal ranges of channels: 191 real
                // channels x 191 waves 3.01 ms, this 1.87)
                nlo += q.part;
            }
            for (int64_t w0 = 0; w0 < A.W; w0 += WC) {
                const int wc = (int)min((int64_t)WC, A.W - w0);
                load_tx(w0, wc);
                IDX wbase[WC];
#pragma unroll
                for (int k = 0; k < WC; ++k) wbase[k] = (IDX)(A.LN * (w0 + (k < wc ? k : 0)) + f0 * A.LNW);
                if (MODE == USTB_DIM_RECEIVE)
#pragma unroll
                    for (int k = 0; k < WC; ++k) acc[k].zero();
                // receive values are loaded two channels ahead and the next channel's
                // sample lines prefetched into L1 while this channel is computed
                // (no receive weight in this warp: nhi < nlo, the loop below runs no channel)
                const int64_t step = P * PARTS;
                const float* pa = A.apo_rx + P * max(nlo, 0) + p;
                const float* pd = A.d_rx + P * max(nlo, 0) + p;
                float rxa1 = 0.f, rxd1 = 0.f, rxa2 = 0.f, rxd2 = 0.f;
                if (nlo <= nhi) {
                    rxa1 = ld_stream(pa);
                    rxd1 = ld_stream(pd);
                }
                if (nlo + PARTS <= nhi) {
                    rxa2 = ld_stream(pa + step);
                    rxd2 = ld_stream(pd + step);
                }
                pa += 2 * step;
                pd += 2 * step;
                const IDX ahead = (IDX)A.L * PARTS;  // to the next channel of this part
                IDX nL = (IDX)A.L * (IDX)nlo;
                if constexpr (CPLX) {
                    // complex: the register count left by the per-unit phase allows no
                    // carried indices; the next channel's lines are prefetched from this
                    // channel's indices shifted by the receive-delay step (the first
                    // channel, and lanes without a weight on this channel, form the next
                    // channel's indices for the prefetch)
                    if (FC == 1 && nlo <= nhi) prefetch_units<CPLX, IDX, MAGIC>(A, nL, wbase, wc, txd, rxd1, rxa1);
                    for (int n = nlo; n <= nhi; n += PARTS, nL += ahead) {
                        const float rxa = rxa1, rxd = rxd1;
                        rxa1 = rxa2;
                        rxd1 = rxd2;
                        if (n + 2 * PARTS <= nhi) {
                            rxa2 = ld_stream(pa);
                            rxd2 = ld_stream(pd);
                            pa += step;
                            pd += step;
                        }
                        const bool pf = FC == 1 && n + PARTS <= nhi && rxa1 != 0.0f;
                        if (rxa == 0.0f) {
                            if (pf) prefetch_units<CPLX, IDX, MAGIC>(A, nL + ahead, wbase, wc, txd, rxd1, rxa1);
                            continue;
                        }
                        const int dn = __float2int_rn(__fmul_rn(__fsub_rn(rxd1, rxd), A.fs));
                        chunk_units<CPLX, FC, PER_WAVE, NACC, IDX, MAGIC, true>(A, nL, wbase, wc, f0, nf, txd, txa, rxd, rxa,
                                                                          acc, pf, dn, ahead);
                    }
                } else {
                // real: the indices formed with the prefetch are carried to the units
                UnitIdx<IDX> cur, nxt;
                if (nlo <= nhi) unit_index<CPLX, IDX, MAGIC>(A, nL, wbase, wc, txd, txa, rxd1, rxa1, FC == 1, cur);
                for (int n = nlo; n <= nhi; n += PARTS, nL += ahead) {
                    const float rxa = rxa1;
                    rxa1 = rxa2;
                    rxd1 = rxd2;
                    if (n + 2 * PARTS <= nhi) {
                        rxa2 = ld_stream(pa);
                        rxd2 = ld_stream(pd);
                        pa += step;
                        pd += step;
                    }
                    if (n + PARTS <= nhi)
                        unit_index<CPLX, IDX, MAGIC>(A, nL + ahead, wbase, wc, txd, txa, rxd1, rxa1, FC == 1, nxt);
                    if (rxa != 0.0f) unit_sum<CPLX, FC, PER_WAVE, IDX>(A, cur, txa, rxa, nf, acc);
                    cur = nxt;
                }
                }
                if (MODE == USTB_DIM_RECEIVE)
#pragma unroll
                    for (int k = 0; k < WC; ++k)
                        if (k < wc) {
                            sum_parts(q, acc[k]);
                            if (stores) store<CPLX, FC>(A, p + A.w_f * (w0 + k), f0, nf, acc[k]);
                        }
            }
            if (MODE == USTB_DIM_BOTH) {
                sum_parts(q, acc[0]);
                if (stores) store<CPLX, FC>(A, p, f0, nf, acc[0]);
            }
        } else if (q.live) {
            for (int64_t n = q.part; n < A.N; n += PARTS) {
                const float rxa = __ldg(A.apo_rx + P * n + p);
                const float rxd = __ldg(A.d_rx + P * n + p);
                if (MODE == USTB_DIM_TRANSMIT) acc[0].zero();
                for (int64_t w0 = 0; w0 < A.W; w0 += WC) {
                    const int wc = (int)min((int64_t)WC, A.W - w0);
                    load_tx(w0, wc);
                    IDX wbase[WC];
#pragma unroll
                    for (int k = 0; k < WC; ++k) wbase[k] = (IDX)(A.LN * (w0 + (k < wc ? k : 0)) + f0 * A.LNW);
                    if (MODE == USTB_DIM_NONE)
#pragma unroll
                        for (int k = 0; k < WC; ++k) acc[k].zero();
                    if (rxa != 0.0f)
                        chunk_units<CPLX, FC, PER_WAVE, NACC, IDX, MAGIC, false>(A, (IDX)(A.L * n), wbase, wc, f0, nf, txd, txa, rxd,
                                                                   rxa, acc);
                    if (MODE == USTB_DIM_NONE)
#pragma unroll
                        for (int k = 0; k < WC; ++k)
                            if (k < wc) store<CPLX, FC>(A, p + A.rx_f * n + A.w_f * (w0 + k), f0, nf, acc[k]);
                }
                if (MODE == USTB_DIM_TRANSMIT) store<CPLX, FC>(A, p + A.rx_f * n, f0, nf, acc[0]);
            }
        }
    }
}

// Few waves: the chunks of WC units run over channels instead, so that a single wave fills
// them too (chunks of waves would evaluate WC units for the one).  The roles of the tables
// are swapped in chunk_units (delays and weights add and multiply in either order): the
// channels' values are the chunk's, the wave's the common one.  The next chunk's receive
// values are loaded a chunk ahead.
template <int MODE, bool CPLX, int FC, typename IDX, bool MAGIC, int PARTS>
__global__ void __launch_bounds__(kThreads) das_table_few_waves(const TableArgs A) {
    const Place<PARTS> q(A);
    if (PARTS == 1 && !q.live) return;
    const int64_t p = q.p, P = A.P;
    const bool stores = PARTS == 1 || (q.live && q.part == 0);
    const int first = q.part * WC;
    constexpr int step = PARTS * WC;  // chunks of channels of this part
    const int N = (int)A.N, W = (int)A.W;
    constexpr bool PER_CHANNEL = (MODE == USTB_DIM_TRANSMIT || MODE == USTB_DIM_NONE);
    Acc<CPLX, FC> acc[PER_CHANNEL ? WC : 1];
    float rxd[WC], rxa[WC];
    IDX nbase[WC];
    auto load_rx = [&](int n0, float* d, float* a) {
#pragma unroll
        for (int k = 0; k < WC; ++k) {
            const bool in = n0 + k < N;
            a[k] = in ? ld_stream(A.apo_rx + P * (n0 + k) + p) : 0.f;
            d[k] = in ? ld_stream(A.d_rx + P * (n0 + k) + p) : 0.f;
        }
    };
    for (int64_t f0 = 0; f0 < A.F; f0 += FC) {
        const int nf = (int)min((int64_t)FC, A.F - f0);
        // one chunk of channels from n0 on with wave w
        auto units = [&](int n0, int w, const float* d, const float* a) {
            const float txd = __ldg(A.d_tx + P * w + p), txa = __ldg(A.apo_tx + P * w + p);
            if (txa == 0.0f) return;
            chunk_units<CPLX, FC, PER_CHANNEL, (PER_CHANNEL ? WC : 1), IDX, MAGIC, true>(
                A, (IDX)(A.LN * w), nbase, min(WC, N - n0), f0, nf, d, a, txd, txa, acc);
        };
        auto chunk = [&](int n0) {
            bool any = false;
#pragma unroll
            for (int k = 0; k < WC; ++k) {
                any |= rxa[k] != 0.0f;
                nbase[k] = (IDX)(A.L * min(n0 + k, N - 1) + f0 * A.LNW);
            }
            return any;
        };
        if (MODE == USTB_DIM_RECEIVE) {
            for (int w = 0; w < W; ++w) {
                acc[0].zero();
                for (int n0 = first; n0 < N; n0 += step) {
                    load_rx(n0, rxd, rxa);
                    if (chunk(n0)) units(n0, w, rxd, rxa);
                }
                sum_parts(q, acc[0]);
                if (stores) store<CPLX, FC>(A, p + A.w_f * w, f0, nf, acc[0]);
            }
        } else if (MODE == USTB_DIM_BOTH) {
            acc[0].zero();
            float d1[WC], a1[WC];
            load_rx(first, d1, a1);
            for (int n0 = first; n0 < N; n0 += step) {
#pragma unroll
                for (int k = 0; k < WC; ++k) {
                    rxd[k] = d1[k];
                    rxa[k] = a1[k];
                }
                load_rx(n0 + step, d1, a1);
                if (!chunk(n0)) continue;
                for (int w = 0; w < W; ++w) units(n0, w, rxd, rxa);
            }
            sum_parts(q, acc[0]);
            if (stores) store<CPLX, FC>(A, p, f0, nf, acc[0]);
        } else if (q.live) {
            for (int n0 = first; n0 < N; n0 += step) {
                load_rx(n0, rxd, rxa);
                const bool any = chunk(n0);
                auto put = [&](int64_t o) {
#pragma unroll
                    for (int k = 0; k < WC; ++k)
                        if (n0 + k < N) store<CPLX, FC>(A, p + A.rx_f * (n0 + k) + o, f0, nf, acc[k]);
                };
#pragma unroll
                for (int k = 0; k < WC; ++k) acc[PER_CHANNEL ? k : 0].zero();
                for (int w = 0; w < W; ++w) {
                    if (any) units(n0, w, rxd, rxa);
                    if (MODE == USTB_DIM_NONE) {
                        put(A.w_f * w);
#pragma unroll
                        for (int k = 0; k < WC; ++k) acc[PER_CHANNEL ? k : 0].zero();
                    }
                }
                if (MODE == USTB_DIM_TRANSMIT) put(0);
            }
        }
    }
}

// Whether the four warps of a CTA share 32 pixels' channels (PARTS 4) instead of taking
// 128 pixels.  Few pixels leave SMs without a CTA or end in a long last round; with many,
// the warps of a CTA no longer read neighbouring pixels' sample lines together.  The line
// lies at the CTAs of 128 pixels per SM; one part / four, us, N channels x W waves:
//   2000 pixels 64 x 16 x 2 frames, complex: both 147 / 44, receive 76 / 29, transmit 100 / 29
//   10,000 pixels 128 x 16: complex both 85 / 34, real 73 / 35
//   80,000 pixels 128 x 16 (4 per SM): complex both 196 / 155, receive 199 / 190, transmit
//     394 / 309; real 149 / 136, 164 / 162, 273 / 206
//   160,000 pixels 128 x 16 (8 per SM): complex both 315 / 293, receive 322 / 372, transmit
//     591 / 569; real 248 / 253, 283 / 311, 476 / 369; 1 wave, transmit, 84 / 83 and 54 / 56
//   160,000 pixels 128 x 75: complex both 1199 / 1079
//   40,000 pixels 64 x 16 x 2 frames (2 per SM): complex receive 70 / 75
//   320,000 pixels 64 x 16: complex both 283 / 314, receive 306 / 442
// Complex both of one frame and one chunk of waves stays in one part where its CTAs nearly
// fill one round (four are resident on an SM; with more frames three, so a second round
// follows): 75,878 pixels (3.9 per SM) 128 x 4 57 / 62, 128 x 8 61 / 66, 40 x 4 39 / 43, but
// 128 x 12 107 / 102, 128 x 8 x 2 frames 172 / 138; 60,314 pixels (3.1) 128 x 4 58 / 49;
// 40,858 (2.1) 52 / 36, 128 x 12 99 / 60; a volume's 57,200 pixels, 529 channels x 4 waves,
// 480 / 458.
// A part needs channels of its own (chunks of WC).
int in_parts(int mode, bool cplx, const TableArgs& A, bool& parts) {
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool few = A.W <= few_waves(mode);
    const int64_t per_sm = mode == USTB_DIM_RECEIVE && !few                                             ? 2
                           : (mode == USTB_DIM_BOTH && cplx) || (mode == USTB_DIM_TRANSMIT && !few) ? 9
                                                                                                        : 5;
    const int64_t ctas = (A.P + kThreads - 1) / kThreads;
    const bool one_round = mode == USTB_DIM_BOTH && cplx && !few && A.F == 1 && A.W <= WC && 2 * ctas > 7 * sms && ctas <= 4 * sms;
    parts = A.N >= 4 * WC && ctas <= per_sm * sms && !one_round;
    return USTB_OK;
}

template <int MODE, bool CPLX, typename IDX, bool MAGIC>
int launch_idx(const TableArgs& A, cudaStream_t s) {
    auto start = [&](auto fc, auto parts) {
        constexpr int FC = decltype(fc)::value, PARTS = decltype(parts)::value, per = kThreads / PARTS;
        const unsigned grid = (unsigned)((A.P + per - 1) / per);
        if (A.W <= few_waves(MODE)) das_table_few_waves<MODE, CPLX, FC, IDX, MAGIC, PARTS><<<grid, kThreads, 0, s>>>(A);
        else das_table_kernel<MODE, CPLX, FC, IDX, MAGIC, PARTS><<<grid, kThreads, 0, s>>>(A);
    };
    auto frames = [&](auto parts) {
        if (A.F == 1) start(std::integral_constant<int, 1>{}, parts);
        else if (A.F == 2) start(std::integral_constant<int, 2>{}, parts);
        else start(std::integral_constant<int, 4>{}, parts);
    };
    if constexpr (sizeof(IDX) == 4 && MAGIC) {  // the others are for data of gigabytes
        bool parts = false;
        const int rc = in_parts(MODE, CPLX, A, parts);
        if (rc) return rc;
        if (parts) {
            frames(std::integral_constant<int, 4>{});
            return USTB_OK;
        }
    }
    frames(std::integral_constant<int, 1>{});
    return USTB_OK;
}

// 32-bit sample indices when every index of the call (and one past it) fits 31 bits;
// the float trick of trunc_floor for traces of at most 2^23 samples
template <int MODE, bool CPLX>
int launch_fc(const TableArgs& A, cudaStream_t s) {
    const bool short_traces = A.L <= ((int64_t)1 << 23);
    if (A.LNW * A.F < (int64_t)INT32_MAX - 1 && short_traces)
        return launch_idx<MODE, CPLX, int32_t, true>(A, s);
    if (short_traces) return launch_idx<MODE, CPLX, int64_t, true>(A, s);
    return launch_idx<MODE, CPLX, int64_t, false>(A, s);
}

template <bool CPLX>
int launch_mode(int dim, const TableArgs& A, cudaStream_t s) {
    switch (dim) {
        case USTB_DIM_NONE: return launch_fc<USTB_DIM_NONE, CPLX>(A, s);
        case USTB_DIM_RECEIVE: return launch_fc<USTB_DIM_RECEIVE, CPLX>(A, s);
        case USTB_DIM_TRANSMIT: return launch_fc<USTB_DIM_TRANSMIT, CPLX>(A, s);
        default: return launch_fc<USTB_DIM_BOTH, CPLX>(A, s);
    }
}

int check_table_args(const void* ch, int32_t ch_complex, int64_t L, int64_t N, int64_t W, int64_t F,
                     float fd, int32_t dim, const void* apo_tx, const void* apo_rx,
                     const void* delay_tx, const void* delay_rx, int64_t P, const void* out) {
    USTB_REQUIRE(dim >= 0 && dim <= 3, USTB_E_ARG,
                 "Unknown sum mode %d. Available: 0 -> NONE, 1->RX, 2->TX, 3->BOTH", (int)dim);
    USTB_REQUIRE(L >= 0 && N >= 0 && W >= 0 && F >= 0 && P >= 0, USTB_E_SHAPE,
                 "negative size (L=%lld N=%lld W=%lld F=%lld P=%lld)", (long long)L, (long long)N,
                 (long long)W, (long long)F, (long long)P);
    USTB_REQUIRE(ch_complex == 0 || ch_complex == 1, USTB_E_ARG, "ch_complex must be 0 or 1");
    USTB_REQUIRE(ch_complex || !(fabsf(fd) > 1e-6f), USTB_E_DTYPE,
                 "The modulation frequency > 0 but the input data is real. Check inputs.");
    USTB_REQUIRE(L <= INT32_MAX, USTB_E_SHAPE, "L=%lld exceeds the 32-bit sample index", (long long)L);
    const bool empty_in = L == 0 || N == 0 || W == 0 || F == 0;
    USTB_REQUIRE(empty_in || ch, USTB_E_ARG, "channel data pointer is NULL");
    USTB_REQUIRE(P == 0 || (apo_tx && apo_rx && delay_tx && delay_rx), USTB_E_ARG,
                 "a delay/apodization table pointer is NULL");
    USTB_REQUIRE(out_elems(dim, P, N, W, F) == 0 || out, USTB_E_ARG, "output pointer is NULL");
    return USTB_OK;
}

// Byte counts of the host-pointer entries' device copies: channel data, one tx
// table, one rx table and the output.  Every product is checked for overflow, so
// a request whose sizes wrap 64 bits is rejected instead of under-allocated.
struct StagingBytes {
    size_t ch, tx, rx, out, total;
};

int staging_bytes(int32_t ch_complex, int64_t L, int64_t N, int64_t W, int64_t F, int64_t P, int32_t dim,
                  StagingBytes& b) {
    const uint64_t el = ch_complex ? 8 : 4;
    uint64_t ch = 0, tx = 0, rx = 0, out = 0, t = 0;
    const int64_t nk = (dim == USTB_DIM_NONE || dim == USTB_DIM_TRANSMIT) ? N : 1;
    const int64_t wk = (dim == USTB_DIM_NONE || dim == USTB_DIM_RECEIVE) ? W : 1;
    bool bad = __builtin_mul_overflow((uint64_t)L, (uint64_t)N, &t) || __builtin_mul_overflow(t, (uint64_t)W, &t) ||
               __builtin_mul_overflow(t, (uint64_t)F, &t) || __builtin_mul_overflow(t, el, &ch);
    bad = bad || __builtin_mul_overflow((uint64_t)P, (uint64_t)W, &t) || __builtin_mul_overflow(t, (uint64_t)4, &tx);
    bad = bad || __builtin_mul_overflow((uint64_t)P, (uint64_t)N, &t) || __builtin_mul_overflow(t, (uint64_t)4, &rx);
    bad = bad || __builtin_mul_overflow((uint64_t)P, (uint64_t)nk, &t) || __builtin_mul_overflow(t, (uint64_t)wk, &t) ||
          __builtin_mul_overflow(t, (uint64_t)F, &t) || __builtin_mul_overflow(t, el, &out);
    // each part is padded to 256 bytes; the sum of six padded parts must not wrap either
    const uint64_t lim = (UINT64_MAX >> 4) - 256;
    bad = bad || ch > lim || tx > lim || rx > lim || out > lim;
    USTB_REQUIRE(!bad, USTB_E_SHAPE, "the request's byte counts overflow 64 bits (L=%lld N=%lld W=%lld F=%lld P=%lld)",
                 (long long)L, (long long)N, (long long)W, (long long)F, (long long)P);
    auto align = [](uint64_t v) { return (v + 255) & ~uint64_t(255); };
    b.ch = (size_t)ch;
    b.tx = (size_t)tx;
    b.rx = (size_t)rx;
    b.out = (size_t)out;
    b.total = (size_t)(align(ch) + 2 * align(tx) + 2 * align(rx) + align(out));
    return USTB_OK;
}

// Makes `device` current for the lifetime of the guard and then restores the
// caller's current device, so the host-pointer entries leave the calling thread's
// CUDA state as they found it.
class DeviceGuard {
public:
    int enter(int device) {
        USTB_CUDA(cudaGetDevice(&prev_));
        if (prev_ != device) {
            USTB_CUDA(cudaSetDevice(device));
            restore_ = true;
        }
        return USTB_OK;
    }
    ~DeviceGuard() {
        if (restore_) (void)cudaSetDevice(prev_);
    }

private:
    int prev_ = 0;
    bool restore_ = false;
};

}  // namespace

extern "C" int ustb_das_table_f32(const void* ch, int32_t ch_complex, int64_t L, int64_t N,
                                  int64_t W, int64_t F, float fs, float t0, const float* apo_tx,
                                  const float* apo_rx, const float* delay_tx,
                                  const float* delay_rx, int64_t P, float fd, int32_t dimension,
                                  void* out, void* stream) {
    ustb::clear_error();
    int rc = check_table_args(ch, ch_complex, L, N, W, F, fd, dimension, apo_tx, apo_rx, delay_tx,
                              delay_rx, P, out);
    if (rc) return rc;
    const int64_t n_out = out_elems(dimension, P, N, W, F);
    if (n_out == 0) return USTB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (L < 3 || N == 0 || W == 0) {
        // nothing to sum (a valid unit needs 0 < n0 < L - 1): das_c returns its
        // zero-initialised output
        USTB_CUDA(cudaMemsetAsync(out, 0, (size_t)n_out * (ch_complex ? 8 : 4), s));
        return USTB_OK;
    }
    TableArgs A;
    A.ch = ch;
    A.L = L; A.N = N; A.W = W; A.F = F; A.P = P;
    A.LN = L * N; A.LNW = L * N * W;
    A.fs = fs; A.t0 = t0;
    A.wd = 0.0f;
    if (fabsf(fd) > 1e-6f) A.wd = 2 * (float)kRefPi * fd;
    A.apo_tx = apo_tx; A.apo_rx = apo_rx; A.d_tx = delay_tx; A.d_rx = delay_rx;
    A.out = out;
    const OutStrides os = out_strides(dimension, P, N, W);
    A.rx_f = os.rx_f; A.w_f = os.w_f; A.f_f = os.f_f;
    rc = ch_complex ? launch_mode<true>(dimension, A, s) : launch_mode<false>(dimension, A, s);
    if (rc) return rc;
    USTB_CUDA(cudaGetLastError());
    return USTB_OK;
}

extern "C" int ustb_das_table_f32_host(const void* ch, int32_t ch_complex, int64_t L, int64_t N,
                                       int64_t W, int64_t F, float fs, float t0,
                                       const float* apo_tx, const float* apo_rx,
                                       const float* delay_tx, const float* delay_rx, int64_t P,
                                       float fd, int32_t dimension, void* out, int32_t device) {
    ustb::clear_error();
    int rc = check_table_args(ch, ch_complex, L, N, W, F, fd, dimension, apo_tx, apo_rx, delay_tx,
                              delay_rx, P, out);
    if (rc) return rc;
    StagingBytes sb;
    rc = staging_bytes(ch_complex, L, N, W, F, P, dimension, sb);
    if (rc) return rc;
    DeviceGuard dg;
    rc = dg.enter(device);
    if (rc) return rc;
    const size_t ch_bytes = sb.ch, tx_bytes = sb.tx, rx_bytes = sb.rx, out_bytes = sb.out, total = sb.total;
    cudaStream_t s;
    USTB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    char* buf = nullptr;
    auto align = [](size_t v) { return (v + 255) & ~size_t(255); };
    cudaError_t e = cudaMallocAsync((void**)&buf, total ? total : 256, s);
    if (e != cudaSuccess) {
        cudaStreamDestroy(s);
        return ustb::cuda_fail(e, "cudaMallocAsync", __FILE__, __LINE__);
    }
    char* p = buf;
    void* d_ch = p; p += align(ch_bytes);
    float* d_atx = (float*)p; p += align(tx_bytes);
    float* d_dtx = (float*)p; p += align(tx_bytes);
    float* d_arx = (float*)p; p += align(rx_bytes);
    float* d_drx = (float*)p; p += align(rx_bytes);
    void* d_out = p;
    rc = USTB_OK;
    do {
        if (ch_bytes && (e = cudaMemcpyAsync(d_ch, ch, ch_bytes, cudaMemcpyHostToDevice, s))) break;
        if (tx_bytes && (e = cudaMemcpyAsync(d_atx, apo_tx, tx_bytes, cudaMemcpyHostToDevice, s))) break;
        if (tx_bytes && (e = cudaMemcpyAsync(d_dtx, delay_tx, tx_bytes, cudaMemcpyHostToDevice, s))) break;
        if (rx_bytes && (e = cudaMemcpyAsync(d_arx, apo_rx, rx_bytes, cudaMemcpyHostToDevice, s))) break;
        if (rx_bytes && (e = cudaMemcpyAsync(d_drx, delay_rx, rx_bytes, cudaMemcpyHostToDevice, s))) break;
        rc = ustb_das_table_f32(d_ch, ch_complex, L, N, W, F, fs, t0, d_atx, d_arx, d_dtx, d_drx, P,
                                fd, dimension, d_out, s);
        if (rc) break;
        if (out_bytes && (e = cudaMemcpyAsync(out, d_out, out_bytes, cudaMemcpyDeviceToHost, s))) break;
        e = cudaStreamSynchronize(s);
    } while (0);
    cudaFreeAsync(buf, s);
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    if (rc) return rc;
    if (e != cudaSuccess) return ustb::cuda_fail(e, "host-pointer DAS copy/sync", __FILE__, __LINE__);
    return USTB_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free form of the host-pointer entry point.
//
// Staging buffers live in one file-scope device array instead of memory from
// cudaMalloc.  Host code may not use the array's name as a device address, so
// its address is looked up once per device with cudaGetSymbolAddress (with that
// device current) and cached.  All calls share the array.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[USTB_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};

// The scratch array's device address on the current device `device`.
int noalloc_scratch(int device, void** out) {
    USTB_REQUIRE(device >= 0 && device < kMaxDevices, USTB_E_ARG, "device %d out of range", device);
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[device]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return ustb::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
        g_noalloc_ptr[device] = p;
    }
    *out = g_noalloc_ptr[device];
    return USTB_OK;
}

}  // namespace

extern "C" int ustb_das_table_f32_host_noalloc(const void* ch, int32_t ch_complex, int64_t L, int64_t N,
                                               int64_t W, int64_t F, float fs, float t0,
                                               const float* apo_tx, const float* apo_rx,
                                               const float* delay_tx, const float* delay_rx, int64_t P,
                                               float fd, int32_t dimension, void* out, int32_t device) {
    ustb::clear_error();
    int rc = check_table_args(ch, ch_complex, L, N, W, F, fd, dimension, apo_tx, apo_rx, delay_tx,
                              delay_rx, P, out);
    if (rc) return rc;
    StagingBytes sb;
    rc = staging_bytes(ch_complex, L, N, W, F, P, dimension, sb);
    if (rc) return rc;
    const size_t ch_bytes = sb.ch, tx_bytes = sb.tx, rx_bytes = sb.rx, out_bytes = sb.out, total = sb.total;
    auto align = [](size_t v) { return (v + 255) & ~size_t(255); };
    USTB_REQUIRE(total <= (size_t)USTB_NOALLOC_SCRATCH_BYTES, USTB_E_SHAPE,
                 "this request needs %zu bytes of device scratch; the allocation-free entry point has "
                 "%zu (USTB_NOALLOC_SCRATCH_BYTES): use ustb_das_table_f32_host or split the pixels",
                 total, (size_t)USTB_NOALLOC_SCRATCH_BYTES);
    DeviceGuard dg;
    rc = dg.enter(device);
    if (rc) return rc;
    void* scratch = nullptr;
    rc = noalloc_scratch(device, &scratch);
    if (rc) return rc;
    char* p = static_cast<char*>(scratch);
    void* d_ch = p; p += align(ch_bytes);
    float* d_atx = (float*)p; p += align(tx_bytes);
    float* d_dtx = (float*)p; p += align(tx_bytes);
    float* d_arx = (float*)p; p += align(rx_bytes);
    float* d_drx = (float*)p; p += align(rx_bytes);
    void* d_out = p;
    // Every staged byte is overwritten below and the kernel writes every output
    // element, so nothing in the shared array needs clearing between calls.
    cudaStream_t s = cudaStreamPerThread;
    if (ch_bytes) USTB_CUDA(cudaMemcpyAsync(d_ch, ch, ch_bytes, cudaMemcpyHostToDevice, s));
    if (tx_bytes) USTB_CUDA(cudaMemcpyAsync(d_atx, apo_tx, tx_bytes, cudaMemcpyHostToDevice, s));
    if (tx_bytes) USTB_CUDA(cudaMemcpyAsync(d_dtx, delay_tx, tx_bytes, cudaMemcpyHostToDevice, s));
    if (rx_bytes) USTB_CUDA(cudaMemcpyAsync(d_arx, apo_rx, rx_bytes, cudaMemcpyHostToDevice, s));
    if (rx_bytes) USTB_CUDA(cudaMemcpyAsync(d_drx, delay_rx, rx_bytes, cudaMemcpyHostToDevice, s));
    rc = ustb_das_table_f32(d_ch, ch_complex, L, N, W, F, fs, t0, d_atx, d_arx, d_dtx, d_drx, P, fd,
                            dimension, d_out, s);
    if (rc) return rc;
    if (out_bytes) USTB_CUDA(cudaMemcpyAsync(out, d_out, out_bytes, cudaMemcpyDeviceToHost, s));
    USTB_CUDA(cudaStreamSynchronize(s));
    return USTB_OK;
}

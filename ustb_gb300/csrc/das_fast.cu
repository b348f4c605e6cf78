// Host side of the fast path: the entries pass, request validation and the C entries.
// The beamforming kernels are in das_fast_kernel.cuh.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "das_fast.cuh"

int ustb::ctas_per_sm(size_t smem, int& n) {
    int dev = 0, per_sm = 0, reserved = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    USTB_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
    constexpr size_t kStatic = 512;  // the kernels' static shared memory at most
    n = 2 * (smem + kStatic + (size_t)reserved) <= (size_t)per_sm ? 2 : 1;
    return USTB_OK;
}

namespace {

using ustb::kMaxBatch;
using ustb::Params;

struct WinCoeffs {
    float r1, a, e, b, c, d;  // see the windows in das_fast_kernel.cuh
};

static WinCoeffs window_coeffs(int win) {
    const float twopi = 6.283185307179586f;
    switch (win) {
        case USTB_WIN_BOXCAR: return {0.5f, 0.f, 0.f, 0.f, 0.f, 0.f};
        case USTB_WIN_HANNING: return {-1.f, 0.5f, 0.f, 0.5f, twopi, 0.f};
        case USTB_WIN_HAMMING: return {-1.f, 0.53836f, 0.f, 0.46164f, twopi, 0.f};
        case USTB_WIN_TUKEY25: return {0.375f, 0.5f, 0.f, 0.5f, twopi / 0.25f, 0.625f};
        case USTB_WIN_TUKEY50: return {0.25f, 0.5f, 0.f, 0.5f, twopi / 0.5f, 0.75f};
        case USTB_WIN_TUKEY75: return {0.125f, 0.5f, 0.f, 0.5f, twopi / 0.75f, 0.875f};
        case USTB_WIN_TRIANGLE: return {-1.f, 1.f, -2.f, 0.f, 0.f, 0.f};
        default: return {3.4e38f, 0.f, 0.f, 0.f, 0.f, 0.f};  // none: 1 everywhere
    }
}

// The stage shape a request runs with: ustb_das_geometry.stage_shape when given
// (1: waves outer 2 x 16, 2: channels outer 8 x 4, 3: channels outer 16 x 2),
// else the library's choice.  Returns the Shape<> index.
// dimension.both: 8 x 4 for complex data, 16 x 2 for real data, whose sums take half the
// registers (complex 16 x 2 spills).
// dimension.receive, waves outer: 4 x 8, 8 x 4 up to eight waves and 16 x 2 for one or
// two, whose slots would be padding otherwise (2 x 16, on request, leaves most of its
// slots empty for few waves, and its sums spill).  2 x 16 / 4 x 8 / 8 x 4 / 16 x 2, us,
// 128 complex channels on 120 x 90 pixels: 2 waves 82 / - / 41 / 37, 4 waves
// 94 / 58 / 47 / 38, 8 waves 112 / 70 / 50 / 63, 16 waves 133 / 76 / 84 / 88, 75 waves
// 310 / 237 / 239 / -; 64 real channels on 200 x 200: 4 waves 45 / 31 / 27 / 33, 8 waves
// 53 / 33 / 31 / 40, 75 waves 156 / 129 / 154 / -.
int shape_for(int dim, bool cplx, int32_t requested, int64_t W) {
    if (requested > 0) return requested - 1;
    switch (dim) {
        case USTB_DIM_RECEIVE: return W <= 2 ? 4 : W <= 8 ? 3 : 5;
        case USTB_DIM_BOTH: return cplx ? 1 : 2;
        default: return 1;
    }
}

// A sub-tile's work in stages, and a CTA's that has one of `parts` of it.
struct Work {
    int64_t groups, chunks;
    double setup;
    double cta(int parts) const { return setup + (double)groups * (double)chunks / parts; }
};
Work work_of(const Params& A) {
    const ustb::StageShape sh = ustb::kShapes[A.shape];
    return {(A.N + sh.cg - 1) / sh.cg, (A.W + sh.kw - 1) / sh.kw, 4.5 + (double)(A.N + A.W) / 128.0};
}

// CTAs (parts) per sub-tile of a grid launch.  Few sub-tiles leave SMs without work or a
// last round of long CTAs; each part sets the tile up again.  The number taken minimises
//   (rounds + uneven) (set-up + stages / parts),
// rounds of CTAs (two per SM; half a round at least: one CTA per SM) and half a round for
// CTAs of different lengths, a quarter from one and a half rounds on, times a CTA's length
// in stages (its set-up is worth 4.5 and one for every 128 channels and waves); another
// part must shorten it by 1 %, and a part of dimension.both keeps four stages (a call of a
// few stages is bound by the host).  Measured, one part against this rule: synthetic
// aperture of real traces, 128 x 128, 640 and 591 us, 115 x 115 on 223 x 73 pixels, 480 and
// 225; a transmit image of 145 channels x 9 waves on 73 x 252 pixels, 97 and 60; 75-wave IQ
// compounding, 525 either way.
// transmit and receive split where their outputs do not overlap; the epilogue's sums over
// channels are added like dimension.both's (81 channels x 29 waves into 68 x 89 pixels with
// coherence factors: one part 159 us, three 78).
int parts_for(const Params& A, int dim, int32_t requested, int& parts) {
    parts = 1;
    if (dim == USTB_DIM_BOTH && requested > 0) {
        parts = requested;
        return USTB_OK;
    }
    if (dim == USTB_DIM_NONE) return USTB_OK;
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const Work w = work_of(A);
    const int64_t most = dim == USTB_DIM_RECEIVE ? w.chunks : dim == USTB_DIM_TRANSMIT ? w.groups : w.groups * w.chunks / 4;
    const double rounds = (double)A.n_tiles * (double)A.F / sms;  // of one part each (A.subs CTAs per SM)
    double best = 0.0;
    for (int k = 1; k <= 8 && k <= most; ++k) {
        const double r = std::max(k * rounds, 1.0 / A.subs), uneven = 0.25 + 0.5 * std::min(std::max(1.5 - r, 0.0), 0.5);
        const double cost = (r + uneven) * w.cta(k);
        if (k == 1 || cost < 0.99 * best) {
            parts = k;
            best = cost;
        }
    }
    return USTB_OK;
}

// Sub-tiles per tile: two CTAs of half a tile share an SM.  Where a request's tables leave
// room for one CTA (from about 1180 channels with a few waves, 970 with 128), dimension.both
// takes the whole tile with twice the threads, and FP32 entries.  Half / whole tiles, us:
// 35 x 35 elements x 9 waves on 32 x 32 x 48 pixels 662 / 460, on 16 x 16 x 48 257 / 205, 48 x 48
// real x 4 waves 406 / 283, 1024 x 128 half-precision 2687 / 2459.  Transmit and receive
// images keep halves: 35 x 35 x 4 waves on 24 x 24 x 32 354 / 367; receive, 9 waves on
// 32 x 32 x 48, 653 / 708, 48 x 48 real x 2 waves 333 / 417.
int subs_for(Params& A, int dim) {
    int fit = 0;
    const int rc = ustb::ctas_per_sm(ustb::smem_bytes(A.shape, A.N, A.W), fit);
    if (rc) return rc;
    A.subs = dim == USTB_DIM_BOTH && fit == 1 ? 1 : 2;
    if (A.subs == 1 && A.ent != ustb::kEntReal) A.ent = ustb::kEntComplex;
    return USTB_OK;
}

// one stored sample (global memory) as float2
template <int ST, bool CPLX>
__device__ __forceinline__ float2 load_sample(const void* ch, int64_t i) {
    if constexpr (CPLX) {
        if constexpr (ST == USTB_STORE_F32) return __ldg(reinterpret_cast<const float2*>(ch) + i);
        else if constexpr (ST == USTB_STORE_F16) return __half22float2(reinterpret_cast<const __half2*>(ch)[i]);
        else return __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(ch)[i]);
    } else {
        if constexpr (ST == USTB_STORE_F32) return make_float2(__ldg(reinterpret_cast<const float*>(ch) + i), 0.f);
        else if constexpr (ST == USTB_STORE_F16) return make_float2(__half2float(reinterpret_cast<const __half*>(ch)[i]), 0.f);
        else return make_float2(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ch)[i]), 0.f);
    }
}

// Both entry kernels also zero the tickets of the parts (das_fast.cuh) of the launch that
// follows them: a memset of its own costs the host as much as a launch.
__device__ __forceinline__ void zero_tickets(unsigned* tickets, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        tickets[i] = 0u;
}

// Interpolation entries of every trace: E[t][i] = {x_i, x_{i+1} - x_i} for
// 0 < i < L-1 (das_c.cpp:381-383's validity rule), zero elsewhere.  HBM-bound:
// one pass over the channel data.
template <int ST, bool CPLX>
__global__ void __launch_bounds__(256) build_entries_kernel(const void* __restrict__ ch,
                                                            void* __restrict__ entries, int64_t L, int64_t Lp,
                                                            int64_t n_traces, unsigned* tickets, int64_t n_tickets) {
    zero_tickets(tickets, n_tickets);
    // CTAs stride over traces, threads over the samples of a trace (no 64-bit divisions)
    for (int64_t t = blockIdx.x; t < n_traces; t += gridDim.x) {
        const int64_t in0 = t * L, out0 = t * Lp;
        for (int i = threadIdx.x; i < (int)Lp; i += blockDim.x) {
            float2 x0 = make_float2(0.f, 0.f), d = make_float2(0.f, 0.f);
            if (i >= 1 && i < (int)L - 1) {
                x0 = load_sample<ST, CPLX>(ch, in0 + i);
                const float2 x1 = load_sample<ST, CPLX>(ch, in0 + i + 1);
                d = make_float2(x1.x - x0.x, x1.y - x0.y);
            }
            if constexpr (CPLX) reinterpret_cast<float4*>(entries)[out0 + i] = make_float4(x0.x, x0.y, d.x, d.y);
            else reinterpret_cast<float2*>(entries)[out0 + i] = make_float2(x0.x, d.x);
        }
    }
}

// The same for complex 16-bit samples as they are stored: E[t][i] = {x_i, x_{i+1}}.
__global__ void __launch_bounds__(256) build_pairs_kernel(const unsigned* __restrict__ ch, uint2* __restrict__ entries,
                                                          int64_t L, int64_t n_traces, unsigned* tickets,
                                                          int64_t n_tickets) {
    zero_tickets(tickets, n_tickets);
    for (int64_t t = blockIdx.x; t < n_traces; t += gridDim.x) {
        const unsigned* x = ch + t * L;
        uint2* e = entries + t * L;
        for (int i = threadIdx.x; i < (int)L; i += blockDim.x) {
            const bool in = i >= 1 && i < (int)L - 1;
            e[i] = in ? make_uint2(__ldg(x + i), __ldg(x + i + 1)) : make_uint2(0u, 0u);
        }
    }
}

// ---- entries scratch ---------------------------------------------------------
int64_t entry_bytes(int64_t L, int64_t N, int64_t W, int64_t F, int ent) {
    return L * N * W * F * ustb::entry_size(ent);
}

// What a request's entries hold.  Complex 16-bit samples keep their storage type: a unit
// loads 8 bytes of shared memory instead of 16 and forms the difference itself, in the
// same FP32 roundings, and the pre-pass writes half as much.  Measured, FP32 entries
// against these: matrix volume 7.74 and 7.22 ms, int16 ensemble of 50 frames 4.62 and 4.14
// ms, sector with coherence factors 300 and 272 us; 200 x 200 pixels x 4 frames, 32 waves,
// 424 and 345 us (its windows need the half-size stages with FP32 entries), 400 x 400
// pixels, 75 waves, 517 and 507 us.  FP32 entries stay for one or two waves (7 draws of
// them 0 to 12 % slower here), receive images of more than eight waves (50 waves on
// 297 x 455 pixels 297 and 323 us), dimension.none (bound by its stores) and the shapes
// that are asked for.
int entries_for(int32_t storage, bool cplx, int dim, int shape, int64_t W) {
    if (!cplx) return ustb::kEntReal;
    if (storage == USTB_STORE_F32 || dim == USTB_DIM_NONE || W <= 2 || (dim == USTB_DIM_RECEIVE && W > 8) ||
        shape != shape_for(dim, true, 0, W))
        return ustb::kEntComplex;
    return storage == USTB_STORE_F16 ? ustb::kEntHalf : ustb::kEntBf16;
}

// A stream-ordered memory pool owned by the library (one per device) that keeps
// freed entry arrays for the next call instead of returning them to the driver.
cudaMemPool_t entry_pool(int dev) {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64) return nullptr;
    if (!pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        uint64_t keep = UINT64_MAX;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[dev] = p;
    }
    return pools[dev];
}

// Fill one request's entry array `dst` (entry_bytes(...) bytes of device memory) and zero
// its tickets.
int fill_entries(const void* ch, int32_t storage, int ent, int64_t L, int64_t N, int64_t W, int64_t F, void* dst,
                 cudaStream_t s, unsigned* tickets = nullptr, int64_t n_tickets = 0) {
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t traces = N * W * F, total = traces * L;
    if (total == 0) return USTB_OK;
    const unsigned grid = (unsigned)std::min<int64_t>(traces, (int64_t)sms * 32);
    if (ent == ustb::kEntHalf || ent == ustb::kEntBf16) {
        build_pairs_kernel<<<grid, 256, 0, s>>>(static_cast<const unsigned*>(ch), static_cast<uint2*>(dst), L, traces,
                                                tickets, n_tickets);
        USTB_CUDA(cudaGetLastError());
        return USTB_OK;
    }
    switch (storage * 2 + (ent == ustb::kEntComplex ? 1 : 0)) {
        case USTB_STORE_F32 * 2 + 1: build_entries_kernel<USTB_STORE_F32, true><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
        case USTB_STORE_F16 * 2 + 1: build_entries_kernel<USTB_STORE_F16, true><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
        case USTB_STORE_BF16 * 2 + 1: build_entries_kernel<USTB_STORE_BF16, true><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
        case USTB_STORE_F32 * 2: build_entries_kernel<USTB_STORE_F32, false><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
        case USTB_STORE_F16 * 2: build_entries_kernel<USTB_STORE_F16, false><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
        default: build_entries_kernel<USTB_STORE_BF16, false><<<grid, 256, 0, s>>>(ch, dst, L, L, traces, tickets, n_tickets); break;
    }
    USTB_CUDA(cudaGetLastError());
    return USTB_OK;
}

// Bytes of device memory from the library pool (stream-ordered).
int pool_alloc(int64_t bytes, const char* what, void** out, cudaStream_t s) {
    *out = nullptr;
    if (bytes == 0) return USTB_OK;
    int dev = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    cudaMemPool_t pool = entry_pool(dev);
    USTB_REQUIRE(pool, USTB_E_CUDA, "could not create the entry memory pool on device %d", dev);
    const cudaError_t e = cudaMallocFromPoolAsync(out, (size_t)bytes, pool, s);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        *out = nullptr;
        ustb::set_error("%lld bytes of %s: %s", (long long)bytes, what, cudaGetErrorString(e));
        return USTB_E_OOM;
    }
    return USTB_OK;
}

// Allocate and fill one request's entries.
int build_entries(const void* ch, int32_t storage, int ent_kind, int64_t L, int64_t N, int64_t W, int64_t F,
                  void** out, cudaStream_t s) {
    const int rc = pool_alloc(entry_bytes(L, N, W, F, ent_kind), "interpolation entries", out, s);
    if (rc || !*out) return rc;
    return fill_entries(ch, storage, ent_kind, L, N, W, F, *out, s);
}

// Bytes of the sums of a request's parts, where parts are added, and its number of tickets.
int64_t part_bytes(const Params& A, int dim, bool epi, int64_t& tickets) {
    tickets = 0;
    if (A.split <= 1 || (dim != USTB_DIM_BOTH && !epi)) return 0;
    tickets = A.n_tiles * A.subs * A.F;
    return tickets * A.split * (ustb::kTile / A.subs) * (epi ? 3 : 1) * (int64_t)sizeof(float2);
}
void set_parts(Params& A, void* scratch, int64_t sums) {
    A.partial = static_cast<float2*>(scratch);
    A.tickets = reinterpret_cast<unsigned*>(static_cast<char*>(scratch) + sums);
}

// The launch of reqs' entry kind.
template <bool BATCH>
int dispatch(int dim, int epi, const Params* reqs, const int64_t* frames, int n, unsigned long long* counter,
             int64_t nt, int64_t F, cudaStream_t s, int max_ctas) {
    auto run = [&](auto ent) {
        constexpr int ENT = decltype(ent)::value;
        if constexpr (ENT == ustb::kEntReal || ENT == ustb::kEntComplex)
            if (reqs[0].subs == 1)
                return ustb::das_dispatch<ENT, BATCH, 1>(dim, epi, reqs[0].shape, reqs, frames, n, counter, nt, F, s, max_ctas);
        return ustb::das_dispatch<ENT, BATCH, 2>(dim, epi, reqs[0].shape, reqs, frames, n, counter, nt, F, s, max_ctas);
    };
    switch (reqs[0].ent) {
        case ustb::kEntReal: return run(std::integral_constant<int, ustb::kEntReal>{});
        case ustb::kEntComplex: return run(std::integral_constant<int, ustb::kEntComplex>{});
        case ustb::kEntHalf: return run(std::integral_constant<int, ustb::kEntHalf>{});
        default: return run(std::integral_constant<int, ustb::kEntBf16>{});
    }
}

// Bytes of a caller workspace that holds the entries of every request of a batch
// (each request's array starts on a 256-byte boundary).
int64_t batch_workspace_bytes(const ustb_das_request* reqs, int32_t n) {
    int64_t total = 0;
    for (int i = 0; i < n; ++i) {
        const ustb_das_request& q = reqs[i];
        if (q.L <= 0 || q.N <= 0 || q.W <= 0 || q.F <= 0) continue;
        total += (entry_bytes(q.L, q.N, q.W, q.F, q.is_complex ? ustb::kEntComplex : ustb::kEntReal) + 255) & ~int64_t(255);
    }
    return total;
}

}  // namespace

// Validate one request and fill its kernel parameters.  Returns USTB_OK, or a
// status; *empty is set when the request has no work (its outputs are already
// handled, e.g. zero-filled).
static int make_params(const void* ch, int32_t storage, int32_t is_complex, int64_t L, int64_t N, int64_t W,
                       int64_t F, const ustb_das_geometry* g, int32_t dimension, int32_t epilogue,
                       const ustb_das_outputs* out, uint32_t* flags, cudaStream_t s, Params& A, bool& empty) {
    empty = false;
    USTB_REQUIRE(g && out, USTB_E_ARG, "geometry and outputs must be given");
    USTB_REQUIRE(dimension >= 0 && dimension <= 3, USTB_E_ARG, "Unknown sum mode %d", (int)dimension);
    USTB_REQUIRE(storage >= 0 && storage <= 2, USTB_E_DTYPE, "unknown storage type %d", (int)storage);
    USTB_REQUIRE(is_complex == 0 || is_complex == 1, USTB_E_ARG, "is_complex must be 0 or 1");
    USTB_REQUIRE(L >= 0 && N >= 0 && W >= 0 && F >= 0, USTB_E_SHAPE, "negative size");
    USTB_REQUIRE(g->n_elements == N && g->n_waves == W, USTB_E_SHAPE,
                 "geometry has %lld elements / %lld waves, channel data %lld / %lld",
                 (long long)g->n_elements, (long long)g->n_waves, (long long)N, (long long)W);
    USTB_REQUIRE(is_complex || !(fabsf(g->fd) > 1e-6f), USTB_E_DTYPE,
                 "The modulation frequency > 0 but the input data is real. Check inputs.");
    USTB_REQUIRE(!epilogue || (dimension == USTB_DIM_TRANSMIT && is_complex), USTB_E_ARG,
                 "the coherence-factor / DMAS epilogue needs dimension.transmit and complex data");
    USTB_REQUIRE(flags, USTB_E_ARG, "flags pointer is NULL");
    USTB_REQUIRE(F <= 65535, USTB_E_SHAPE, "at most 65535 frames per call");
    USTB_REQUIRE(L <= INT32_MAX - 256, USTB_E_SHAPE, "L=%lld exceeds the 32-bit sample index", (long long)L);
    USTB_REQUIRE(N <= 1000000 && W <= 1000000, USTB_E_SHAPE, "N and W must be below 10^6");
    USTB_REQUIRE(g->n_tiles <= INT32_MAX, USTB_E_SHAPE, "too many tiles");
    USTB_REQUIRE(g->sound_speed > 0.f && g->fs > 0.f, USTB_E_ARG, "sound speed and fs must be > 0");
    if (g->n_tiles == 0 || F == 0 || g->n_pixels == 0) { empty = true; return USTB_OK; }
    USTB_REQUIRE(g->element_xyz && g->pixel_xyz && g->tile_pixels && (W == 0 || g->waves), USTB_E_ARG,
                 "a geometry pointer is NULL");
    USTB_REQUIRE(L == 0 || N == 0 || W == 0 || ch, USTB_E_ARG, "channel data pointer is NULL");
    USTB_REQUIRE(((uintptr_t)ch & 15) == 0, USTB_E_ARG, "channel data must be 16-byte aligned");
    const int64_t P = g->n_pixels;
    if (L == 0 || N == 0 || W == 0) {
        const int64_t nout = out_elems(dimension, P, N, W, F);
        if (out->cube && nout)
            USTB_CUDA(cudaMemsetAsync(out->cube, 0, (size_t)nout * (is_complex ? 8 : 4), s));
        empty = true;
        return USTB_OK;
    }
    A.entries = nullptr;  // built by the caller of make_params
    A.L = L; A.Lp = L; A.N = N; A.W = W; A.F = F; A.P = P;
    A.el = g->element_xyz;
    A.px = g->pixel_xyz;
    A.tiles = g->tile_pixels;
    A.n_tiles = g->n_tiles;
    A.waves = g->waves;
    A.tx_delay_tab = g->tx_delay_table;
    A.tx_apo_tab = g->tx_apo_table;
    A.rx_apo_tab = g->rx_apo_table;
    A.pix_phase = reinterpret_cast<const float2*>(g->pixel_phase);
    A.fs = g->fs; A.t0 = g->t0; A.fd = (fabsf(g->fd) > 1e-6f) ? g->fd : 0.f;
    A.fd_fs = (double)A.fd / (double)A.fs;
    A.wave_step = N * A.Lp;
    A.frame_step = W * A.wave_step;
    A.c = g->sound_speed;
    A.inv_c = 1.f / g->sound_speed;
    A.fs_c = (double)A.fs / (double)A.c;
    A.lens = g->lens_delay;
    A.rx_window = g->rx_window;
    {
        const WinCoeffs wc = window_coeffs(g->rx_window);
        A.win_r1 = wc.r1; A.win_a = wc.a; A.win_e = wc.e; A.win_b = wc.b; A.win_c = wc.c; A.win_d = wc.d;
    }
    A.fnx = g->rx_f_number[0]; A.fny = g->rx_f_number[1];
    A.minx = g->rx_min_aperture[0]; A.miny = g->rx_min_aperture[1];
    A.maxx = g->rx_max_aperture[0]; A.maxy = g->rx_max_aperture[1];
    A.rx_origin = g->rx_use_origin;
    A.ox = g->rx_origin[0]; A.oy = g->rx_origin[1]; A.oz = g->rx_origin[2];
    A.cf_thr = g->cf_threshold;
    A.cube = out->cube;
    A.o_das = reinterpret_cast<float2*>(out->das);
    A.o_cf = out->cf;
    A.o_cfimg = reinterpret_cast<float2*>(out->cf_image);
    A.o_sdmas = out->sdmas;
    const OutStrides os = out_strides(dimension, P, N, W);
    A.rx_f = os.rx_f; A.w_f = os.w_f; A.f_f = os.f_f;
    A.flags = flags;
    USTB_REQUIRE(g->ctas_per_tile >= 0 && g->ctas_per_tile <= 4, USTB_E_ARG, "ctas_per_tile must be 0 to 4");
    A.after_entries = false;
    A.partial = nullptr;
    A.tickets = nullptr;
    USTB_REQUIRE(g->stage_shape >= 0 && g->stage_shape <= 3, USTB_E_ARG, "stage_shape must be 0, 1, 2 or 3");
    USTB_REQUIRE(g->stage_shape == 0 || dimension == USTB_DIM_BOTH ||
                     (dimension == USTB_DIM_RECEIVE) == (g->stage_shape == 1),
                 USTB_E_ARG, "stage_shape %d does not fit dimension %d (receive: 1; transmit/none: 2 or 3)",
                 (int)g->stage_shape, (int)dimension);
    A.shape = shape_for(dimension, is_complex != 0, g->stage_shape, W);
    A.ent = entries_for(storage, is_complex != 0, dimension, A.shape, W);
    int rc = subs_for(A, dimension);
    if (rc) return rc;
    rc = parts_for(A, dimension, g->ctas_per_tile, A.split);
    if (rc) return rc;
    A.fpi = 1;
    return USTB_OK;
}

extern "C" int ustb_das_fast(const void* ch, int32_t storage, int32_t is_complex, int64_t L, int64_t N,
                             int64_t W, int64_t F, const ustb_das_geometry* g, int32_t dimension,
                             int32_t epilogue, const ustb_das_outputs* out, uint32_t* flags, void* stream) {
    ustb::clear_error();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    USTB_REQUIRE(flags, USTB_E_ARG, "flags pointer is NULL");
    USTB_CUDA(cudaMemsetAsync(flags, 0, sizeof(uint32_t), s));
    Params A;
    bool empty = false;
    int rc = make_params(ch, storage, is_complex, L, N, W, F, g, dimension, epilogue, out, flags, s, A, empty);
    if (rc || empty) return rc;
    // entries, then the parts' sums and tickets
    const int64_t ent_bytes = (entry_bytes(L, N, W, F, A.ent) + 255) & ~int64_t(255);
    int64_t tickets = 0;
    const int64_t sums = part_bytes(A, dimension, epilogue != 0, tickets);
    void* ent = nullptr;
    rc = pool_alloc(ent_bytes + sums + tickets * (int64_t)sizeof(unsigned), "interpolation entries", &ent, s);
    if (rc == USTB_E_OOM && tickets) {  // room for the entries alone: whole sub-tiles
        A.split = 1;
        tickets = 0;
        ustb::clear_error();
        rc = pool_alloc(ent_bytes, "interpolation entries", &ent, s);
    }
    if (rc) return rc;
    A.entries = ent;
    A.after_entries = true;
    if (tickets) set_parts(A, static_cast<char*>(ent) + ent_bytes, sums);
    rc = fill_entries(ch, storage, A.ent, L, N, W, F, ent, s, A.tickets, tickets);
    if (!rc) rc = dispatch<false>(dimension, epilogue, &A, nullptr, 1, nullptr, g->n_tiles, F, s, 0);
    const cudaError_t fe = cudaFreeAsync(ent, s);
    if (rc) return rc;
    USTB_CUDA(fe);
    return USTB_OK;
}

extern "C" int64_t ustb_entries_bytes(int64_t L, int64_t N, int64_t W, int64_t F, int32_t is_complex) {
    if (L < 0 || N < 0 || W < 0 || F < 0) return 0;
    return entry_bytes(L, N, W, F, is_complex != 0);
}

extern "C" int ustb_build_entries(const void* ch, int32_t storage, int32_t is_complex, int64_t L, int64_t N,
                                  int64_t W, int64_t F, void* entries, void* stream) {
    ustb::clear_error();
    USTB_REQUIRE(storage >= 0 && storage <= 2, USTB_E_DTYPE, "unknown storage type %d", (int)storage);
    USTB_REQUIRE(L >= 0 && N >= 0 && W >= 0 && F >= 0, USTB_E_SHAPE, "negative size");
    USTB_REQUIRE(L <= INT32_MAX - 256, USTB_E_SHAPE, "L=%lld exceeds the 32-bit sample index", (long long)L);
    if (L == 0 || N == 0 || W == 0 || F == 0) return USTB_OK;
    USTB_REQUIRE(ch && entries, USTB_E_ARG, "NULL pointer");
    USTB_REQUIRE(((uintptr_t)entries & 15) == 0, USTB_E_ARG, "entries must be 16-byte aligned");
    return fill_entries(ch, storage, is_complex ? ustb::kEntComplex : ustb::kEntReal, L, N, W, F, entries, static_cast<cudaStream_t>(stream));
}

extern "C" int ustb_das_fast_entries(const void* entries, int32_t is_complex, int64_t L, int64_t N, int64_t W,
                                     int64_t F, const ustb_das_geometry* g, int32_t dimension, int32_t epilogue,
                                     const ustb_das_outputs* out, uint32_t* flags, void* stream) {
    ustb::clear_error();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    USTB_REQUIRE(flags, USTB_E_ARG, "flags pointer is NULL");
    USTB_CUDA(cudaMemsetAsync(flags, 0, sizeof(uint32_t), s));
    Params A;
    bool empty = false;
    // make_params validates the request; the storage type is irrelevant for entries
    int rc = make_params(entries, USTB_STORE_F32, is_complex, L, N, W, F, g, dimension, epilogue, out, flags, s, A,
                         empty);
    if (rc || empty) return rc;
    USTB_REQUIRE(((uintptr_t)entries & 15) == 0, USTB_E_ARG, "entries must be 16-byte aligned");
    A.entries = entries;
    int64_t tickets = 0;
    const int64_t sums = part_bytes(A, dimension, epilogue != 0, tickets);
    if (!tickets) return dispatch<false>(dimension, epilogue, &A, nullptr, 1, nullptr, g->n_tiles, F, s, 0);
    void* scratch = nullptr;
    rc = pool_alloc(sums + tickets * (int64_t)sizeof(unsigned), "partial sums", &scratch, s);
    if (rc == USTB_E_OOM) {  // whole sub-tiles
        A.split = 1;
        ustb::clear_error();
        return dispatch<false>(dimension, epilogue, &A, nullptr, 1, nullptr, g->n_tiles, F, s, 0);
    }
    if (rc) return rc;
    set_parts(A, scratch, sums);
    const cudaError_t me = cudaMemsetAsync(A.tickets, 0, (size_t)tickets * sizeof(unsigned), s);
    if (me == cudaSuccess) rc = dispatch<false>(dimension, epilogue, &A, nullptr, 1, nullptr, g->n_tiles, F, s, 0);
    const cudaError_t fe = cudaFreeAsync(scratch, s);
    if (rc) return rc;
    USTB_CUDA(me);
    USTB_CUDA(fe);
    return USTB_OK;
}

// Requests of one dimension, data kind and epilogue whose variants differ only by the
// library's choices (entries in the storage type, receive stages by the number of waves)
// run as one launch, with FP32 entries and the 8 x 4 stages, while they make at most 16
// rounds of CTAs: launches of a few rounds each leave SMs idle one after the other, and in
// longer ones the variants' own speed weighs more.  Measured, a launch per variant / one:
// six requests of FP32, FP16 and bfloat16 data, 11 waves, on 64 x 64 pixels 194 / 124 us, on
// 128 x 128 (1.3 rounds) 349 / 210, 31 waves on 256 x 256 (5 rounds) 657 / 650, twelve of
// them (10 rounds) 1236 / 1257, six on 400 x 400 (12 rounds) 1196 / 1182; receive images of 1,
// 4 and 20 waves on 64 x 64 182 / 142, on 200 x 200 in the three types 461 / 362.
// Whole tiles (subs_for) need enough of them here, where no parts fill the SMs: 35 x 35
// elements x 4 waves with 3 requests of 64 elements, 64 tiles, 576 us as halves, 846 whole;
// 9 waves, 256 tiles, 3138 / 2808.
constexpr int64_t kShareRounds = 16;
static int share_variants(const ustb_das_request* reqs, int32_t n, const std::vector<int>& key, std::vector<Params>& P) {
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (int dim = 0; dim < 4; ++dim)
        for (int epi = 0; epi < 2; ++epi)
            for (int cplx = 0; cplx < 2; ++cplx) {
                auto member = [&](int i) {
                    const ustb_das_request& q = reqs[i];
                    return key[i] >= 0 && q.dimension == dim && (q.epilogue != 0) == (epi != 0) && q.is_complex == cplx &&
                           P[i].shape == shape_for(dim, cplx != 0, 0, q.W);  // the library's, or the same asked for
                };
                int first = -1;
                bool differ = false;
                int64_t items = 0, whole = 0;  // tiles x frames; of requests that take whole tiles
                for (int i = 0; i < n; ++i) {
                    if (!member(i)) continue;
                    if (first < 0) first = i;
                    differ |= P[i].ent != P[first].ent || P[i].shape != P[first].shape || P[i].subs != P[first].subs;
                    items += P[i].n_tiles * P[i].F;
                    if (P[i].subs == 1) whole += P[i].n_tiles * P[i].F;
                }
                // too few whole tiles for every SM: halves go to twice as many
                const int subs = whole > sms / 2 ? 1 : 2;
                for (int i = 0; i < n; ++i)
                    if (member(i)) P[i].subs = std::max(P[i].subs, subs);
                if (!differ || items > kShareRounds * sms) continue;
                for (int i = 0; i < n; ++i) {
                    if (!member(i)) continue;
                    P[i].subs = subs;
                    if (cplx) P[i].ent = ustb::kEntComplex;
                    if (dim == USTB_DIM_RECEIVE) P[i].shape = 3;
                }
            }
    return USTB_OK;
}

// Scratch of a request's parts on a 256-byte boundary.
static int64_t parts_room(int64_t sums, int64_t tickets) {
    return (sums + tickets * (int64_t)sizeof(unsigned) + 255) & ~int64_t(255);
}

// Whether the requests of one variant run faster one after the other as grid launches, whose
// parts fill the SMs, than as one persistent launch of whole sub-tiles.  With fewer of these
// than SMs, the persistent launch takes as long as the longest request's one CTA, the grid
// launches the sum of their parts' (and a launch each, about 3 stages).  `room`: bytes of a
// caller's workspace left for the sums of parts, < 0: from the pool.  Persistent / grid, us:
// receive images of 64 channels x 75 waves, 100 x 100 pixels x 3 frames, 535 / 272, x 16 waves
// 122 / 63; 128 channels x 3 waves on 256 x 256 49 / 37; both, 64 x 75 on 50 x 50 328 / 90, 128 x
// 16 on 256 x 256 111 / 80; transmit with factors, 64 x 16 on 50 x 50 101 / 42.
static int grids_faster(const ustb_das_request& q, std::vector<Params>& gp, int sms, int64_t room, bool& yes) {
    yes = false;
    int64_t items = 0, need = 0;
    double one = 0.0, all = 0.0;
    for (Params& A : gp) {
        items += A.n_tiles * A.F;
        if (items > sms || q.dimension == USTB_DIM_NONE) return USTB_OK;
        const int rc = parts_for(A, q.dimension, 0, A.split);
        if (rc) return rc;
        int64_t tickets = 0;
        const int64_t sums = part_bytes(A, q.dimension, q.epilogue != 0, tickets);
        need += parts_room(sums, tickets);
        const Work w = work_of(A);
        one = std::max(one, w.cta(1));
        all += 3.0 + w.cta(A.split);
    }
    yes = all < 0.9 * one && (room < 0 || need <= room);
    return USTB_OK;
}

static int das_fast_batch_impl(const ustb_das_request* reqs, int32_t n, uint64_t* scratch, void* workspace,
                               int64_t workspace_bytes, int32_t max_ctas, void* stream) {
    ustb::clear_error();
    USTB_REQUIRE(n >= 0 && (n == 0 || reqs), USTB_E_ARG, "bad request array");
    USTB_REQUIRE(max_ctas >= 0, USTB_E_ARG, "max_ctas must be >= 0 (0: every SM)");
    USTB_REQUIRE(scratch, USTB_E_ARG, "scratch pointer is NULL");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint32_t* flags = reinterpret_cast<uint32_t*>(scratch);
    USTB_CUDA(cudaMemsetAsync(scratch, 0, sizeof(uint64_t), s));
    if (n == 0) return USTB_OK;
    // validate all requests first, then launch one persistent kernel per kernel variant.
    // Complex data takes the library's stages: beside the loop over frames the sums of the
    // others spill (2 x 16: 1.7 KB a thread, 16 x 2 1.2 KB).  128 channels on 256 x 256 pixels,
    // 2 x 16 / 16 x 2 / 8 x 4, us: 5 waves 80 / 79 / 64, 16 waves 115 / 134 / 110, 75 waves
    // 495 / 469 / 399.
    std::vector<Params> P(n);
    std::vector<int64_t> frames(n);
    std::vector<int> key(n, -1);
    for (int i = 0; i < n; ++i) {
        const ustb_das_request& q = reqs[i];
        bool empty = false;
        int rc = make_params(q.ch, q.storage, q.is_complex, q.L, q.N, q.W, q.F, q.geometry, q.dimension,
                             q.epilogue, q.out, flags, s, P[i], empty);
        if (rc) {
            char msg[1200];
            snprintf(msg, sizeof msg, "request %d: %s", i, ustb_last_error());
            ustb::set_error("%s", msg);
            return rc;
        }
        frames[i] = q.F;
        if (empty) continue;
        key[i] = 0;
        if (q.is_complex) {  // the library's own stages
            P[i].shape = shape_for(q.dimension, true, 0, q.W);
            P[i].ent = entries_for(q.storage, true, q.dimension, P[i].shape, q.W);
            rc = subs_for(P[i], q.dimension);
            if (rc) return rc;
        }
    }
    int rc = share_variants(reqs, n, key, P);
    if (rc) return rc;
    for (int i = 0; i < n; ++i)
        if (key[i] >= 0)
            key[i] = (((reqs[i].dimension * 4 + P[i].ent) * 2 + (reqs[i].epilogue ? 1 : 0)) * 8 + P[i].shape) * 2 + P[i].subs - 1;
    // every request's entry array: carved from the caller's workspace, or allocated
    // from the library pool and freed (stream-ordered) after the launches
    std::vector<void*> ents;
    auto release = [&]() {
        for (void* e : ents) (void)cudaFreeAsync(e, s);
        ents.clear();
    };
    if (workspace) {
        const int64_t need = batch_workspace_bytes(reqs, n);
        USTB_REQUIRE(need <= workspace_bytes, USTB_E_SHAPE, "the workspace holds %lld bytes, the batch needs %lld",
                     (long long)workspace_bytes, (long long)need);
        USTB_REQUIRE(((uintptr_t)workspace & 255) == 0, USTB_E_ARG, "the workspace must be 256-byte aligned");
    }
    int64_t ws_off = 0;
    for (int i = 0; i < n; ++i) {
        if (key[i] < 0) continue;
        const ustb_das_request& q = reqs[i];
        void* ent = nullptr;
        int rc;
        if (workspace) {
            ent = static_cast<char*>(workspace) + ws_off;
            ws_off += (entry_bytes(q.L, q.N, q.W, q.F, P[i].ent) + 255) & ~int64_t(255);
            rc = fill_entries(q.ch, q.storage, P[i].ent, q.L, q.N, q.W, q.F, ent, s);
        } else {
            rc = build_entries(q.ch, q.storage, P[i].ent, q.L, q.N, q.W, q.F, &ent, s);
            if (!rc) ents.push_back(ent);
        }
        if (rc) {
            release();
            return rc;
        }
        P[i].entries = ent;
    }
    int group = 0, dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    std::vector<bool> done(n, false);
    for (int i = 0; i < n; ++i) {
        if (key[i] < 0 || done[i]) continue;
        std::vector<Params> gp;
        std::vector<int64_t> gf;
        for (int j = i; j < n; ++j)
            if (!done[j] && key[j] == key[i]) {
                gp.push_back(P[j]);
                gf.push_back(frames[j]);
                done[j] = true;
            }
        const ustb_das_request& q = reqs[i];
        bool grids = false;
        int rc = max_ctas > 0 ? (int)USTB_OK : grids_faster(q, gp, sms, workspace ? workspace_bytes - ws_off : -1, grids);
        for (size_t k = 0; grids && !rc && k < gp.size(); ++k) {
            Params& A = gp[k];
            int64_t tickets = 0;
            const int64_t sums = part_bytes(A, q.dimension, q.epilogue != 0, tickets);
            const int64_t room = parts_room(sums, tickets);
            void* scr = workspace ? static_cast<char*>(workspace) + ws_off : nullptr;
            if (workspace) {
                ws_off += room;
            } else if (tickets) {
                rc = pool_alloc(room, "partial sums", &scr, s);
                if (!rc) ents.push_back(scr);
            }
            if (rc == USTB_E_OOM) {  // whole sub-tiles
                ustb::clear_error();
                A.split = 1;
                tickets = 0;
                rc = USTB_OK;
            }
            if (tickets) {
                set_parts(A, scr, sums);
                const cudaError_t e = cudaMemsetAsync(A.tickets, 0, (size_t)tickets * sizeof(unsigned), s);
                if (e != cudaSuccess) rc = ustb::cuda_fail(e, "cudaMemsetAsync", __FILE__, __LINE__);
            }
            if (!rc) rc = dispatch<false>(q.dimension, q.epilogue, &A, nullptr, 1, nullptr, A.n_tiles, A.F, s, 0);
        }
        if (rc) {
            release();
            return rc;
        }
        if (grids) continue;
        for (size_t off = 0; off < gp.size(); off += kMaxBatch) {
            const int cnt = (int)std::min<size_t>(kMaxBatch, gp.size() - off);
            unsigned long long* counter = reinterpret_cast<unsigned long long*>(scratch + 1 + group);
            ++group;
            if (group > n) {
                release();
                ustb::set_error("scratch holds n + 1 words");
                return USTB_E_ARG;
            }
            rc = dispatch<true>(q.dimension, q.epilogue, gp.data() + off, gf.data() + off, cnt, counter, 0, 0, s, max_ctas);
            if (rc) {
                release();
                return rc;
            }
        }
    }
    release();
    return USTB_OK;
}

extern "C" int ustb_das_fast_batch(const ustb_das_request* reqs, int32_t n, uint64_t* scratch, void* stream) {
    return das_fast_batch_impl(reqs, n, scratch, nullptr, 0, 0, stream);
}

extern "C" int ustb_das_fast_batch_ex(const ustb_das_request* reqs, int32_t n, uint64_t* scratch, void* workspace,
                                      int64_t workspace_bytes, int32_t max_ctas, void* stream) {
    return das_fast_batch_impl(reqs, n, scratch, workspace, workspace_bytes, max_ctas, stream);
}

extern "C" int64_t ustb_das_fast_workspace_bytes(const ustb_das_request* reqs, int32_t n) {
    if (n <= 0 || !reqs) return 0;
    return batch_workspace_bytes(reqs, n);
}

extern "C" int ustb_das_fast_batch_ws(const ustb_das_request* reqs, int32_t n, uint64_t* scratch, void* workspace,
                                      int64_t workspace_bytes, void* stream) {
    if (!workspace) {
        ustb::clear_error();
        ustb::set_error("workspace pointer is NULL (ustb_das_fast_batch allocates its own)");
        return USTB_E_ARG;
    }
    return das_fast_batch_impl(reqs, n, scratch, workspace, workspace_bytes, 0, stream);
}

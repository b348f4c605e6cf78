// Capon minimum-variance beamforming on a kept channel cube
// (+postprocess/capon_minimum_variance.m:117-177), one warp per pixel or group of pixels.
//
// For pixel (iz, ix) of a scan grid with depth fastest, over the M values x[c] of
// its channels (or waves) and the rows r of its depth window [iz-K, iz+K] (clipped):
//   active channels c: |apod[c]| > criterion; first a, last b, count Ma.
//   All |x| <= eps -> 0; Ma < 2 -> sum_c x[c].
//   L = clamp(floor(L_elements / M * Ma), 1, Ma - 1); subarray starts l = a .. b-L+1.
//   R = sum_r sum_l X_r[l:l+L]^H X_r[l:l+L] / ((2K+1)(Ma - L + 1))  (rows of A' * A),
//   optionally R = (R + J conj(R) J) / 2 (forward-backward),
//   w = (R + I regCoef/L trace R)^-1 1 / (1^T (...)^-1 1),
//   z = Ma / (Ma - L + 1) * sum_l conj(w)^T conj(x_iz[l:l+L])   (w' * x', as written).
//
// Summed over the rows first, R needs only the band P(c, d) = sum_r conj(X_r[c]) X_r[c + d],
// d < L, of the channels' Gram matrix:
//   R[i][i + d] = sum_{l = a}^{b - L + 1} P(l + i, d).
// Up to 64 channels the band is cut into 8 x 8 tiles (at most 30), one per lane with its
// sums in registers, so a row costs 16 shared-memory values per 64 products.  One warp takes
// up to 4 neighbouring pixels of a depth column: the rows their windows share are summed once
// and stay in registers, each pixel adds its own few rows.  Each lane then walks one diagonal
// of P with a compensated sliding sum.  With more channels the band no longer fits one tile
// per lane and leaves room for few warps: there a warp takes one pixel and lane d slides over
// diagonal d of each row's products, adding to R in shared memory.
// The system is solved by a Cholesky factorisation R = U^H U, one column per lane and four
// rows at a time, the forward substitution carried along, and a backward substitution with
// one unknown per lane.
//
// Latency-bound: 8 warps per SM (the tiles take 244 registers), 41 % issue.  GB300, 131072
// pixels of 64 channels, 32-element subarrays, 15 rows: 2.51 ms; 5.57 ms with each row's
// diagonals slid through shared memory and the triangular solves on one lane.  16384 pixels,
// 15 rows, tiles in several passes / row by row: 96 channels 642 / 612 us, 128 1088 / 732, 256
// 4143 / 1202; one row: 451 / 142, 722 / 162, 2136 / 223.  (At 64 channels row by row takes
// 513 us against 375 with 15 rows, 291 against 336 with 7, 129 against 301 with one.)
// Not kept: the factorisation unrolled with the column in registers (3.9 ms together with
// pixel groups: the warps wait for instructions), packed pairs for the tiles (2.83 ms against
// 2.69 ms), 12 warps of 168 registers (2.80 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace {

constexpr int kLMax = 32;        // subarray length <= one lane per diagonal and column
constexpr int kWarps = 4;        // warps per CTA
constexpr int kMMax = 256;       // channels per pixel
constexpr int kTileC = 8;        // channels per tile side
constexpr int kTileStride = 20;  // words per staged block of 8 channels: 8 real, 8 imaginary parts, padding (the
                                 // tiles' 16-byte loads hit distinct banks)
constexpr int kRows = 8;         // rows staged at a time
constexpr int kGroup = 4;        // pixels per warp at most
constexpr int kTileM = 64;       // channels of the tile kernel at most
constexpr int kBand = kLMax + 2;  // stride of the band and of R in shared memory

// Words of shared memory per warp: staged rows, the band P (its space then takes R and U)
// and the pixel's own row.
__host__ __device__ __forceinline__ int blocks_of(int M) { return (M + kTileC - 1) / kTileC; }
__host__ __device__ __forceinline__ int band_offset(int M) { return kRows * blocks_of(M) * kTileStride; }
__host__ __device__ __forceinline__ int own_offset(int M) {
    const int band = 2 * blocks_of(M) * kTileC * kBand, R = 2 * kLMax * kBand;
    return band_offset(M) + (band > R ? band : R);
}
__host__ __device__ __forceinline__ int warp_words(int M) { return (own_offset(M) + 2 * M + 3) & ~3; }

struct CaponArgs {
    int64_t nz, nx, F, M;
    int K;                 // depth half-window in samples
    float l_frac;          // L_elements / M
    float crit;            // active-element criterion
    float reg;             // regularisation coefficient
    int fb;                // forward-backward averaging
    int group;             // neighbouring pixels (in depth) per warp, 1 .. kGroup
};

__device__ __forceinline__ float norm_of(const CaponArgs& a, int cnt, int L) {
    return 1.f / ((float)(2 * a.K + 1) * (float)(cnt - L + 1));
}

__device__ __forceinline__ float2 shfl2(float2 v, int src) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// A compensated (Kahan) sum: what a sliding window gains and loses leaves no drift.
struct Slide {
    float2 g = make_float2(0.f, 0.f), lost = make_float2(0.f, 0.f);
    __device__ __forceinline__ void add(float x, float y) {
        const float px = x - lost.x, py = y - lost.y;
        const float nx = g.x + px, ny = g.y + py;
        lost = make_float2((nx - g.x) - px, (ny - g.y) - py);
        g = make_float2(nx, ny);
    }
};

// A pixel's active channels, all-zero test and plain sum of its own row `x` (channels P apart).
struct Aperture {
    int lo, hi, cnt, L;  // first and last active channel, their number, the subarray's length
    bool any;            // a value that is not zero
    float2 sum;
    __device__ __forceinline__ bool adaptive() const { return any && cnt >= 2 && hi - L + 1 >= lo; }
    // silent: 0; no subarray fits: the plain sum
    __device__ __forceinline__ float2 plain() const { return any ? sum : make_float2(0.f, 0.f); }
};
__device__ __forceinline__ Aperture aperture_of(const float2* x, const float* apod, int M, int64_t P, const CaponArgs& a,
                                                int lane) {
    Aperture q = {M, -1, 0, 0, false, make_float2(0.f, 0.f)};
    for (int c = lane; c < M; c += 32) {
        const float2 v = __ldg(x + (int64_t)c * P);
        q.any |= hypotf(v.x, v.y) > 2.220446049250313e-16f;
        q.sum.x += v.x;
        q.sum.y += v.y;
        if (fabsf(__ldg(apod + (int64_t)c * P)) > a.crit) {
            q.lo = min(q.lo, c);
            q.hi = max(q.hi, c);
            ++q.cnt;
        }
    }
    q.lo = __reduce_min_sync(0xffffffffu, q.lo);
    q.hi = __reduce_max_sync(0xffffffffu, q.hi);
    q.cnt = __reduce_add_sync(0xffffffffu, q.cnt);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        q.sum.x += __shfl_xor_sync(0xffffffffu, q.sum.x, o);
        q.sum.y += __shfl_xor_sync(0xffffffffu, q.sum.y, o);
    }
    q.any = __any_sync(0xffffffffu, q.any);
    q.L = max(1, min((int)floorf(a.l_frac * (float)q.cnt), q.cnt - 1));
    return q;
}

// R of one pixel, in the place of its band P (rows from channel c0 on), along its
// diagonals: lane d slides over diagonal d.  `start`: l0 - c0; nl subarrays.
__device__ __forceinline__ void matrix_of_band(float2* band, int lane, int L, int start, int nl, float norm) {
    const float2* Pd = band + start * kBand + lane;  // P(l0 + i, d) at i * kBand
    Slide s;
    if (lane < L)
        for (int l = 0; l < nl; ++l) s.add(Pd[l * kBand].x, Pd[l * kBand].y);
    // row i of R takes the place of the band's row i, which every lane has read then
    // (row i of the band is the first of those that a later window drops)
    for (int i = 0; i < L; ++i) {
        const float2 v = make_float2(s.g.x * norm, s.g.y * norm);
        if (i + 1 + lane < L) {
            const float2 add = Pd[(nl + i) * kBand], sub = Pd[i * kBand];
            s.add(add.x - sub.x, add.y - sub.y);
        }
        __syncwarp();
        if (i + lane < L) band[i * kBand + i + lane] = v;
    }
    __syncwarp();
}

// The Capon value of one pixel from the upper triangle of its R: the factorisation, the
// weights and their sum over the pixel's own row.
__device__ __forceinline__ float2 capon_value(float2 (*R)[kBand], const float2* own, const CaponArgs& a, int lane, int L,
                                              int cnt, int l0, int l1) {
    if (a.fb) {
        // (J conj(R) J)[i][j] = conj(R[L-1-i][L-1-j]); average the upper triangle
        for (int idx = lane; idx < L * L; idx += 32) {
            const int i = idx / L, j = idx - (idx / L) * L;
            if (j < i) R[i][j] = make_float2(R[j][i].x, -R[j][i].y);
        }
        __syncwarp();
        float2 nv[kLMax];
        int n = 0;
        for (int idx = lane; idx < L * L; idx += 32, ++n) {
            const int i = idx / L, j = idx - (idx / L) * L;
            const float2 q = R[L - 1 - i][L - 1 - j];
            nv[n] = make_float2(0.5f * (R[i][j].x + q.x), 0.5f * (R[i][j].y - q.y));
        }
        __syncwarp();
        n = 0;
        for (int idx = lane; idx < L * L; idx += 32, ++n) {
            const int i = idx / L, j = idx - (idx / L) * L;
            R[i][j] = nv[n];
        }
        __syncwarp();
    }
    float tr = lane < L ? R[lane][lane].x : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    // ---- Cholesky R = U^H U, lane j column j, four rows at a time, and U^H y = 1 ----
    // (rolled loops: unrolled over all rows with the column in registers, the warps of an SM
    // waited for instructions)
    const float load = a.reg / (float)L * tr;
    float2 y = make_float2(lane < L ? 1.f : 0.f, 0.f);
    float inv_diag = 0.f;
    for (int k0 = 0; k0 < L; k0 += 4) {
        float2 s[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            s[r] = k0 + r <= lane && lane < L ? R[k0 + r][lane] : make_float2(0.f, 0.f);
            if (k0 + r == lane) s[r].x += load;
        }
        auto take = [](float2& v, float2 c, float2 u) {  // v -= conj(c) u
            v.x = fmaf(-c.x, u.x, fmaf(-c.y, u.y, v.x));
            v.y = fmaf(-c.x, u.y, fmaf(c.y, u.x, v.y));
        };
#pragma unroll 2
        for (int m = 0; m < k0; ++m) {
            const float2 u = R[m][lane];
            const float4 c0 = *reinterpret_cast<const float4*>(&R[m][k0]), c1 = *reinterpret_cast<const float4*>(&R[m][k0 + 2]);
            take(s[0], make_float2(c0.x, c0.y), u);
            take(s[1], make_float2(c0.z, c0.w), u);
            take(s[2], make_float2(c1.x, c1.y), u);
            take(s[3], make_float2(c1.z, c1.w), u);
        }
        __syncwarp();  // R's rows k0 .. k0 + 3 are read: U's take their place
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = k0 + r;
            if (k >= L) continue;
            const float inv = 1.f / sqrtf(fmaxf(__shfl_sync(0xffffffffu, s[r].x, k), 1e-30f));
            const float2 u = lane > k && lane < L ? make_float2(s[r].x * inv, s[r].y * inv) : make_float2(0.f, 0.f);
            R[k][lane] = u;
            if (lane == k) {
                inv_diag = inv;
                y = make_float2(y.x * inv, y.y * inv);
            }
            take(y, u, shfl2(y, k));
#pragma unroll
            for (int q = r + 1; q < 4; ++q) take(s[q], shfl2(u, (k0 + q) & 31), u);
        }
        __syncwarp();
    }
    // ---- U x = y, then w = x / (1^T x) ----
    for (int m = L - 1; m >= 0; --m) {
        if (lane == m) y = make_float2(y.x * inv_diag, y.y * inv_diag);
        const float2 x = shfl2(y, m);
        if (lane < m) {
            const float2 u = R[lane][m];
            y.x -= u.x * x.x - u.y * x.y;
            y.y -= u.x * x.y + u.y * x.x;
        }
    }
    float2 den = lane < L ? y : make_float2(0.f, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        den.x += __shfl_xor_sync(0xffffffffu, den.x, o);
        den.y += __shfl_xor_sync(0xffffffffu, den.y, o);
    }
    // z = sum_i conj(w_i) sum_l conj(x_iz[l + i]) * Ma / (Ma - L + 1)
    float2 z = make_float2(0.f, 0.f);
    if (lane < L) {
        const float dd = den.x * den.x + den.y * den.y;
        const float2 w = make_float2((y.x * den.x + y.y * den.y) / dd, (y.y * den.x - y.x * den.y) / dd);
        float2 s = make_float2(0.f, 0.f);
        for (int l = l0; l <= l1; ++l) {
            s.x += own[l + lane].x;
            s.y += own[l + lane].y;
        }
        z = make_float2(w.x * s.x - w.y * s.y, -(w.x * s.y + w.y * s.x));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
        z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
    }
    const float sc = (float)cnt / (float)(cnt - L + 1);
    return make_float2(z.x * sc, z.y * sc);
}

__global__ void __launch_bounds__(32 * kWarps, 2) capon_kernel(const float2* __restrict__ cube,
                                                               const float* __restrict__ apod, float2* __restrict__ out,
                                                               const CaponArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int M = (int)a.M;
    float* rows = smem + wi * warp_words(M);
    float2* band = reinterpret_cast<float2*>(rows + band_offset(M));
    float2* own = reinterpret_cast<float2*>(rows + own_offset(M));
    const int64_t P = a.nz * a.nx;
    const int64_t per_col = (a.nz + a.group - 1) / a.group, total = per_col * a.nx * a.F;
    for (int64_t t = (int64_t)blockIdx.x * nwarps + wi; t < total; t += (int64_t)gridDim.x * nwarps) {
        const int64_t f = t / (per_col * a.nx), rest = t - f * per_col * a.nx;
        const int64_t ix = rest / per_col;
        const int iz0 = (int)(rest - ix * per_col) * a.group, nz = (int)a.nz;
        const int np = min(a.group, nz - iz0);                      // this warp's pixels iz0 .. iz0 + np - 1
        const float2* base = cube + f * a.M * P + ix * a.nz;        // [M][P] at this column's first depth
        // every pixel's active channels, all-zero test and plain sum of its own row
        int my_lo = 0, my_hi = 0, my_L = 0, my_cnt = 0;  // lane g: pixel iz0 + g
        int first = M, last = -1;  // over the pixels that need weights
        int Lmax = 0;
#pragma unroll
        for (int g = 0; g < kGroup; ++g) {
            if (g >= np) continue;
            const int64_t p = ix * a.nz + iz0 + g;
            const Aperture q = aperture_of(base + iz0 + g, apod + p, M, P, a, lane);
            if (!q.adaptive()) {
                if (lane == 0) out[f * P + p] = q.plain();
                continue;
            }
            if (lane == g) {
                my_lo = q.lo;
                my_hi = q.hi;
                my_L = q.L;
                my_cnt = q.cnt;
            }
            first = min(first, q.lo);
            last = max(last, q.hi);
            Lmax = max(Lmax, q.L);
        }
        if (Lmax == 0) continue;

        // ---- the band of the Gram matrix over the rows that every pixel's window shares ----
        const int r0 = max(0, iz0 + np - 1 - a.K), r1 = min(nz - 1, iz0 + a.K);
        const int fb = first / kTileC, nblk = last / kTileC - fb + 1, c0 = fb * kTileC;
        const int wide = (Lmax + kTileC - 2) / kTileC + 1;  // tiles of one block row that reach d < L
        int ntiles = 0;
        for (int i = 0; i < nblk; ++i) ntiles += min(wide, nblk - i);
        // rows [ra, rb) (at most kRows) of the staged channels; kRows neighbouring rows of 4
        // channels per load; channels past M are zeros
        auto stage = [&](int ra, int nr) {
            __syncwarp();
            const int r = lane % kRows;
            const float2* src = base + (int64_t)c0 * P + ra + r;
            for (int c = lane / kRows; c < nblk * kTileC; c += 32 / kRows) {
                float2 x = make_float2(0.f, 0.f);
                if (r < nr && c0 + c < M) x = __ldg(src + (int64_t)c * P);
                float* dst = rows + (r * nblk + c / kTileC) * kTileStride + c % kTileC;
                dst[0] = x.x;
                dst[kTileC] = x.y;
            }
            __syncwarp();
        };
        int ti = 0, tj = lane;  // this lane's tile (block row ti, block column tj)
        const bool mine = tj < ntiles;
        if (!mine) tj = 0;
        while (tj >= min(wide, nblk - ti)) {
            tj -= min(wide, nblk - ti);
            ++ti;
        }
        tj += ti;
        // one staged row's 8 channels of a block: real parts, then imaginary parts
        auto block_at = [&](int q, int blk) { return rows + (q * nblk + blk) * kTileStride; };
        auto load8 = [&](const float* src, float (&x)[kTileC], float (&y)[kTileC]) {
            const float4* v = reinterpret_cast<const float4*>(src);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 p = v[h], q = v[2 + h];
                x[4 * h] = p.x; x[4 * h + 1] = p.y; x[4 * h + 2] = p.z; x[4 * h + 3] = p.w;
                y[4 * h] = q.x; y[4 * h + 1] = q.y; y[4 * h + 2] = q.z; y[4 * h + 3] = q.w;
            }
        };
        float re[kTileC][kTileC], im[kTileC][kTileC];  // sums of the tile over the common rows
#pragma unroll
        for (int u = 0; u < kTileC; ++u)
#pragma unroll
            for (int v = 0; v < kTileC; ++v) re[u][v] = im[u][v] = 0.f;
        for (int rb = r0; rb <= r1; rb += kRows) {
            const int nr = min(kRows, r1 - rb + 1);
            stage(rb, nr);
            for (int q = 0; q < nr; ++q) {
                float bx[kTileC], by[kTileC];
                load8(block_at(q, tj), bx, by);
                const float4* xa = reinterpret_cast<const float4*>(block_at(q, ti));
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 ax4 = xa[h], ay4 = xa[2 + h];
                    const float ax[4] = {ax4.x, ax4.y, ax4.z, ax4.w}, ay[4] = {ay4.x, ay4.y, ay4.z, ay4.w};
#pragma unroll
                    for (int w = 0; w < 4; ++w)
#pragma unroll
                        for (int v = 0; v < kTileC; ++v) {  // += conj(a) b
                            const int u = 4 * h + w;
                            re[u][v] = fmaf(ax[w], bx[v], fmaf(ay[w], by[v], re[u][v]));
                            im[u][v] = fmaf(ax[w], by[v], fmaf(-ay[w], bx[v], im[u][v]));
                        }
                }
            }
        }
        // ---- each pixel: its own rows besides the common ones, then its weights ----
        for (int g = 0; g < np; ++g) {
            const int L = __shfl_sync(0xffffffffu, my_L, g);
            if (L == 0) continue;
            const int below = r0 - max(0, iz0 + g - a.K), above = min(nz - 1, iz0 + g + a.K) - r1;  // own rows
            if (below > 0) stage(r0 - below, below);
            __syncwarp();  // (no own row: the pixel before has read the band)
            auto own_rows = [&](int n, int u, float (&tx)[kTileC], float (&ty)[kTileC]) {
                for (int q = 0; q < n; ++q) {
                    float bx[kTileC], by[kTileC];
                    load8(block_at(q, tj), bx, by);
                    const float ax = block_at(q, ti)[u], ay = block_at(q, ti)[kTileC + u];
#pragma unroll
                    for (int v = 0; v < kTileC; ++v) {
                        tx[v] = fmaf(ax, bx[v], fmaf(ay, by[v], tx[v]));
                        ty[v] = fmaf(ax, by[v], fmaf(-ay, bx[v], ty[v]));
                    }
                }
            };
            // `above` rows are staged behind the `below` ones: together at most kGroup - 1
            if (above > 0) {
                const int r = lane % kRows;
                for (int c = lane / kRows; c < nblk * kTileC; c += 32 / kRows) {
                    if (r >= above) continue;
                    float2 x = make_float2(0.f, 0.f);
                    if (c0 + c < M) x = __ldg(base + (int64_t)(c0 + c) * P + r1 + 1 + r);
                    float* dst = rows + ((below + r) * nblk + c / kTileC) * kTileStride + c % kTileC;
                    dst[0] = x.x;
                    dst[kTileC] = x.y;
                }
                __syncwarp();
            }
#pragma unroll
            for (int u = 0; u < kTileC; ++u) {
                float tx[kTileC], ty[kTileC];
#pragma unroll
                for (int v = 0; v < kTileC; ++v) {
                    tx[v] = re[u][v];
                    ty[v] = im[u][v];
                }
                own_rows(below + above, u, tx, ty);
#pragma unroll
                for (int v = 0; v < kTileC; ++v) {
                    const int d = (tj - ti) * kTileC + v - u;
                    if (mine && d >= 0 && d < L) band[(ti * kTileC + u) * kBand + d] = make_float2(tx[v], ty[v]);
                }
            }
            const int cnt = __shfl_sync(0xffffffffu, my_cnt, g), l0 = __shfl_sync(0xffffffffu, my_lo, g);
            const int l1 = __shfl_sync(0xffffffffu, my_hi, g) - L + 1;  // subarray starts l0 .. l1
            for (int c = lane; c < M; c += 32) own[c] = __ldg(base + (int64_t)c * P + iz0 + g);
            __syncwarp();
            matrix_of_band(band, lane, L, l0 - c0, l1 - l0 + 1, norm_of(a, cnt, L));
            const float2 z = capon_value(reinterpret_cast<float2 (*)[kBand]>(band), own, a, lane, L, cnt, l0, l1);
            if (lane == 0) out[f * P + ix * a.nz + iz0 + g] = z;
            __syncwarp();
        }
        
    }
}

// More than kTileM channels: one pixel per warp, R summed row by row of the depth window, lane
// d sliding over diagonal d of the row's products (bound by the two shared-memory loads of a
// product, 20 warps per SM).
__host__ __device__ __forceinline__ int row_warp_words(int M) { return (2 * kLMax * kBand + 2 * M + 3) & ~3; }

__global__ void __launch_bounds__(32 * kWarps, 5) capon_rows_kernel(const float2* __restrict__ cube,
                                                                    const float* __restrict__ apod,
                                                                    float2* __restrict__ out, const CaponArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int M = (int)a.M, nz = (int)a.nz;
    float* mine = smem + wi * row_warp_words(M);
    float2 (*R)[kBand] = reinterpret_cast<float2 (*)[kBand]>(mine);
    float2* row = reinterpret_cast<float2*>(mine + 2 * kLMax * kBand);
    const int64_t P = a.nz * a.nx, total = P * a.F;
    for (int64_t t = (int64_t)blockIdx.x * nwarps + wi; t < total; t += (int64_t)gridDim.x * nwarps) {
        const int64_t f = t / P, p = t - f * P;
        const int iz = (int)(p % a.nz);
        const float2* own = cube + f * a.M * P + p;  // [M][P] from this pixel on
        const Aperture q = aperture_of(own, apod + p, M, P, a, lane);
        if (!q.adaptive()) {
            if (lane == 0) out[t] = q.plain();
            continue;
        }
        const int L = q.L, l0 = q.lo, l1 = q.hi - L + 1;
        auto load_row = [&](int r) {  // the row r samples below the pixel's own
            __syncwarp();
            for (int c = q.lo + lane; c <= q.hi; c += 32) row[c] = __ldg(own + (int64_t)c * P + r);
            __syncwarp();
        };
        const int ra = max(0, iz - a.K) - iz, rb = min(nz - 1, iz + a.K) - iz;
        const float norm = norm_of(a, q.cnt, L);
        for (int r = ra; r <= rb; ++r) {
            load_row(r);
            if (lane >= L) continue;
            const float2 *x = row + l0, *y = x + lane;  // products conj(x[l]) y[l]
            auto product = [](float2 u, float2 v) {
                return make_float2(fmaf(u.x, v.x, u.y * v.y), fmaf(u.x, v.y, -(u.y * v.x)));
            };
            const int nl = l1 - l0 + 1;
            auto take = [](float2& g, float2 u, float2 v) {
                g.x = fmaf(u.x, v.x, fmaf(u.y, v.y, g.x));
                g.y = fmaf(u.x, v.y, fmaf(-u.y, v.x, g.y));
            };
            Slide s;  // the first window in blocks of 8 products
            int l = 0;
            for (; l + 8 <= nl; l += 8) {
                float2 g0 = make_float2(0.f, 0.f), g1 = g0;
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    take(g0, x[l + u], y[l + u]);
                    take(g1, x[l + u + 1], y[l + u + 1]);
                }
                s.add(g0.x + g1.x, g0.y + g1.y);
            }
            float2 g0 = make_float2(0.f, 0.f);
            for (; l < nl; ++l) take(g0, x[l], y[l]);
            s.add(g0.x, g0.y);
            for (int i = 0;; ++i) {
                const float2 v = r > ra ? R[i][i + lane] : make_float2(0.f, 0.f);
                R[i][i + lane] = make_float2(fmaf(s.g.x, norm, v.x), fmaf(s.g.y, norm, v.y));
                if (i + 1 + lane >= L) break;
                const float2 add = product(x[nl + i], y[nl + i]), sub = product(x[i], y[i]);
                s.add(add.x - sub.x, add.y - sub.y);
            }
        }
        load_row(0);
        const float2 z = capon_value(R, row, a, lane, L, q.cnt, l0, l1);
        if (lane == 0) out[t] = z;
        __syncwarp();
    }
}

}  // namespace

extern "C" int ustb_capon(const void* cube, const float* apodization, int64_t nz, int64_t nx, int64_t M, int64_t F,
                          float L_elements, int32_t K_samples, float regularisation, float criterion,
                          int32_t forward_backward, void* out, void* stream) {
    ustb::clear_error();
    USTB_REQUIRE(nz >= 0 && nx >= 0 && M >= 0 && F >= 0, USTB_E_SHAPE, "negative size");
    USTB_REQUIRE(M >= 2 && M <= kMMax, USTB_E_SHAPE, "Capon needs 2..%d channels per pixel, got %lld", kMMax,
                 (long long)M);
    USTB_REQUIRE(L_elements >= 1.f, USTB_E_ARG, "L_elements must be >= 1");
    USTB_REQUIRE(K_samples >= 0 && K_samples < 4096, USTB_E_ARG, "K_samples must be in [0, 4096)");
    USTB_REQUIRE(regularisation >= 0.f, USTB_E_ARG, "regularisation must be >= 0");
    if (nz == 0 || nx == 0 || F == 0) return USTB_OK;
    USTB_REQUIRE(cube && apodization && out, USTB_E_ARG, "NULL pointer");
    CaponArgs a;
    a.nz = nz; a.nx = nx; a.F = F; a.M = M;
    a.K = K_samples;
    a.l_frac = L_elements / (float)M;
    a.crit = criterion;
    a.reg = regularisation;
    a.fb = forward_backward ? 1 : 0;
    // the subarray length the active count can produce must fit one warp
    USTB_REQUIRE((int)floorf(a.l_frac * (float)M) <= kLMax, USTB_E_ARG,
                 "L_elements = %g gives subarrays longer than %d", (double)L_elements, kLMax);
    int dev = 0, sms = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    USTB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // neighbouring pixels per warp: they share 2K + 2 - g rows of the Gram matrix and add
    // g - 1 of their own each, so the rows per pixel are (2K + 2 - g) / g + g - 1
    const bool tiles = M <= kTileM;
    a.group = 1;
    if (tiles) {
        auto rows_of = [&](int g) { return (double)(2 * K_samples + 2 - g) / g + g - 1; };
        for (int g = 2; g <= std::min(kGroup, 2 * K_samples + 1); ++g)
            if (rows_of(g) < rows_of(a.group)) a.group = g;
    }
    const int64_t total = (nz + a.group - 1) / a.group * nx * F;
    auto kern = tiles ? capon_kernel : capon_rows_kernel;
    const size_t smem = kWarps * sizeof(float) * (size_t)(tiles ? warp_words((int)M) : row_warp_words((int)M));
    size_t limit = 0;
    const int rc = ustb::shared_limit((const void*)kern, limit);
    if (rc) return rc;
    USTB_REQUIRE(smem <= limit, USTB_E_SHAPE, "%lld channels need %zu bytes of shared memory (limit %zu)", (long long)M,
                 smem, limit);
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((total + kWarps - 1) / kWarps,
                                                                          (int64_t)sms * 64));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    kern<<<grid, 32 * kWarps, smem, s>>>(static_cast<const float2*>(cube), apodization, static_cast<float2*>(out), a);
    USTB_CUDA(cudaGetLastError());
    return USTB_OK;
}

// sm_100a kernels of the spectral correlation form.
//
// The numerator surface of a tile pair, sum_ij r'(i, j) t(u + i, v + j) over every placement, is
// a 2-D correlation; the reference evaluates it as a direct sum (correlate.cu:69-135), which costs
// C^2 R^2 multiply-adds per pair.  Here one CTA per pair does it with FFTs in shared memory:
// the window t (real parts) and the zero-mean chip r' (imaginary parts) share one N x N complex
// tile (N >= W, so no placement wraps around), one forward 2-D transform gives both spectra, their
// product T conj(R) is formed in place and one inverse transform (pruned to the C placement rows)
// returns the numerators.  About 20x fewer operations than the direct sum at the production
// geometry (64^2 chips, 128^2 windows).
//
// Around it: the amplitudes of each raster are detected once (detect_kernel; neighbouring
// windows overlap, so every sample is shared by many pairs) and the correlation kernel takes float
// amplitudes through asynchronous copies.  The placement statistics (1/sigma of every window box)
// come from the window while it sits in shared memory (spec_box_stats), or, for the coarse stage
// of windows that tile a raster, from FP64 sums over the whole raster (raster_stats.cu).
//
// Accuracy.  The window is centred on its mean before the transform (sum r' = 0, so the
// numerators keep their value) and the twiddles are correctly rounded, which keeps the transform
// error of a normalised correlation near 1e-7; the plain form's FP32 direct sums land in the same
// range.  Where a nearly flat box would magnify the transform error, the numerator is recomputed
// as a direct sum (spec_surface).
#include <algorithm>

#include <cuda.h>

#include "fft.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"
#include "tile_common.cuh"

namespace ampcor_b200 {

namespace {

struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// two block-wide FP64 sums in a fixed order (one pair of barriers) over a CTA of NW warps; every
// thread gets both; red holds 2 NW doubles
template <int NW>
__device__ void block_sum2(double& a, double& b, double* red)
{
    a = warp_sum(a);
    b = warp_sum(b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        red[2 * warp] = a;
        red[2 * warp + 1] = b;
    }
    __syncthreads();
    a = 0.0;
    b = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        a += red[2 * w];
        b += red[2 * w + 1];
    }
    __syncthreads();
}

// one warp: the positions of fft::half_positions (one member of every Hermitian pair of the
// permuted spectrum, increasing), 32 candidates per ballot
template <int N1, int N2>
__device__ void build_half(int* half)
{
    constexpr int N = N1 * N2;
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int p0 = 0; p0 < N; p0 += 32) {
        const int p = p0 + lane;
        const bool in = p < N && fft::in_half<N1, N2>(p);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) half[base + __popc(m & ((1u << lane) - 1u))] = p;
        base += __popc(m);
    }
}

__device__ __forceinline__ const float* spec_chip(const SpecSource& s, long long pair0, int b)
{
    return s.chip + (s.chip_off ? s.chip_off[pair0 + b] : (long long)b * s.chip_step);
}

__device__ __forceinline__ const float* spec_win(const SpecSource& s, long long pair0, int b)
{
    return s.win + (s.win_off ? s.win_off[pair0 + b] : (long long)b * s.win_step);
}

// The transform's error on a numerator is a small multiple of eps |r'| |t'| (|.|: Euclidean norms
// of the zero-mean chip and the centred window; below 1.4e-7 |r'| |t'| over the compiled lengths
// in host runs against FP64 sums), so its error on gamma is bounded by kSpecErr |t'| / sigma_box.
// Where a box is nearly flat that bound grows; a placement whose bound exceeds kSpecTol (half the
// 2e-5 surface tolerance the parity tests hold every form to) has its numerator recomputed as a
// direct FP32 sum whenever its value matters (it could be the maximum, or the surface is
// returned).  On speckle the bound is about kSpecErr W / R (|t'| / sigma_box is about W / R, the
// chip blocks of a blocked stage add theirs), 5e-6 for a 32 px chip in a +-64 px search
// (W / R = 5), while the errors measured there stay below 3e-7; zero-padded or masked windows
// exceed it.
constexpr float kSpecErr = 1e-6f;
constexpr float kSpecTol = 1e-5f;

// Scratch of the placement statistics: slot k is z[st k] for k below nz (the imaginary parts of
// the tile while the chip waits in registers, st = 2; or a free stretch of the tile, st = 1), and
// past them it continues in the tail buffer.
struct StatSlots {
    float* z;  // slot 0
    float* tail;
    int nz;
    int st;    // slot stride (floats)
    __device__ __forceinline__ float* at(int k) const { return k < nz ? z + st * k : tail + (k - nz); }
};

__device__ __forceinline__ float box_inv_of(double b1, double b2, double rcells)
{
    const float var = (float)(b2 - b1 * b1 * rcells);
    return var > 0.0f ? __frsqrt_rn(var) : 0.0f;
}

// 1/sigma_box of every placement from the window (win(y, x): the tile's real parts, or a staged
// copy of the window), the values shifted by sx (the window mean: the box variance does not
// change and the column sums keep their digits).  sigma^2 = S2 - S1^2 / R^2 over the R x R box, its sum of squared deviations
// from its mean: the target variance of correlate.cu:196-309, whose box mean comes from the
// summed-area table (tgtStats.cu).
//
// Column sums V(u, x) over window rows [u, u + R), nseg threads per column: thread s sums band s
// of the first placement's rows (FP32 runs of 8 rows added in FP64) and the slides
// delta(i) = t(i + R) - t(i) of its share of the placement rows (FP32: a slide is small next to a
// column sum); after one exchange (part, FP64) each thread starts its share at V(0) plus the
// earlier shares' slides (as a float pair) and adds the FP32 sum of its own slides so far, and
// writes V(u, x) of its rows as floats into the slots (V1 at slot u W + x, V2 at C W + u W + x).
// Then one warp per placement row (three rows at a time) forms the box sums
// S(v) = sum_{x in [v, v + R)} V(x): S(0) as an FP64 warp sum, the others as S(0) plus an FP32 scan
// of V(v + R) - V(v) across the lanes.  The phases are bound by instruction issue, so the FP64
// work and the float-double conversions are kept to a few per column.  Ends with a barrier.
template <int NT, class Win>
__device__ void spec_box_stats(Win win, const SpecGeom& g, float sx, StatSlots vs, double* part,
                               float* invs)
{
    const int R = g.R, W = g.W, C = g.C, nseg = g.nseg, D = C - 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x = tid % W, s = tid / W;
    auto tv = [&](int y) { return win(y, x) - sx; };
    constexpr int kRun = 8;
    if (s < nseg) {
        double b1 = 0.0, b2 = 0.0;
        const int ya = s * R / nseg, yb = (s + 1) * R / nseg;
        for (int y0 = ya; y0 < yb; y0 += kRun) {
            float r1 = 0.0f, r2 = 0.0f;
#pragma unroll
            for (int k = 0; k < kRun; ++k)
                if (y0 + k < yb) {
                    const float t = tv(y0 + k);
                    r1 += t;
                    r2 = fmaf(t, t, r2);
                }
            b1 += (double)r1;
            b2 += (double)r2;
        }
        float e1 = 0.0f, e2 = 0.0f;
        constexpr int kA = 4;  // window rows read ahead of the sums
        for (int i0 = s * D / nseg, i1 = (s + 1) * D / nseg; i0 < i1; i0 += kA) {
            float a[kA], b[kA];
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                const int i = min(i0 + k, i1 - 1);
                a[k] = win(i + R, x);
                b[k] = win(i, x);
            }
#pragma unroll
            for (int k = 0; k < kA; ++k)
                if (i0 + k < i1) {
                    const float d = a[k] - b[k];
                    e1 += d;
                    e2 = fmaf(d, (a[k] + b[k]) - 2.0f * sx, e2);
                }
        }
        part[(0 * nseg + s) * W + x] = b1;
        part[(1 * nseg + s) * W + x] = b2;
        part[(2 * nseg + s) * W + x] = (double)e1;
        part[(3 * nseg + s) * W + x] = (double)e2;
    }
    __syncthreads();
    if (s < nseg) {
        double v1 = 0.0, v2 = 0.0;
        for (int q = 0; q < nseg; ++q) {
            v1 += part[(0 * nseg + q) * W + x];
            v2 += part[(1 * nseg + q) * W + x];
        }
        for (int q = 0; q < s; ++q) {
            v1 += part[(2 * nseg + q) * W + x];
            v2 += part[(3 * nseg + q) * W + x];
        }
        // V(u) = V(start) + P(u), P the FP32 sum of this share's slides so far (small next to
        // V); V(start) as a float pair
        const float h1 = (float)v1, l1 = (float)(v1 - (double)h1);
        const float h2 = (float)v2, l2 = (float)(v2 - (double)h2);
        float p1 = 0.0f, p2 = 0.0f;
        const int i1 = (s + 1) * D / nseg;
        constexpr int kB = 4;  // window rows read ahead of the running sums
        for (int i0 = s * D / nseg; i0 < i1; i0 += kB) {
            float a[kB], b[kB];
#pragma unroll
            for (int k = 0; k < kB; ++k) {
                const int i = min(i0 + k, i1 - 1);
                a[k] = win(i + R, x);
                b[k] = win(i, x);
            }
#pragma unroll
            for (int k = 0; k < kB; ++k)
                if (i0 + k < i1) {
                    *vs.at((i0 + k) * W + x) = h1 + (l1 + p1);
                    *vs.at((C + i0 + k) * W + x) = h2 + (l2 + p2);
                    const float d = a[k] - b[k];
                    p1 += d;
                    p2 = fmaf(d, (a[k] + b[k]) - 2.0f * sx, p2);
                }
        }
        if (s == nseg - 1) {
            *vs.at(D * W + x) = h1 + (l1 + p1);
            *vs.at((C + D) * W + x) = h2 + (l2 + p2);
        }
    }
    __syncthreads();
    const double rcells = 1.0 / ((double)R * (double)R);
    // KR placement rows per warp at a time, u0, u0 + NW, ...; rows past the end repeat row C - 1
    // (not stored), so that every warp runs one pass for C <= KR NW
    constexpr int NW = NT / 32, KR = 3;
    for (int u0 = warp; u0 < C; u0 += KR * NW) {
        int uu[KR];
        bool keep[KR];
#pragma unroll
        for (int r = 0; r < KR; ++r) {
            uu[r] = min(u0 + r * NW, C - 1);
            keep[r] = u0 + r * NW < C;
        }
        double s1[KR], s2[KR];
#pragma unroll
        for (int r = 0; r < KR; ++r) {
            float f1 = 0.0f, f2 = 0.0f;
            for (int c = lane; c < R; c += 32) {
                f1 += *vs.at(uu[r] * W + c);
                f2 += *vs.at((C + uu[r]) * W + c);
            }
            s1[r] = (double)f1;
            s2[r] = (double)f2;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < KR; ++r) {
                s1[r] += __shfl_xor_sync(kFull, s1[r], o);
                s2[r] += __shfl_xor_sync(kFull, s2[r], o);
            }
        if (lane == 0)
#pragma unroll
            for (int r = 0; r < KR; ++r)
                if (keep[r]) invs[uu[r] * C] = box_inv_of(s1[r], s2[r], rcells);
        for (int j0 = 0; j0 < D; j0 += 32) {
            const int j = j0 + lane;
            float i1[KR], i2[KR];
#pragma unroll
            for (int r = 0; r < KR; ++r) {
                i1[r] = 0.0f;
                i2[r] = 0.0f;
                if (j < D) {
                    i1[r] = *vs.at(uu[r] * W + j + R) - *vs.at(uu[r] * W + j);
                    i2[r] = *vs.at((C + uu[r]) * W + j + R) - *vs.at((C + uu[r]) * W + j);
                }
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int r = 0; r < KR; ++r) {
                    const float y1 = __shfl_up_sync(kFull, i1[r], o);
                    const float y2 = __shfl_up_sync(kFull, i2[r], o);
                    if (lane >= o) {
                        i1[r] += y1;
                        i2[r] += y2;
                    }
                }
            if (j < D)
#pragma unroll
                for (int r = 0; r < KR; ++r)
                    if (keep[r])
                        invs[uu[r] * C + j + 1] = box_inv_of(s1[r] + (double)i1[r], s2[r] + (double)i2[r], rcells);
#pragma unroll
            for (int r = 0; r < KR; ++r) {
                s1[r] += (double)__shfl_sync(kFull, i1[r], 31);
                s2[r] += (double)__shfl_sync(kFull, i2[r], 31);
            }
        }
    }
    __syncthreads();
}

// two floats at a time
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t pk_of(float x, float y)
{
    return (pair_t)__float_as_uint(x) | (pair_t)__float_as_uint(y) << 32;
}
__device__ __forceinline__ float pk_lo(pair_t v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float pk_hi(pair_t v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ pair_t pk_add(pair_t a, pair_t b)
{
    pair_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair_t pk_sub(pair_t a, pair_t b)
{
    pair_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair_t pk_fma(pair_t a, pair_t b, pair_t c)
{
    pair_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// spec_box_stats for a staged refined window (W dense floats a row, W a multiple of 4): the same sums
// in the same precision, two columns to a thread in packed FP32, and the box sums' first warp sum
// carries both moments at once (one half of the warp each).  V: 2 C W floats, part: 4 nseg W
// doubles, both in the tile's first bytes.  Clock stamps at the production geometry: 10.7K cycles a
// pair (3.0K, 2.9K and 4.7K in its three phases) against 13.1K of spec_box_stats on the same copy.
template <int NT>
__device__ void staged_box_stats(const float* win, const SpecGeom& g, float sx, float* V, double* part, float* invs)
{
    const int R = g.R, W = g.W, C = g.C, nseg = g.nseg, D = C - 1, W2 = W >> 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = tid / W2, x = 2 * (tid - s * W2);
    const pair_t* col = reinterpret_cast<const pair_t*>(win + x);
    const pair_t msx = pk_of(-sx, -sx), m2sx = pk_of(-2.0f * sx, -2.0f * sx);
    const int d0 = s * D / nseg, d1 = (s + 1) * D / nseg;
    constexpr int kRun = 8, kA = 4;
    if (s < nseg) {
        double b1x = 0.0, b1y = 0.0, b2x = 0.0, b2y = 0.0;
        for (int y0 = s * R / nseg, y1 = (s + 1) * R / nseg; y0 < y1; y0 += kRun) {
            pair_t r1 = 0, r2 = 0;
#pragma unroll
            for (int k = 0; k < kRun; ++k)
                if (y0 + k < y1) {
                    const pair_t t = pk_add(col[(y0 + k) * W2], msx);
                    r1 = pk_add(r1, t);
                    r2 = pk_fma(t, t, r2);
                }
            b1x += (double)pk_lo(r1);
            b1y += (double)pk_hi(r1);
            b2x += (double)pk_lo(r2);
            b2y += (double)pk_hi(r2);
        }
        pair_t e1 = 0, e2 = 0;
        for (int i0 = d0; i0 < d1; i0 += kA) {
            pair_t a[kA], b[kA];
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                const int i = min(i0 + k, d1 - 1);
                a[k] = col[(i + R) * W2];
                b[k] = col[i * W2];
            }
#pragma unroll
            for (int k = 0; k < kA; ++k)
                if (i0 + k < d1) {
                    const pair_t d = pk_sub(a[k], b[k]);
                    e1 = pk_add(e1, d);
                    e2 = pk_fma(d, pk_add(pk_add(a[k], b[k]), m2sx), e2);
                }
        }
        double2* out = reinterpret_cast<double2*>(part + s * W + x);
        out[0 * nseg * W2] = make_double2(b1x, b1y);
        out[1 * nseg * W2] = make_double2(b2x, b2y);
        out[2 * nseg * W2] = make_double2((double)pk_lo(e1), (double)pk_hi(e1));
        out[3 * nseg * W2] = make_double2((double)pk_lo(e2), (double)pk_hi(e2));
    }
    __syncthreads();
    if (s < nseg) {
        double v1x = 0.0, v1y = 0.0, v2x = 0.0, v2y = 0.0;
        auto take = [&](int q, int k) {
            const double2 p1 = *reinterpret_cast<const double2*>(part + (q * nseg + k) * W + x);
            const double2 p2 = *reinterpret_cast<const double2*>(part + ((q + 1) * nseg + k) * W + x);
            v1x += p1.x;
            v1y += p1.y;
            v2x += p2.x;
            v2y += p2.y;
        };
        for (int k = 0; k < nseg; ++k) take(0, k);
        for (int k = 0; k < s; ++k) take(2, k);
        const float h1x = (float)v1x, h1y = (float)v1y, h2x = (float)v2x, h2y = (float)v2y;
        const pair_t h1 = pk_of(h1x, h1y), l1 = pk_of((float)(v1x - (double)h1x), (float)(v1y - (double)h1y));
        const pair_t h2 = pk_of(h2x, h2y), l2 = pk_of((float)(v2x - (double)h2x), (float)(v2y - (double)h2y));
        pair_t p1 = 0, p2 = 0;
        pair_t* o1 = reinterpret_cast<pair_t*>(V + x);
        pair_t* o2 = reinterpret_cast<pair_t*>(V + C * W + x);
        for (int i0 = d0; i0 < d1; i0 += kA) {
            pair_t a[kA], b[kA];
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                const int i = min(i0 + k, d1 - 1);
                a[k] = col[(i + R) * W2];
                b[k] = col[i * W2];
            }
#pragma unroll
            for (int k = 0; k < kA; ++k)
                if (i0 + k < d1) {
                    o1[(i0 + k) * W2] = pk_add(h1, pk_add(l1, p1));
                    o2[(i0 + k) * W2] = pk_add(h2, pk_add(l2, p2));
                    const pair_t d = pk_sub(a[k], b[k]);
                    p1 = pk_add(p1, d);
                    p2 = pk_fma(d, pk_add(pk_add(a[k], b[k]), m2sx), p2);
                }
        }
        if (s == nseg - 1) {
            o1[D * W2] = pk_add(h1, pk_add(l1, p1));
            o2[D * W2] = pk_add(h2, pk_add(l2, p2));
        }
    }
    __syncthreads();
    const double rcells = 1.0 / ((double)R * (double)R);
    constexpr int NW = NT / 32, KR = 3;
    for (int u0 = warp; u0 < C; u0 += KR * NW) {
        const float* row1[KR];
        float* to[KR];
        bool keep[KR];
        double m[KR];  // lanes below 16: the first box's sum, the others: its sum of squares
#pragma unroll
        for (int r = 0; r < KR; ++r) {
            const int u = min(u0 + r * NW, C - 1);
            row1[r] = V + u * W;
            to[r] = invs + u * C;
            keep[r] = u0 + r * NW < C;
            float f1 = 0.0f, f2 = 0.0f;
            for (int c = lane; c < R; c += 32) {
                f1 += row1[r][c];
                f2 += row1[r][C * W + c];
            }
            const double mine = lane < 16 ? f1 : f2, other = lane < 16 ? f2 : f1;
            m[r] = mine + __shfl_xor_sync(kFull, other, 16);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < KR; ++r) m[r] += __shfl_xor_sync(kFull, m[r], o);
        double s1[KR], s2[KR];
#pragma unroll
        for (int r = 0; r < KR; ++r) {
            s1[r] = __shfl_sync(kFull, m[r], 0);
            s2[r] = __shfl_sync(kFull, m[r], 16);
            if (lane == 0 && keep[r]) to[r][0] = box_inv_of(s1[r], s2[r], rcells);
        }
        for (int j0 = 0; j0 < D; j0 += 32) {
            const int j = j0 + lane;
            float i1[KR], i2[KR];
#pragma unroll
            for (int r = 0; r < KR; ++r) {
                i1[r] = j < D ? row1[r][j + R] - row1[r][j] : 0.0f;
                i2[r] = j < D ? row1[r][C * W + j + R] - row1[r][C * W + j] : 0.0f;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int r = 0; r < KR; ++r) {
                    const float y1 = __shfl_up_sync(kFull, i1[r], o);
                    const float y2 = __shfl_up_sync(kFull, i2[r], o);
                    if (lane >= o) {
                        i1[r] += y1;
                        i2[r] += y2;
                    }
                }
#pragma unroll
            for (int r = 0; r < KR; ++r)
                if (j < D && keep[r])
                    to[r][j + 1] = box_inv_of(s1[r] + (double)i1[r], s2[r] + (double)i2[r], rcells);
            if (j0 + 32 < D)
#pragma unroll
                for (int r = 0; r < KR; ++r) {
                    s1[r] += (double)__shfl_sync(kFull, i1[r], 31);
                    s2[r] += (double)__shfl_sync(kFull, i2[r], 31);
                }
        }
    }
    __syncthreads();
}

// The normalised surface G (C x C in shared memory, formed by the last transform step) -> its
// first maximum (valid in every thread) and optional copies; a CTA of NT threads, red holding
// NT / 32 floats and as many ints.  On entry every thread holds the
// maximum of the placements it formed whose transform bound is tight, and whether it formed any
// whose bound is loose (flagged); inv holds 1/sigma_box of the placements (row stride C).
template <int NT>
__device__ void spec_surface(float* G, double* red, const SpecGeom& g, const float* inv,
                             float inv_sigma, double mean_c, float ebox, const float* chip,
                             long long cs, const float* win, long long ws, float* out1, float* out2,
                             float& bv, int& bi, int flagged)
{
    const int C = g.C, R = g.R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    block_argmax_n<NT>(bv, bi, reinterpret_cast<float*>(red), reinterpret_cast<int*>(red) + NT / 32);
    if (__syncthreads_or(flagged)) {
        // direct FP32 numerators where the transform's bound is loose and the value matters: one
        // warp per placement, lanes across the chip columns
        const bool all = out1 || out2;
        float wv = -INFINITY;
        int wi = INT_MAX;
        for (int idx = warp; idx < C * C; idx += NT / 32) {
            const int u = idx / C, v = idx - u * C;
            const float inv_box = inv[idx];
            const float e = ebox * inv_box;
            if (!(e > kSpecTol) || !(all || G[idx] + e >= bv)) continue;
            // the window less the box's own mean (sum r' (t - c) = sum r' t for any constant c):
            // the FP32 sums round on the box's variation, not on its level, and an all-zero box
            // keeps a numerator of exactly zero
            float sb = 0.0f;
            for (int i = 0; i < R; ++i)
                for (int j = lane; j < R; j += 32) sb += __ldg(win + (u + i) * ws + v + j);
            const float wsh = (float)(warp_sum((double)sb) / ((double)R * (double)R));
            float acc = 0.0f;
            for (int i = 0; i < R; ++i)
                for (int j = lane; j < R; j += 32) {
                    const float rp = (float)((double)__ldg(chip + i * cs + j) - mean_c);
                    acc = fmaf(rp, __ldg(win + (u + i) * ws + v + j) - wsh, acc);
                }
            const double num = warp_sum((double)acc);
            const float gv = (float)num * inv_box * inv_sigma;
            __syncwarp();
            if (lane == 0) G[idx] = gv;
            better(wv, wi, gv, idx);
        }
        // every flagged placement that could win has its exact value now; the others stay below
        // the unflagged maximum
        better(bv, bi, wv, wi);
        block_argmax_n<NT>(bv, bi, reinterpret_cast<float*>(red), reinterpret_cast<int*>(red) + NT / 32);
    }
    if (out1 || out2) {
        for (int idx = threadIdx.x; idx < C * C; idx += NT) {
            const float gv = G[idx];
            if (out1) out1[idx] = gv;
            if (out2) out2[idx] = gv;
        }
    }
}

// the stage's result of pair p from the first maximum bv at placement bi: the coarse cell and its
// nudged refinement corners (stage 0), or the refined cell and peak (stage 1)
__device__ void spec_result(const SpecOut& out, long long p, int R, int W, int C, float bv, int bi)
{
    const int u = bi / C, v = bi - u * C;
    if (out.stage == 0) {
        out.coarse[p] = nudged(u, v, R, W, out.m);
        out.coarse_peak[p] = bv;
    } else {
        out.fine[p] = FineOut{u, v, bv, 0.0f};
    }
}

template <int N1, int N2>
__global__ void __launch_bounds__(kSpecThreads, 1)
spec_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, SpecGeom g,
            InvSource inv, const float2* tw_g, SpecOut out)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    if (blockIdx.x >= pairs) return;
    const long long p = pair0 + blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (valid[p] < 0) {
        if (out.stage == 0 && tid == 0) {
            out.coarse[p] = CoarseOut{-1, -1, -1, -1};
            out.coarse_peak[p] = NAN;
        }
        return;
    }
    constexpr int N = N1 * N2;
    // the tile's row stride is always N + 1 (odd); as a constant every element offset of a row or
    // column walk is an immediate
    constexpr int RS = N + 1;
    const int W = g.W, R = g.R, C = g.C;
    float2* Z = reinterpret_cast<float2*>(ssm + g.off_z);
    float2* tw = reinterpret_cast<float2*>(ssm + g.off_tw);
    int* neg = reinterpret_cast<int*>(ssm + g.off_neg);
    int* half = reinterpret_cast<int*>(ssm + g.off_half);
    double* red = reinterpret_cast<double*>(ssm + g.off_red);
    float* invs = reinterpret_cast<float*>(ssm + g.off_inv);
    float* G = reinterpret_cast<float*>(ssm + g.off_gam);
    float* Zf = reinterpret_cast<float*>(Z);
    // placement statistics: given (inv.base), else computed here from the window
    const float* inv_b = !inv.base ? nullptr : inv.off ? inv.base + inv.off[p] : inv.base + (long long)blockIdx.x * C * C;
    const long long is = inv.off ? inv.stride : C;
    const float* chip = spec_chip(src, pair0, blockIdx.x);
    const float* win = spec_win(src, pair0, blockIdx.x);
    const long long cs = src.chip_stride, ws = src.win_stride;

    // The chip goes to registers (its loads in flight with the window's), the window amplitudes
    // to the real parts of the tile by 4-byte asynchronous copies, zeros to the other real parts.
    // The imaginary parts are the placement statistics' scratch until the chip is stored there.
    constexpr int JN = (N + kSpecWarps - 1) / kSpecWarps, IN = (N + 31) / 32;
    float cr[JN][IN];
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const int y = warp + kSpecWarps * j, x = lane + 32 * i;
            cr[j][i] = y < R && x < R ? __ldg(chip + y * cs + x) : 0.0f;
        }
    for (int y = warp; y < N; y += kSpecWarps) {
        float* zr = Zf + 2 * y * RS;
        for (int x = lane; x < N; x += 32) {
            if (y < W && x < W)
                cp_async4(zr + 2 * x, win + y * ws + x);
            else
                zr[2 * x] = 0.0f;
        }
    }
    // given placement statistics land in shared memory with the window
    if (inv_b)
        for (int u = warp; u < C; u += kSpecWarps)
            for (int v = lane; v < C; v += 32) cp_async4(invs + u * C + v, inv_b + u * is + v);
    for (int k = tid; k < N; k += kSpecThreads) {
        tw[k] = __ldg(tw_g + k);
        neg[k] = fft::neg_pos<N1, N2>(k);
    }
    if (warp == 0) build_half<N1, N2>(half);
    cp_async_wait_all();
    __syncthreads();

    // Two sweeps of sums, each combined across the block in FP64 (refStats.cu:118-302).  The first
    // takes the chip's sum (compensated) and, about a pivot k (the window's first sample), the
    // window's sums of t - k and (t - k)^2; the second the chip's sum of squares with its FP64
    // mean off (two floats, so that r' carries the FP64 mean; r' stays in the registers): |r'|
    // exactly, where squares of the uncentred amplitudes would cancel in proportion to the squared
    // level of a strong steady return.  The window mean comes off as the first transform pass reads
    // the tile; it only conditions the transform.  |t'|^2 only scales the transform's error bound,
    // so it is taken as an upper bound: sum (t - k)^2 - (sum (t - k))^2 / W^2 plus 1e-5 sum (t - k)^2,
    // more than the FP32 rounding of the per-thread sums (at most 50 terms each, 3e-6 relative).
    double acc4[4];
    const float pk = Z[0].x;
    {
        float sw = 0.0f, sw2 = 0.0f, sc = 0.0f, cc = 0.0f;
        for (int y = warp; y < W; y += kSpecWarps) {
            const float2* zr = Z + y * RS;
            for (int x = lane; x < W; x += 32) {
                const float t = zr[x].x - pk;
                sw += t;
                sw2 = fmaf(t, t, sw2);
            }
        }
        // register slots past the chip hold zeros in every lane: skipped (warp-uniform tests)
#pragma unroll
        for (int j = 0; j < JN; ++j)
            if (warp + kSpecWarps * j < R)
#pragma unroll
                for (int i = 0; i < IN; ++i)
                    if (32 * i < R) {
                        const float yk = cr[j][i] - cc;
                        const float tk = sc + yk;
                        cc = (tk - sc) - yk;
                        sc = tk;
                    }
        acc4[0] = (double)sc - (double)cc;
        acc4[1] = sw;
        acc4[3] = sw2;
        block_sum2<kSpecWarps>(acc4[0], acc4[1], red);
    }
    const double cells_c = (double)R * (double)R, cells_w = (double)W * (double)W;
    const double mean_c = acc4[0] / cells_c;
    const double mean_w = (double)pk + acc4[1] / cells_w;
    const float mc_hi = (float)mean_c, mc_lo = (float)(mean_c - (double)mc_hi);
    const fft::Centre centre{(float)mean_w, W};
    {
        float sc2 = 0.0f;
#pragma unroll
        for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int i = 0; i < IN; ++i)
                if (warp + kSpecWarps * j < R && lane + 32 * i < R) {
                    const float r = (cr[j][i] - mc_hi) - mc_lo;
                    cr[j][i] = r;
                    sc2 = fmaf(r, r, sc2);
                }
        acc4[2] = sc2;
        block_sum2<kSpecWarps>(acc4[2], acc4[3], red);
    }
    const double ss = acc4[2];
    const double st = fmax(acc4[3] - acc4[1] * acc4[1] / cells_w, 0.0) + 1e-5 * acc4[3];
    const float inv_sigma = ss > 0.0 ? (float)(1.0 / sqrt(ss)) : 0.0f;
    if (!inv_b) {
        double* part = reinterpret_cast<double*>(ssm + g.off_gam);
        const StatSlots vs{Zf + 1, reinterpret_cast<float*>(part + 4 * g.nseg * W), N * RS, 2};
        spec_box_stats<kSpecThreads>([&](int y, int x) { return Z[y * RS + x].x; }, g, centre.sx, vs,
                                     part, invs);
    }
    // the zero-mean chip into the imaginary parts, zeros around it
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const int y = warp + kSpecWarps * j, x = lane + 32 * i;
            if (y < N && x < N) Zf[2 * (y * RS + x) + 1] = y < R && x < R ? cr[j][i] : 0.0f;
        }
    __syncthreads();

    // the last transform step forms gamma of every placement straight from its outputs and keeps
    // this thread's maximum of those whose transform bound is tight
    const float scale = (float)(1.0 / (4.0 * (double)N * (double)N));
    const float ebox = kSpecErr * (float)sqrt(st);
    float bv = -INFINITY;
    int bi = INT_MAX;
    int flagged = 0;
    fft::correlate_tile<N1, N2>(Z, RS, W, C, tw, neg, half, centre, tid, kSpecThreads, BlockSync{},
                                [&](int u, int v, float2 val) {
                                    if (v < C) {
                                        const int idx = u * C + v;
                                        const float inv_box = invs[idx];
                                        const float gv = val.x * scale * inv_box * inv_sigma;
                                        G[idx] = gv;
                                        if (ebox * inv_box > kSpecTol)
                                            flagged = 1;
                                        else
                                            better(bv, bi, gv, idx);
                                    }
                                });

    float* surf = out.surfaces ? out.surfaces + (size_t)p * C * C : nullptr;
    float* gam = out.stage == 1 ? out.gam + (long long)blockIdx.x * C * C : nullptr;
    spec_surface<kSpecThreads>(G, red, g, invs, inv_sigma, mean_c, ebox, chip, cs, win, ws, gam, surf, bv, bi, flagged);
    if (tid == 0) spec_result(out, p, R, W, C, bv, bi);
}

// ------------------------------------------------------------------------------------------
// staged spectral correlation: one resident CTA per SM walks the pairs of a chunk
// ------------------------------------------------------------------------------------------
//
// spec_kernel holds one CTA per SM (its tile fills the shared memory), so nothing hides the wait
// for its tiles or the two sweeps of block sums that precede the transform; clock stamps put them
// at a third of the fine stage.  Here a CTA stays resident and walks pairs blockIdx.x,
// blockIdx.x + gridDim.x, ...: once a pair's inverse column pass is done (from then on its
// correlation touches only the tile's first rows) the bulk-copy engine brings the next pair's
// window (W x W dense floats, one cp.async.bulk completing on an mbarrier) into the tile's last
// bytes, and the chip's bytes are sent toward L2.  The statistics of the refined chips and windows
// come from the refinement, which forms them on the way out; a raster's chip is summed here, from the
// amplitudes that are correlated.  A pair starts with its
// window in shared memory: the placement statistics of a refined window read from the staged copy
// (the tile's first bytes are their scratch), then one pass that writes the window and the chip
// (loaded from L2 meanwhile) into the tile; the first transform pass takes the window's mean (and
// a refined chip's) off.  Every wait is bounded; one that runs out is counted in errs, the CTA lets
// the copy in flight land (again bounded) and returns.

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes)
                 : "memory");
}

// bytes (a multiple of 16) from global src to shared dst, both 16-byte aligned; completes on bar
__device__ __forceinline__ void bulk_to_smem(void* dst, const void* src, unsigned bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     saddr(dst)),
                 "l"(src), "r"(bytes), "r"(saddr(bar))
                 : "memory");
}

__device__ __forceinline__ void bulk_prefetch_l2(const void* src, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// the box of a 2-D tensor map at (x, y) (x a multiple of 4 floats) into shared dst; completes on bar
__device__ __forceinline__ void tensor_to_smem(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            saddr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(saddr(bar))
        : "memory");
}

// the same of a 3-D map at (x, y, z)
__device__ __forceinline__ void tensor3_to_smem(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            saddr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(saddr(bar))
        : "memory");
}

__device__ __forceinline__ void tensor3_prefetch_l2(const CUtensorMap* map, int x, int y, int z)
{
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(z)
                 : "memory");
}

__device__ __forceinline__ void tensor_prefetch_l2(const CUtensorMap* map, int x, int y)
{
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y)
                 : "memory");
}

// RASTER false: the refined tiles, every pair's window W x W dense floats on a 16-byte boundary
// (one copy), its statistics formed here; RASTER true: windows cut from a raster, copied as the
// box of wmap (stage_rs x W floats) whose first column is the 16-byte boundary at or before the
// window's first sample, with the box of the raster's statistics (imap, inv_rs x C floats) at the
// same corner, the chip's box of cmap sent toward L2
template <int N1, int N2, bool RASTER, int NT, int CTAS>
__global__ void __launch_bounds__(NT, CTAS)
spec_staged_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, SpecGeom g,
                   InvSource inv, const float2* tw_g, SpecOut out, const TileStat* cstat, const TileStat* wstat,
                   unsigned int* errs, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap cmap,
                   const __grid_constant__ CUtensorMap imap, int stall)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    constexpr int NW = NT / 32;
    constexpr int N = N1 * N2;
    constexpr int RS = N + 1;
    constexpr int JN = (N + NW - 1) / NW, IN = (N + 31) / 32;
    constexpr int PJ = 5;  // row groups of a piece read whole before it is written
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = g.W, R = g.R, C = g.C, SW = g.stage_rs;
    float2* Z = reinterpret_cast<float2*>(ssm + g.off_z);
    float* Zf = reinterpret_cast<float*>(Z);
    float2* tw = reinterpret_cast<float2*>(ssm + g.off_tw);
    int* neg = reinterpret_cast<int*>(ssm + g.off_neg);
    int* half = reinterpret_cast<int*>(ssm + g.off_half);
    double* red = reinterpret_cast<double*>(ssm + g.off_red);
    float* invs = reinterpret_cast<float*>(ssm + g.off_inv);
    float* G = reinterpret_cast<float*>(ssm + g.off_gam);
    float* stage = reinterpret_cast<float*>(ssm + g.off_stage);
    float* inv_raw = reinterpret_cast<float*>(ssm + g.off_inv_raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(ssm + g.off_bar);
    int& s_err = *reinterpret_cast<int*>(ssm + g.off_bar + 8);  // a wait ran out (CTA-wide)
    const long long cs = src.chip_stride, ws = src.win_stride;
    const int jA = g.stage_y0 / NW;

    for (int k = tid; k < N; k += NT) {
        tw[k] = __ldg(tw_g + k);
        neg[k] = fft::neg_pos<N1, N2>(k);
    }
    if (warp == 0) build_half<N1, N2>(half);
    if (tid == 0) {
        s_err = 0;
        mbar_init(bar, 1);
        mbar_init(bar + 2, 1);  // completed by nothing: the wait of a failure-detection test
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // a failure-detection test: before any copy is issued, every thread waits on a barrier that
    // nothing completes; the bounded wait runs out, sets the error flag, and the CTA skips its
    // pairs and reports the time-out like any other expired wait
    if (stall) {
        mbar_wait(bar + 2, 0u, &s_err, kStallCycles);
        __syncthreads();
    }
    // Lane 0 of warp 0 brings in the windows: `look` finds out early where chunk pair b's tiles lie
    // (loads and divisions whose latency must not hold up the copy), `issue` copies its window into
    // the staging bytes and sends its chip toward L2.  A pair without tiles (its offsets are -1)
    // copies nothing and completes the phase at once.
    bool next_ok = false;
    int nwx = 0, nwy = 0, ncx = 0, ncy = 0;
    auto look = [&](long long b) {
        next_ok = valid[pair0 + b] >= 0;
        if constexpr (RASTER) {
            if (!next_ok) return;
            const long long wo = src.win_off[pair0 + b], co = src.chip_off[pair0 + b];
            nwy = (int)(wo / ws);
            nwx = (int)(wo - (long long)nwy * ws);
            ncy = (int)(co / cs);
            ncx = (int)(co - (long long)ncy * cs);
        }
    };
    auto issue = [&](long long b) {
        if (!next_ok) {
            mbar_arrive(bar);
            return;
        }
        if constexpr (!RASTER) {
            const unsigned bytes = (unsigned)W * (unsigned)W * 4u;
            mbar_expect_tx(bar, bytes);
            bulk_to_smem(stage, spec_win(src, pair0, b), bytes, bar);
            bulk_prefetch_l2(spec_chip(src, pair0, b), (unsigned)R * (unsigned)cs * 4u);
        } else {
            mbar_expect_tx(bar, ((unsigned)W * (unsigned)SW + (unsigned)C * (unsigned)g.inv_rs) * 4u);
            tensor_to_smem(stage, &wmap, nwx & ~3, nwy, bar);
            tensor_to_smem(inv_raw, &imap, nwx & ~3, nwy, bar);
            tensor_prefetch_l2(&cmap, ncx & ~3, ncy);
        }
    };
    const bool run = !stall || !s_err;
    if (tid == 0 && blockIdx.x < pairs && run) {
        look(blockIdx.x);
        issue(blockIdx.x);
    }
    uint32_t parity = 0;
    bool inflight = blockIdx.x < pairs && run;
    long long b_left = blockIdx.x;  // (raster windows) the first pair left without a result
    for (long long b = blockIdx.x; b < pairs && run; b += gridDim.x) {
        const long long p = pair0 + b;
        const long long bn = b + gridDim.x;
        const bool ok = valid[p] >= 0;
        const float* chip = spec_chip(src, pair0, b);
        const float* win = spec_win(src, pair0, b);
        // refined tiles: the chip's mean and 1/|r'|, the window's mean and |t'|
        double mean_c = 0.0;
        float inv_sigma = 0.0f, sx = 0.0f, norm_w = 0.0f;
        if constexpr (!RASTER) {
            mean_c = cstat[b].mean;
            inv_sigma = (float)cstat[b].inv_norm;
            sx = (float)wstat[b].mean;
            norm_w = (float)wstat[b].norm;
        }
        const bool landed = mbar_wait(bar, parity, &s_err);
        if (__syncthreads_or(!landed)) {
            if constexpr (RASTER) b_left = b;
            break;
        }
        parity ^= 1u;
        inflight = false;
        if (tid == 0 && bn < pairs) look(bn);
        if (!ok) {
            if (out.stage == 0 && tid == 0) {
                out.coarse[p] = CoarseOut{-1, -1, -1, -1};
                out.coarse_peak[p] = NAN;
            }
            if (bn < pairs) {
                fence_async_smem();
                __syncthreads();
                if (tid == 0) issue(bn);
                inflight = true;
            }
            continue;
        }
        // window sample (y, x) in the staging bytes: the box starts xo samples before the window
        const int xo = RASTER ? (int)((src.win_off[p] % ws) & 3) : 0;
        // the chip to registers: for a raster window at once (its loads in flight while the
        // statistics are moved and its sum taken before the tile is written), for the refined
        // tiles after the statistics (registers are short there)
        float cr[JN][IN];
        auto load_chip = [&]() {
#pragma unroll
            for (int j = 0; j < JN; ++j)
#pragma unroll
                for (int i = 0; i < IN; ++i) {
                    const int y = warp + NW * j, x = lane + 32 * i;
                    cr[j][i] = y < R && x < R ? __ldg(chip + y * cs + x) : 0.0f;
                }
        };
        if constexpr (RASTER) {
            load_chip();
            // the raster's placement statistics, copied with the window, into their C x C layout
            for (int u = warp; u < C; u += NW)
                for (int v = lane; v < C; v += 32) invs[u * C + v] = inv_raw[u * g.inv_rs + xo + v];
            // the chip's FP64 mean (spec_kernel's first sweep)
            double c1 = 0.0;
#pragma unroll
            for (int j = 0; j < JN; ++j)
                if (warp + NW * j < R)
#pragma unroll
                    for (int i = 0; i < IN; ++i)
                        if (32 * i < R) c1 += (double)cr[j][i];
            c1 = warp_sum(c1);
            if (lane == 0) red[warp] = c1;
            __syncthreads();
            double t1 = 0.0;
#pragma unroll
            for (int w = 0; w < NW; ++w) t1 += red[w];
            mean_c = t1 / ((double)R * (double)R);
            __syncthreads();
        }
        const float mc_hi = (float)mean_c, mc_lo = (float)(mean_c - (double)mc_hi);
        auto wat = [&](int y, int x) {
            if constexpr (RASTER)
                return stage[y * SW + xo + x];
            else
                return stage[y * W + x];
        };

        // placement statistics of a refined window from the staged copy; their scratch is the
        // tile's first bytes
        if constexpr (!RASTER)
            staged_box_stats<NT>(stage, g, sx, Zf, reinterpret_cast<double*>(Zf + ((2 * C * W + 3) & ~3)), invs);

        // window (real parts) and chip (imaginary parts; its bytes were sent toward L2 with the
        // window) into the tile, zeros around them.  Raster windows: the chip goes in zero-mean and
        // |r'|^2 is summed from the very values that go in, as spec_kernel sums it; the window's sums of
        // t - k and (t - k)^2 about a pivot k (its first sample) are taken on the way, as spec_kernel
        // takes them (in another order).  Refined tiles: the first transform pass takes the chip's
        // mean off.
        const float pk = wat(0, 0);
        if constexpr (!RASTER) load_chip();
        float sw = 0.0f, sw2 = 0.0f, sc2 = 0.0f;
        auto put = [&](int j, int i, float t) {
            const int y = warp + NW * j, x = lane + 32 * i;
            if (y < N && x < N) {
                float c = cr[j][i];
                if constexpr (RASTER) {
                    if (y < R && x < R) {
                        c = (c - mc_hi) - mc_lo;
                        sc2 = fmaf(c, c, sc2);
                    }
                    if (y < W && x < W) {
                        const float d = t - pk;
                        sw += d;
                        sw2 = fmaf(d, d, sw2);
                    }
                }
                Z[y * RS + x] = make_float2(t, c);
            }
        };
        auto staged = [&](int j, int i) {
            const int y = warp + NW * j, x = lane + 32 * i;
            return y < W && x < W ? wat(y, x) : 0.0f;
        };
        // rows below stage_y0 lie below the staged bytes: written as they are read
#pragma unroll
        for (int j = 0; j < JN; ++j)
            if (j < jA)
#pragma unroll
                for (int i = 0; i < IN; ++i) put(j, i, staged(j, i));
        __syncthreads();
        // the others cover staged bytes: each piece is read whole, then written (a piece's rows
        // never reach the staged rows of a later piece)
#pragma unroll
        for (int j0 = 0; j0 < JN; j0 += PJ) {
            if (j0 + PJ <= jA) continue;
            float v[PJ][IN];
#pragma unroll
            for (int q = 0; q < PJ; ++q)
#pragma unroll
                for (int i = 0; i < IN; ++i) v[q][i] = j0 + q < JN && j0 + q >= jA ? staged(j0 + q, i) : 0.0f;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < PJ; ++q)
                if (j0 + q < JN && j0 + q >= jA)
#pragma unroll
                    for (int i = 0; i < IN; ++i) put(j0 + q, i, v[q][i]);
        }
        fft::Centre centre{sx, W};
        if constexpr (RASTER) {
            const double d0 = warp_sum((double)sc2), d1 = warp_sum((double)sw), d2 = warp_sum((double)sw2);
            if (lane == 0) {
                red[3 * warp] = d0;
                red[3 * warp + 1] = d1;
                red[3 * warp + 2] = d2;
            }
            __syncthreads();
            double ss = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                ss += red[3 * w];
                s1 += red[3 * w + 1];
                s2 += red[3 * w + 2];
            }
            inv_sigma = ss > 0.0 ? (float)(1.0 / sqrt(ss)) : 0.0f;
            const double cells = (double)W * (double)W;
            centre.sx = (float)((double)pk + s1 / cells);
            norm_w = sqrtf((float)(fmax(s2 - s1 * s1 / cells, 0.0) + 1e-5 * s2));
        } else {
            centre.ci_hi = mc_hi;
            centre.ci_lo = mc_lo;
            centre.ci = R;
            __syncthreads();
        }
        const float scale = (float)(1.0 / (4.0 * (double)N * (double)N));
        const float ebox = kSpecErr * norm_w;
        float bv = -INFINITY;
        int bi = INT_MAX;
        int flagged = 0;
        fft::correlate_tile<N1, N2, RASTER ? 2 : 0>(
            Z, RS, W, C, tw, neg, half, centre, tid, NT, BlockSync{},
            [&](int u, int v, float2 val) {
                if (v < C) {
                    const int idx = u * C + v;
                    const float inv_box = invs[idx];
                    const float gv = val.x * scale * inv_box * inv_sigma;
                    G[idx] = gv;
                    if (ebox * inv_box > kSpecTol)
                        flagged = 1;
                    else
                        better(bv, bi, gv, idx);
                }
            },
            [&]() {
                // the staged bytes are free from here on: the next pair's window comes in
                fence_async_smem();
                __syncthreads();
                if (bn < pairs) {
                    if (tid == 0) issue(bn);
                    inflight = true;
                }
            });

        float* surf = out.surfaces ? out.surfaces + (size_t)p * C * C : nullptr;
        float* gam = out.stage == 1 ? out.gam + b * C * C : nullptr;
        spec_surface<NT>(G, red, g, invs, inv_sigma, mean_c, ebox, chip, cs, win, ws, gam, surf, bv, bi,
                                   flagged);
        if (tid == 0) spec_result(out, p, R, W, C, bv, bi);
    }
    if (s_err) {
        // a wait ran out: count it once per CTA, give the pairs left a coarse result whose
        // refinement corners stay inside their windows, and let the copy in flight land before
        // the shared memory is given up
        if (tid == 0) {
            atomicAdd(errs, 1u);
            if constexpr (RASTER)
                for (long long q = b_left; q < pairs; q += gridDim.x) {
                    out.coarse[pair0 + q] = CoarseOut{-1, -1, 0, 0};
                    out.coarse_peak[pair0 + q] = NAN;
                }
            if (inflight) {
                const long long t0 = clock64();
                while (!mbar_try(bar, parity) && clock64() - t0 < kSpinCycles) {
                }
            }
        }
        __syncthreads();
    }
}

// transform lengths: N, N1, N2 (N1 N2 = N)
#define AMPCOR_SPEC_LENGTHS(X) \
    X(16, 4, 4)                \
    X(24, 4, 6)                \
    X(32, 4, 8)                \
    X(40, 5, 8)                \
    X(48, 6, 8)                \
    X(64, 8, 8)                \
    X(80, 8, 10)               \
    X(96, 8, 12)               \
    X(120, 8, 15)              \
    X(128, 8, 16)              \
    X(144, 12, 12)             \
    X(160, 10, 16)

// ------------------------------------------------------------------------------------------
// blocked spectral correlation: tiles beyond one CTA's shared memory
// ------------------------------------------------------------------------------------------
//
// The numerator surface is a sum over the chip's pixels, so it splits over square blocks of the
// chip: block k (rows [i0, i0 + B), columns [j0, j0 + B)) meets the sub-window of rows
// [i0, i0 + B + C - 1), columns [j0, j0 + B + C - 1), and its placements are those of the whole
// window.  spec_block_kernel runs the in-shared-memory FFT correlation of one block (one CTA per
// pair and block) and writes its partial numerators; spec_reduce_kernel sums a pair's partials in
// a fixed order, normalises them, bounds the transform error and takes the first maximum, as
// spec_kernel does for a tile that fits.  The chip is centred on the whole chip's mean
// (spec_chip_stats_kernel), each sub-window on its own mean s_k: the block then computes
// sum c (t - s_k), c the centred chip values the block placed in its tile, and the pair's numerator is
// the sum over blocks of that plus (s_k - s) sum_k c, for any s, since a whole centred chip sums to 0.
// s is the mean of the s_k: the c do not sum to 0 but to their roundings, and a steady return's level
// must not multiply those (128 px chips under a return of 300: off by up to 8.4e-6 with s = 0).

// one CTA of 256 threads per pair: the FP64 statistics of the R x R chip, from sums about its first
// sample (the differences and their squares are exact, so that a strong steady return costs their sums
// no digits)
__global__ void __launch_bounds__(256)
spec_chip_stats_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, int R,
                       TileStat* out)
{
    __shared__ double red[16];
    if (blockIdx.x >= pairs) return;
    const long long p = pair0 + blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (valid[p] < 0) {
        if (tid == 0) out[blockIdx.x] = TileStat{0.0, 0.0, 0.0};
        return;
    }
    const float* chip = spec_chip(src, pair0, blockIdx.x);
    const long long cs = src.chip_stride;
    const double pivot = __ldg(chip);
    double s1 = 0.0, s2 = 0.0;
    for (int y = warp; y < R; y += 8)
        for (int x = lane; x < R; x += 32) {
            const double v = (double)__ldg(chip + y * cs + x) - pivot;
            s1 += v;
            s2 += v * v;
        }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) {
        red[2 * warp] = s1;
        red[2 * warp + 1] = s2;
    }
    __syncthreads();
    if (tid == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; ++w) {
            a += red[2 * w];
            b += red[2 * w + 1];
        }
        out[blockIdx.x] = chip_stat(pivot, a, b, (double)R * (double)R, 0.0);
    }
}

// 1/sigma of every placement box of a window read straight from global memory (windows larger
// than a CTA stages): FP64 column sums sliding down the window, FP64 prefix sums along the rows,
// SR placement rows at a time (window_stats_xs); inv: C^2 floats per chunk-local pair.  W <= kThreads.
__global__ void __launch_bounds__(kThreads, 2)
spec_tile_stats_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, int R, int W,
                       int SR, float* inv)
{
    extern __shared__ __align__(16) double tsm[];
    if (blockIdx.x >= pairs) return;
    const long long p = pair0 + blockIdx.x;
    if (valid[p] < 0) return;
    const int C = W - R + 1;
    window_stats_xs<1>(spec_win(src, pair0, blockIdx.x), (int)src.win_stride, W, R, C, SR,
                       inv + (long long)blockIdx.x * C * C, tsm);
}

// The partial numerators of one chip block of one pair (CTA b K + k): g is the tile of a block
// (g.R = B, g.W = B + C - 1, g.C = C), nb blocks per axis.  part: C^2 floats per (pair, block),
// already scaled; scal: kBlockScalars doubles per (pair, block), s_k, sum_k c and |c| |t - s_k|.
template <int N1, int N2>
__global__ void __launch_bounds__(kSpecThreads, 1)
spec_block_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, SpecGeom g,
                  int nb, const TileStat* cstat, const float2* tw_g, float* part, double* scal)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    const int K = nb * nb;
    const int b = blockIdx.x / K, k = blockIdx.x - b * K;
    if (b >= pairs) return;
    const long long p = pair0 + b;
    if (valid[p] < 0) return;
    constexpr int N = N1 * N2;
    constexpr int RS = N + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int B = g.R, S = g.W, C = g.C;
    const int i0 = (k / nb) * B, j0 = (k - (k / nb) * nb) * B;
    float2* Z = reinterpret_cast<float2*>(ssm + g.off_z);
    float2* tw = reinterpret_cast<float2*>(ssm + g.off_tw);
    int* neg = reinterpret_cast<int*>(ssm + g.off_neg);
    int* half = reinterpret_cast<int*>(ssm + g.off_half);
    double* red = reinterpret_cast<double*>(ssm + g.off_red);
    float* Zf = reinterpret_cast<float*>(Z);
    const long long cs = src.chip_stride, ws = src.win_stride;
    const float* chip = spec_chip(src, pair0, b) + i0 * cs + j0;
    const float* win = spec_win(src, pair0, b) + i0 * ws + j0;
    const TileStat cst = cstat[b];
    const float mc_hi = (float)cst.mean, mc_lo = (float)(cst.mean - (double)mc_hi);

    // the block of the chip, centred on the whole chip's mean, to registers; the sub-window to the
    // tile's real parts by asynchronous copies, zeros around it
    constexpr int JN = (N + kSpecWarps - 1) / kSpecWarps, IN = (N + 31) / 32;
    float cr[JN][IN];
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const int y = warp + kSpecWarps * j, x = lane + 32 * i;
            cr[j][i] = y < B && x < B ? (__ldg(chip + y * cs + x) - mc_hi) - mc_lo : 0.0f;
        }
    for (int y = warp; y < N; y += kSpecWarps) {
        float* zr = Zf + 2 * y * RS;
        for (int x = lane; x < N; x += 32) {
            if (y < S && x < S)
                cp_async4(zr + 2 * x, win + y * ws + x);
            else
                zr[2 * x] = 0.0f;
        }
    }
    for (int q = tid; q < N; q += kSpecThreads) {
        tw[q] = __ldg(tw_g + q);
        neg[q] = fft::neg_pos<N1, N2>(q);
    }
    if (warp == 0) build_half<N1, N2>(half);
    cp_async_wait_all();
    __syncthreads();

    // FP64 sums of the centred chip block (its sum and sum of squares) and of the sub-window about
    // a pivot k (its first sample): the sums of t - k and (t - k)^2 give its mean and an upper bound
    // of |t'|^2 (which only scales the error bound), as in spec_kernel
    double a0 = 0.0, a1 = 0.0, a2, a3;
    const float pk = Z[0].x;
    {
        float sw = 0.0f, sw2 = 0.0f;
        for (int y = warp; y < S; y += kSpecWarps) {
            const float2* zr = Z + y * RS;
            for (int x = lane; x < S; x += 32) {
                const float t = zr[x].x - pk;
                sw += t;
                sw2 = fmaf(t, t, sw2);
            }
        }
#pragma unroll
        for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int i = 0; i < IN; ++i) {
                const double c = cr[j][i];
                a0 += c;
                a1 += c * c;
            }
        a2 = sw;
        a3 = sw2;
        block_sum2<kSpecWarps>(a0, a1, red);
        block_sum2<kSpecWarps>(a2, a3, red);
    }
    const double cells_w = (double)S * (double)S;
    const double mean_w = (double)pk + a2 / cells_w;
    const double st = fmax(a3 - a2 * a2 / cells_w, 0.0) + 1e-5 * a3;
    const fft::Centre centre{(float)mean_w, S};
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const int y = warp + kSpecWarps * j, x = lane + 32 * i;
            if (y < N && x < N) Zf[2 * (y * RS + x) + 1] = cr[j][i];
        }
    __syncthreads();
    // the last inverse step hands placement row u to the store, which puts it in tile row u (no
    // later step reads those rows), so the numerators need no buffer beside the tile
    fft::correlate_tile<N1, N2>(Z, RS, S, C, tw, neg, half, centre, tid, kSpecThreads, BlockSync{},
                                [&](int u, int v, float2 val) { Z[u * RS + v] = val; });
    const float scale = (float)(1.0 / (4.0 * (double)N * (double)N));
    float* out = part + ((long long)b * K + k) * C * C;
    for (int idx = tid; idx < C * C; idx += kSpecThreads) {
        const int u = idx / C, v = idx - u * C;
        out[idx] = Z[u * RS + v].x * scale;
    }
    if (tid == 0) {
        double* to = scal + kBlockScalars * ((long long)b * K + k);
        to[0] = (double)centre.sx;
        to[1] = a0;
        to[2] = sqrt(a1 * st);
    }
}

// The blocks of a stage whose tiles the copy engine can bring (a raster's windows, or refined
// windows), staged as spec_staged_kernel stages whole windows: one resident CTA per SM walks the
// blocks, and the next block's sub-window arrives in the tile's last bytes while this one's inverse
// transform finishes.  ACC (tiles of up to 128 samples, whose summed spectrum fits beside them): a
// CTA takes all blocks of a pair in turn, adds up their spectra and transforms back once, part
// holding C^2 floats per pair; else one block at a time, C^2 floats per (pair, block).  The sums and
// the centring are spec_block_kernel's.  Bounded waits as in spec_staged_kernel; the partial
// numerators of pairs left out after one ran out are undefined, their maxima still placements.
// Measured on B200, 3,844 pairs of 128 px chips: the coarse stage (four 128-sample tiles a pair) 2,136
// us unstaged, 1,910 staged block by block, 1,534 with the spectra summed (60 more with every sample of a
// chip block summed in FP64); the fine stage (four 160-sample tiles, whose 104 KB spectrum fits nowhere
// beside them) 3,025 -> 2,603 us.
template <int N1, int N2, bool ACC>
__global__ void __launch_bounds__(kSpecThreads, 1)
spec_block_staged_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, SpecGeom g,
                         int nb, const TileStat* cstat, const float2* tw_g, float* part, double* scal,
                         unsigned int* errs, const __grid_constant__ CUtensorMap wmap,
                         const __grid_constant__ CUtensorMap cmap, int raster, int stall)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    constexpr int NT = kSpecThreads, NW = NT / 32, N = N1 * N2, RS = N + 1;
    constexpr int JN = (N + NW - 1) / NW, IN = (N + 31) / 32;
    constexpr int PJ = 5;  // row groups of a piece read whole before it is written
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int B = g.R, S = g.W, C = g.C, SW = g.stage_rs, K = nb * nb;
    float2* Z = reinterpret_cast<float2*>(ssm + g.off_z);
    float2* tw = reinterpret_cast<float2*>(ssm + g.off_tw);
    int* neg = reinterpret_cast<int*>(ssm + g.off_neg);
    int* half = reinterpret_cast<int*>(ssm + g.off_half);
    double* red = reinterpret_cast<double*>(ssm + g.off_red);
    float2* acc = reinterpret_cast<float2*>(ssm + g.off_gam);
    float* stage = reinterpret_cast<float*>(ssm + g.off_stage);
    uint64_t* bar = reinterpret_cast<uint64_t*>(ssm + g.off_bar);
    int& s_err = *reinterpret_cast<int*>(ssm + g.off_bar + 8);
    const long long cs = src.chip_stride, ws = src.win_stride;
    const int jA = g.stage_y0 / NW;

    for (int k = tid; k < N; k += NT) {
        tw[k] = __ldg(tw_g + k);
        neg[k] = fft::neg_pos<N1, N2>(k);
    }
    if (warp == 0) build_half<N1, N2>(half);
    if (tid == 0) {
        s_err = 0;
        mbar_init(bar, 1);
        mbar_init(bar + 2, 1);  // completed by nothing: the wait of a failure-detection test
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // a failure-detection test, as in spec_staged_kernel: the CTA skips its blocks
    if (stall) {
        mbar_wait(bar + 2, 0u, &s_err, kStallCycles);
        __syncthreads();
    }
    const bool run = !stall || !s_err;
    // item n of this CTA: chunk pair b and its block k; false past the end
    auto item = [&](long long n, long long& b, int& k) {
        const long long t = ACC ? (blockIdx.x + n / K * gridDim.x) * K + n % K : blockIdx.x + n * gridDim.x;
        b = t / K;
        k = (int)(t - b * K);
        return b < pairs;
    };
    // first sample of a block's sub-window and chip block within the pair's window and chip
    auto corner = [&](int k, int& i0, int& j0) {
        i0 = k / nb * B;
        j0 = (k - k / nb * nb) * B;
    };
    // thread 0: where the next item's tiles lie, found out early, and their copy (as in
    // spec_staged_kernel)
    bool next_ok = false;
    int nx = 0, ny = 0, nz = 0, ncx = 0, ncy = 0;
    auto look = [&](long long n) {
        long long b;
        int k, i0, j0;
        item(n, b, k);
        corner(k, i0, j0);
        next_ok = valid[pair0 + b] >= 0;
        if (!next_ok) return;
        nx = ncx = j0;
        ny = ncy = i0;
        nz = (int)b;
        if (raster) {
            const long long wo = src.win_off[pair0 + b], co = src.chip_off[pair0 + b];
            const int wy = (int)(wo / ws), cy = (int)(co / cs);
            ny += wy;
            nx += (int)(wo - (long long)wy * ws);
            ncy += cy;
            ncx += (int)(co - (long long)cy * cs);
        }
    };
    auto issue = [&]() {
        if (!next_ok) {
            mbar_arrive(bar);
            return;
        }
        mbar_expect_tx(bar, (unsigned)S * (unsigned)SW * 4u);
        if (raster) {
            tensor_to_smem(stage, &wmap, nx & ~3, ny, bar);
            tensor_prefetch_l2(&cmap, ncx & ~3, ncy);
        } else {
            tensor3_to_smem(stage, &wmap, nx & ~3, ny, nz, bar);
            tensor3_prefetch_l2(&cmap, ncx & ~3, ncy, nz);
        }
    };
    long long b;
    int k;
    bool inflight = run && item(0, b, k);
    if (tid == 0 && inflight) {
        look(0);
        issue();
    }
    uint32_t parity = 0;
    for (long long n = 0; run && item(n, b, k); ++n) {
        const long long p = pair0 + b;
        const bool ok = valid[p] >= 0;
        long long bn;
        int kn, i0, j0;
        const bool more = item(n + 1, bn, kn);
        corner(k, i0, j0);
        const TileStat cst = cstat[b];
        const float mc_hi = (float)cst.mean, mc_lo = (float)(cst.mean - (double)mc_hi);
        const bool landed = mbar_wait(bar, parity, &s_err);
        if (__syncthreads_or(!landed)) break;
        parity ^= 1u;
        inflight = false;
        if (tid == 0 && more) look(n + 1);
        auto next = [&]() {
            // the staged bytes are free: the next block's sub-window comes in
            fence_async_smem();
            __syncthreads();
            if (more) {
                if (tid == 0) issue();
                inflight = true;
            }
        };
        const bool late = ACC && g.late && k == K - 1;
        auto early = [&]() {
            if (!late) next();
        };
        if (!ok) {
            next();
            continue;
        }
        const float* chip = spec_chip(src, pair0, b) + i0 * cs + j0;
        float cr[JN][IN];
#pragma unroll
        for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int i = 0; i < IN; ++i) {
                const int y = warp + NW * j, x = lane + 32 * i;
                cr[j][i] = y < B && x < B ? (__ldg(chip + y * cs + x) - mc_hi) - mc_lo : 0.0f;
            }
        // sub-window sample (y, x) in the staging bytes: the box starts xo samples before it
        const int xo = raster ? (int)((src.win_off[p] + j0) % ws & 3) : j0 & 3;
        const float pk = stage[xo];
        float sw = 0.0f, sw2 = 0.0f;
        auto put = [&](int j, int i, float t) {
            const int y = warp + NW * j, x = lane + 32 * i;
            if (y < N && x < N) {
                if (y < S && x < S) {
                    const float d = t - pk;
                    sw += d;
                    sw2 = fmaf(d, d, sw2);
                }
                Z[y * RS + x] = make_float2(t, cr[j][i]);
            }
        };
        auto staged = [&](int j, int i) {
            const int y = warp + NW * j, x = lane + 32 * i;
            return y < S && x < S ? stage[y * SW + xo + x] : 0.0f;
        };
        // the tile, as spec_staged_kernel writes it
#pragma unroll
        for (int j = 0; j < JN; ++j)
            if (j < jA)
#pragma unroll
                for (int i = 0; i < IN; ++i) put(j, i, staged(j, i));
        __syncthreads();
#pragma unroll
        for (int q0 = 0; q0 < JN; q0 += PJ) {
            if (q0 + PJ <= jA) continue;
            float v[PJ][IN];
#pragma unroll
            for (int q = 0; q < PJ; ++q)
#pragma unroll
                for (int i = 0; i < IN; ++i) v[q][i] = q0 + q < JN && q0 + q >= jA ? staged(q0 + q, i) : 0.0f;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < PJ; ++q)
                if (q0 + q < JN && q0 + q >= jA)
#pragma unroll
                    for (int i = 0; i < IN; ++i) put(q0 + q, i, v[q][i]);
        }
        // FP64 sums over the block: sum c, sum c^2 of the centred chip block (every sample in FP64:
        // the level of a strong steady return multiplies the first), sum t - k, sum (t - k)^2 of the
        // sub-window (FP32 per thread)
        double a[4] = {0.0, 0.0, (double)sw, (double)sw2};
#pragma unroll
        for (int j = 0; j < JN; ++j)
            if (warp + NW * j < B)
#pragma unroll
                for (int i = 0; i < IN; ++i)
                    if (32 * i < B) {
                        const double c = cr[j][i];
                        a[0] += c;
                        a[1] = fma(c, c, a[1]);
                    }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            a[q] = warp_sum(a[q]);
            if (lane == 0) red[4 * warp + q] = a[q];
        }
        __syncthreads();
        double a2 = 0.0, a3 = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) a2 += red[4 * w + 2];
        const double cells = (double)S * (double)S;
        const fft::Centre centre{(float)((double)pk + a2 / cells), S};
        if (tid == 0) {
            double a0 = 0.0, a1 = 0.0;
            for (int w = 0; w < NW; ++w) {
                a0 += red[4 * w];
                a1 += red[4 * w + 1];
                a3 += red[4 * w + 3];
            }
            const double st = fmax(a3 - a2 * a2 / cells, 0.0) + 1e-5 * a3;
            double* to = scal + kBlockScalars * (b * K + k);
            to[0] = (double)centre.sx;
            to[1] = a0;
            to[2] = sqrt(a1 * st);
        }
        const float scale = (float)(1.0 / (4.0 * (double)N * (double)N));
        float* out = part + (ACC ? b : b * K + k) * C * C;
        auto store = [&](int u, int v, float2 val) {
            if (v < C) out[u * C + v] = val.x * scale;
        };
        if constexpr (ACC)
            fft::correlate_sum<N1, N2, 2>(Z, RS, S, C, tw, neg, half, centre, acc, k == 0, k == K - 1, tid, NT,
                                          BlockSync{}, store, early);
        else
            fft::correlate_tile<N1, N2, 0>(Z, RS, S, C, tw, neg, half, centre, tid, NT, BlockSync{}, store, early);
        if (late) next();
    }
    if (s_err) {
        if (tid == 0) {
            atomicAdd(errs, 1u);
            if (inflight) {
                const long long t0 = clock64();
                while (!mbar_try(bar, parity) && clock64() - t0 < kSpinCycles) {
                }
            }
        }
        __syncthreads();
    }
}

// One CTA per pair: the sum of the K partial numerators of every placement (FP64, in block order,
// plus the centring corrections), normalised by the chip's 1/|r'| and the placement's 1/sigma_box,
// then the direct FP32 recomputation where the transform's bound is loose (spec_surface) and the
// stage's outputs, as in spec_kernel.  kp: partial surfaces per pair, K, or 1 where the spectra of
// the blocks were summed.  g: the whole stage (R, W, C).  Shared memory: the
// placement statistics and the surface (C^2 floats each) and a reduction scratch.
__global__ void __launch_bounds__(kThreads, 1)
spec_reduce_kernel(SpecSource src, long long pair0, long long pairs, const long long* valid, SpecGeom g,
                   int K, int kp, const TileStat* cstat, InvSource inv, const float* part, const double* scal,
                   SpecOut out)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    if (blockIdx.x >= pairs) return;
    const long long p = pair0 + blockIdx.x;
    const int tid = threadIdx.x;
    if (valid[p] < 0) {
        if (out.stage == 0 && tid == 0) {
            out.coarse[p] = CoarseOut{-1, -1, -1, -1};
            out.coarse_peak[p] = NAN;
        }
        return;
    }
    const int R = g.R, W = g.W, C = g.C, CC = C * C;
    float* invs = reinterpret_cast<float*>(ssm);
    float* G = invs + ((CC + 3) & ~3);
    double* red = reinterpret_cast<double*>(G + ((CC + 3) & ~3));
    const float* inv_b = inv.off ? inv.base + inv.off[p] : inv.base + (long long)blockIdx.x * CC;
    const long long is = inv.off ? inv.stride : C;
    {
        const int warp = tid >> 5, lane = tid & 31;
        for (int u = warp; u < C; u += kWarps)
#pragma unroll 4
            for (int v = lane; v < C; v += 32) cp_async4(invs + u * C + v, inv_b + u * is + v);
    }
    const double* sc = scal + kBlockScalars * (long long)blockIdx.x * K;
    double level = 0.0, corr = 0.0, errs = 0.0;
    for (int k = 0; k < K; ++k) level += sc[kBlockScalars * k];
    level /= (double)K;
    for (int k = 0; k < K; ++k) {
        corr += (sc[kBlockScalars * k] - level) * sc[kBlockScalars * k + 1];
        errs += sc[kBlockScalars * k + 2];
    }
    const TileStat cst = cstat[blockIdx.x];
    const float inv_sigma = (float)cst.inv_norm;
    const float ebox = kSpecErr * (float)errs * inv_sigma;
    cp_async_wait_all();
    __syncthreads();
    float bv = -INFINITY;
    int bi = INT_MAX;
    int flagged = 0;
    const float* pp = part + (long long)blockIdx.x * kp * CC;
    // a batch of placements and blocks in flight per thread (one load after the other, 33 placements of
    // four blocks a thread, kept a +-64 px search waiting: 246 -> 182 us for 900 pairs)
    constexpr int kPlace = 4, kBlocks = 4;
    for (int idx0 = tid; idx0 < CC; idx0 += kPlace * kThreads) {
        double num[kPlace];
#pragma unroll
        for (int q = 0; q < kPlace; ++q) num[q] = corr;
        for (int k0 = 0; k0 < kp; k0 += kBlocks) {
            float v[kPlace][kBlocks];
#pragma unroll
            for (int q = 0; q < kPlace; ++q)
#pragma unroll
                for (int k = 0; k < kBlocks; ++k)
                    v[q][k] = idx0 + q * kThreads < CC && k0 + k < kp
                                  ? __ldg(pp + (long long)(k0 + k) * CC + idx0 + q * kThreads)
                                  : 0.0f;
#pragma unroll
            for (int q = 0; q < kPlace; ++q)
#pragma unroll
                for (int k = 0; k < kBlocks; ++k)
                    if (k0 + k < kp) num[q] += (double)v[q][k];
        }
#pragma unroll
        for (int q = 0; q < kPlace; ++q) {
            const int idx = idx0 + q * kThreads;
            if (idx >= CC) break;
            const float inv_box = invs[idx];
            // (one rounding instead of three)
            const float gv = (float)(num[q] * ((double)inv_box * cst.inv_norm));
            G[idx] = gv;
            if (ebox * inv_box > kSpecTol)
                flagged = 1;
            else
                better(bv, bi, gv, idx);
        }
    }
    __syncthreads();
    const float* chip = spec_chip(src, pair0, blockIdx.x);
    const float* win = spec_win(src, pair0, blockIdx.x);
    float* surf = out.surfaces ? out.surfaces + (size_t)p * CC : nullptr;
    float* gam = out.stage == 1 ? out.gam + (long long)blockIdx.x * CC : nullptr;
    spec_surface<kThreads>(G, red, g, invs, inv_sigma, cst.mean, ebox, chip, src.chip_stride, win,
                           src.win_stride, gam, surf, bv, bi, flagged);
    if (tid == 0) spec_result(out, p, R, W, C, bv, bi);
}

}  // namespace

bool spec_radices(int n, int& n1, int& n2)
{
#define AMPCOR_SPEC_CASE(NN, A, B) \
    if (n == NN) {                 \
        n1 = A;                    \
        n2 = B;                    \
        return true;               \
    }
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return false;
}

int spec_next_length(int w)
{
#define AMPCOR_SPEC_CASE(NN, A, B) \
    if (w <= NN) return NN;
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return 0;
}

// CTAs of NT threads that the staged kernel runs side by side on an SM, for the tile lengths of
// which two or more fit: N, N1, N2, NT, CTAS
#define AMPCOR_SPEC_SHARED(X) \
    X(16, 4, 4, 128, 6)       \
    X(24, 4, 6, 128, 6)       \
    X(32, 4, 8, 128, 6)       \
    X(40, 5, 8, 128, 6)       \
    X(48, 6, 8, 192, 4)       \
    X(64, 8, 8, 256, 3)       \
    X(80, 8, 10, 256, 2)      \
    X(96, 8, 12, 192, 2)

bool spec_shared(int n, int& threads, int& ctas)
{
#define AMPCOR_SPEC_CASE(NN, A, B, NT, CTAS) \
    if (n == NN) {                           \
        threads = NT;                        \
        ctas = CTAS;                         \
        return true;                         \
    }
    AMPCOR_SPEC_SHARED(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return false;
}

cudaError_t spec_set_smem_limits()
{
    const int limit = 227 * 1024;
    cudaError_t e = cudaSuccess;
#define AMPCOR_SPEC_CASE(NN, A, B) \
    if (e == cudaSuccess)          \
        e = cudaFuncSetAttribute(spec_kernel<A, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if (e == cudaSuccess)          \
        e = cudaFuncSetAttribute(spec_staged_kernel<A, B, true, kSpecThreads, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if (e == cudaSuccess)          \
        e = cudaFuncSetAttribute(spec_staged_kernel<A, B, false, kSpecThreads, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if (e == cudaSuccess)          \
        e = cudaFuncSetAttribute(spec_block_kernel<A, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if constexpr (NN >= kSumLeast && NN <= kSumMost) \
        if (e == cudaSuccess)      \
            e = cudaFuncSetAttribute(spec_block_staged_kernel<A, B, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if constexpr (NN >= 128)       \
        if (e == cudaSuccess)      \
            e = cudaFuncSetAttribute(spec_block_staged_kernel<A, B, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
#define AMPCOR_SPEC_CASE(NN, A, B, NT, CTAS) \
    if (e == cudaSuccess)                    \
        e = cudaFuncSetAttribute(spec_staged_kernel<A, B, true, NT, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit); \
    if (e == cudaSuccess)                    \
        e = cudaFuncSetAttribute(spec_staged_kernel<A, B, false, NT, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    AMPCOR_SPEC_SHARED(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(spec_reduce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(spec_tile_stats_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    return e;
}

cudaError_t launch_spec_chip_stats(unsigned blocks, cudaStream_t st, SpecSource src, long long pair0,
                                   long long pairs, const long long* valid, int R, TileStat* out)
{
    spec_chip_stats_kernel<<<blocks, 256, 0, st>>>(src, pair0, pairs, valid, R, out);
    return cudaGetLastError();
}

// placement rows per pass of the tile statistics (two CTAs per SM where the window allows) and
// the shared memory that takes; 0 when the window is wider than a CTA has threads
int spec_tile_stats_rows(int W, int C, int& smem)
{
    smem = 0;
    if (W > kThreads || C < 1) return 0;
    // window_stats_xs hands each placement row of a pass to one warp
    int sr = C < kWarps ? C : kWarps;
    while (sr > 1 && 2L * sr * (W + 1) * 8 > 110L * 1024) --sr;
    smem = (int)(2L * sr * (W + 1) * 8);
    return smem <= 227 * 1024 ? sr : 0;
}

cudaError_t launch_spec_tile_stats(unsigned blocks, cudaStream_t st, SpecSource src, long long pair0,
                                   long long pairs, const long long* valid, int R, int W, float* inv)
{
    int smem = 0;
    const int sr = spec_tile_stats_rows(W, W - R + 1, smem);
    if (!sr) return cudaErrorInvalidValue;
    spec_tile_stats_kernel<<<blocks, kThreads, smem, st>>>(src, pair0, pairs, valid, R, W, sr, inv);
    return cudaGetLastError();
}

cudaError_t launch_spec_block(const SpecGeom& tile, int nb, unsigned blocks, cudaStream_t st,
                              SpecSource src, long long pair0, long long pairs,
                              const long long* valid, const TileStat* cstat, const float2* tw,
                              float* part, double* scal)
{
#define AMPCOR_SPEC_CASE(NN, A, B)                                                                   \
    if (tile.N == NN) {                                                                              \
        spec_block_kernel<A, B><<<blocks, kSpecThreads, tile.smem_bytes, st>>>(src, pair0, pairs, valid, \
                                                                           tile, nb, cstat, tw, part, scal); \
        return cudaGetLastError();                                                                   \
    }
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_spec_block_staged(const SpecGeom& tile, int nb, unsigned sms, cudaStream_t st, SpecSource src,
                                     long long pair0, long long pairs, const long long* valid,
                                     const TileStat* cstat, const float2* tw, float* part, double* scal,
                                     unsigned int* errs, const CUtensorMap* wmap, const CUtensorMap* cmap, int raster, int stall)
{
    if (pairs <= 0) return cudaSuccess;
    const long long units = tile.acc ? pairs : pairs * nb * nb;
    const unsigned blocks = (unsigned)std::min<long long>(units, std::max(1u, sms));
    auto run = [&](auto kernel) {
        kernel<<<blocks, kSpecThreads, tile.smem_staged, st>>>(src, pair0, pairs, valid, tile, nb, cstat, tw, part,
                                                               scal, errs, *wmap, *cmap, raster, stall);
        return cudaGetLastError();
    };
#define AMPCOR_SPEC_CASE(NN, A, B)                                                          \
    if (tile.N == NN) {                                                                     \
        if constexpr (NN >= kSumLeast && NN <= kSumMost)                                    \
            if (tile.acc) return run(spec_block_staged_kernel<A, B, true>);                 \
        if constexpr (NN >= 128)                                                            \
            if (!tile.acc) return run(spec_block_staged_kernel<A, B, false>);               \
    }
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return cudaErrorInvalidValue;
}

int spec_reduce_smem(int C)
{
    return 2 * ((C * C + 3) & ~3) * 4 + 256;
}

cudaError_t launch_spec_reduce(const SpecGeom& full, int K, int kp, unsigned blocks, cudaStream_t st,
                               SpecSource src, long long pair0, long long pairs,
                               const long long* valid, const TileStat* cstat, InvSource inv,
                               const float* part, const double* scal, SpecOut out)
{
    spec_reduce_kernel<<<blocks, kThreads, spec_reduce_smem(full.C), st>>>(src, pair0, pairs, valid, full, K,
                                                                           kp, cstat, inv, part, scal, out);
    return cudaGetLastError();
}


cudaError_t launch_spec(const SpecGeom& g, unsigned blocks, cudaStream_t st, SpecSource src,
                        long long pair0, long long pairs, const long long* valid, InvSource inv,
                        const float2* tw, SpecOut out)
{
#define AMPCOR_SPEC_CASE(NN, A, B)                                                               \
    if (g.N == NN) {                                                                             \
        spec_kernel<A, B><<<blocks, kSpecThreads, g.smem_bytes, st>>>(src, pair0, pairs, valid, g,  \
                                                                  inv, tw, out);                 \
        return cudaGetLastError();                                                               \
    }
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_spec_staged(const SpecGeom& g, unsigned sms, cudaStream_t st, SpecSource src,
                               long long pair0, long long pairs, const long long* valid, InvSource inv,
                               const float2* tw, SpecOut out, const TileStat* cstat, const TileStat* wstat,
                               unsigned int* errs, const CUtensorMap* wmap, const CUtensorMap* cmap,
                               const CUtensorMap* imap, int stall)
{
    if (pairs <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)std::min<long long>(pairs, std::max(1u, sms) * (long long)g.ctas);
    auto run = [&](auto raster, auto dense) {
        if (wmap)
            raster<<<blocks, g.threads, g.smem_staged, st>>>(src, pair0, pairs, valid, g, inv, tw, out, cstat, wstat, errs,
                                                             *wmap, *cmap, *imap, stall);
        else
            dense<<<blocks, g.threads, g.smem_staged, st>>>(src, pair0, pairs, valid, g, inv, tw, out, cstat, wstat, errs,
                                                            CUtensorMap{}, CUtensorMap{}, CUtensorMap{}, stall);
        return cudaGetLastError();
    };
#define AMPCOR_SPEC_CASE(NN, A, B, NT, CTAS) \
    if (g.N == NN && g.threads == NT)        \
        return run(spec_staged_kernel<A, B, true, NT, CTAS>, spec_staged_kernel<A, B, false, NT, CTAS>);
    AMPCOR_SPEC_SHARED(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
#define AMPCOR_SPEC_CASE(NN, A, B) \
    if (g.N == NN)                 \
        return run(spec_staged_kernel<A, B, true, kSpecThreads, 1>, spec_staged_kernel<A, B, false, kSpecThreads, 1>);
    AMPCOR_SPEC_LENGTHS(AMPCOR_SPEC_CASE)
#undef AMPCOR_SPEC_CASE
    return cudaErrorInvalidValue;
}

}  // namespace ampcor_b200

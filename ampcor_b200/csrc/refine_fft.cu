// sm_100a kernel of the spectral form's refinement: band-limited upsampling of a complex tile by 2,
// amplitudes out (the reference's zero-padded FFT, refine.cu / cuFFT).
//
// Zero-padding an N-point spectrum to 2 N points (the Nyquist bin split in two halves) keeps every
// sample and puts between neighbours the value of the band-limited interpolant half a sample on:
//   x(n + 1/2) = S x = IDFT(P DFT(x)), P(k) = exp(i pi k / N) for |k| < N / 2, 0 for k = N / 2.
// So no 2 N-point transform is needed: of the four phases of the 2 N x 2 N result one is the tile
// itself, and the others are S along the rows, S down the columns, and both.  S takes three
// in-place passes over a line (fft.cuh): the transform's step A; its step B, P and the inverse's
// step B in registers (`shift_middle`); the inverse's step A.  An upsampled tile costs 3 N lines of
// S (N rows, N columns, N rows again), 6 N transforms of N points, against 2 N of N points and 3 N of
// 2 N points in the padded form, and needs the N x N tile and a strip of rows in shared memory instead
// of a 2 N x N one, so that two to eight CTAs share an SM for tiles up to 96 samples and the larger ones
// need no buffer in global memory.
//
// What bounds it: instruction issue (ncu: 68 % of the slots busy), with shared-memory wavefronts next;
// 15 % of the time goes into the IEEE square roots of the outputs, 15 % into the middle pass.  Measured
// on B200, a chip of 64 and a window of 80 samples for each of 14,641 pairs: 2,426 us padded, 1,594 us by
// shifts, 1,458 us with packed sums and strips of 32 rows, 1,538 us with the tiles' statistics on the way
// out (a chip's amplitudes summed in FP64; they save the fine stage more); 3,844 pairs of 128 and 144
// samples 3,235 -> 1,904 us.
#include <algorithm>
#include <type_traits>

#include "fft.cuh"
#include "kernels.cuh"
#include "tile_common.cuh"

namespace ampcor_b200 {

namespace {

// the middle of S along a line: the group of k1 (positions N2 k1 ..) through the transform's step
// B, the half-sample phases (1 / N included) and the inverse's step B
template <int N1, int N2>
__device__ __forceinline__ void shift_middle(float2* base, int es, int k1, const float2* ph)
{
    float2 a[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) a[j] = base[(N2 * k1 + j) * es];
    fft::Dft<N2, -1>::run(a);
#pragma unroll
    for (int j = 0; j < N2; ++j) a[j] = fft::cmul(a[j], ph[N2 * k1 + j]);
    fft::Dft<N2, 1>::run(a);
#pragma unroll
    for (int j = 0; j < N2; ++j) base[(N2 * k1 + j) * es] = a[j];
}

__device__ __forceinline__ float amplitude(float2 z) { return sqrtf(z.x * z.x + z.y * z.y); }

// N = N1 N2 samples a side; NT threads; SR rows of the tile to a strip; CTAS per SM
template <int N1, int N2, int NT, int SR, int CTAS>
struct HalfGeom {
    static constexpr int N = N1 * N2, RS = N + 1;
    static constexpr int smem = (N * RS + SR * RS + 2 * N) * 8 + 4 * (NT / 32) * 8;
    static_assert(CTAS * (smem + 1024) <= 228 * 1024, "the CTAs of an SM share its memory");
};

// one tile of every pair of a chunk: the chip (coarse == nullptr) or the nudged window.  tab: the
// N twiddles exp(-2 pi i m / N), then P in the order of the transform's positions.
template <int N1, int N2, int NT, int SR, int CTAS, bool DERAMP, bool CHIP>
__global__ void __launch_bounds__(NT, CTAS)
refine_half_kernel(const float2* base, const long long* off, long long stride, const CoarseOut* coarse,
                   long long pair0, long long pairs, const long long* valid, const float2* tab, float* refined,
                   long long refined_stride, long long out_off, double flat, TileStat* stat)
{
    using G = HalfGeom<N1, N2, NT, SR, CTAS>;
    constexpr int N = G::N, F = 2 * N, RS = G::RS;
    extern __shared__ __align__(16) unsigned char rsm[];
    if (blockIdx.x >= pairs) return;
    const long long p = pair0 + blockIdx.x;
    if (valid[p] < 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float2* X = reinterpret_cast<float2*>(rsm);
    float2* Y = X + N * RS;
    float2* tw = Y + SR * RS;
    float2* ph = tw + N;
    double* red = reinterpret_cast<double*>(ph + N);
    const float2* src = base + off[p];
    if constexpr (!CHIP) {
        const CoarseOut co = coarse[p];
        src += co.top * stride + co.left;
    }
    float2* out = reinterpret_cast<float2*>(refined + (long long)blockIdx.x * refined_stride + out_off);

    // the tile into place, its sum taken on the way (FP32 per thread, FP64 across the block)
    constexpr int KT = (N * N + NT - 1) / NT, CH = KT <= 28 ? KT : (KT + 1) / 2;
    float sx = 0.0f, sy = 0.0f;
#pragma unroll 1
    for (int q0 = 0; q0 < KT; q0 += CH) {
        float2 v[CH];
#pragma unroll
        for (int q = 0; q < CH; ++q) {
            const int k = tid + (q0 + q) * NT;
            v[q] = q0 + q < KT && k < N * N ? __ldg(src + (k / N) * stride + k % N) : make_float2(0.0f, 0.0f);
        }
        if (q0 == 0)
            for (int k = tid; k < 2 * N; k += NT) tw[k] = __ldg(tab + k);
#pragma unroll
        for (int q = 0; q < CH; ++q) {
            const int k = tid + (q0 + q) * NT;
            if (q0 + q < KT && k < N * N) {
                X[(k / N) * RS + k % N] = v[q];
                sx += v[q].x;
                sy += v[q].y;
            }
        }
    }
    // The mean comes off as the transforms read the tile and back on with the amplitudes: S keeps a
    // constant as it is, and the transforms round on the tile's variation, not on its level.
    float2 mu;
    if constexpr (DERAMP) {
        __syncthreads();
        deramp_tile<NT>(X, RS, N, red);
        mu = tile_mean<false, false, NT>(X, RS, N, 0.0f, 0.0f, red);
    } else {
        const double a = warp_sum((double)sx), b = warp_sum((double)sy);
        if (lane == 0) {
            red[2 * warp] = a;
            red[2 * warp + 1] = b;
        }
        __syncthreads();
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < NT / 32; ++w) {
            ta += red[2 * w];
            tb += red[2 * w + 1];
        }
        mu = make_float2((float)(ta / ((double)N * N)), (float)(tb / ((double)N * N)));
    }

    // The sums and sums of squares of the upsampled amplitudes.  A chip's make its correlations'
    // mean and norm: FP64 for every amplitude.  A window's mean only conditions the transform and its
    // norm only scales the error bound: FP32 per thread about one of the tile's own amplitudes (so that
    // a strong steady return costs no digits of their variance), FP64 from there on.
    using Sum = std::conditional_t<CHIP, double, float>;
    const Sum pivot = CHIP ? 0.0f : amplitude(X[(tid % N) * RS + (7 * tid) % N]);
    Sum r1 = 0, r2 = 0;
    int lines = 0;  // tasks done: 2 N1 outputs per task
    // Output rows 2 y + odd: row y of the tile (less m, with add back on: the tile as it was loaded
    // gives its own amplitudes exactly) and S of it, a strip at a time
    auto rows = [&](int odd, float2 m, float2 add) {
#pragma unroll 1
        for (int r0 = 0; r0 < N; r0 += SR) {
            const int nr = N - r0 < SR ? N - r0 : SR;
            for (int t = tid; t < nr * N2; t += NT) {
                const int y = t / N2, n2 = t % N2;
                const float2* row = X + (r0 + y) * RS;
                float2 a[N1];
#pragma unroll
                for (int n1 = 0; n1 < N1; ++n1) {
                    const float2 v = row[N2 * n1 + n2];
                    a[n1] = make_float2(v.x - m.x, v.y - m.y);
                }
                fft::Dft<N1, -1>::run(a);
#pragma unroll
                for (int k1 = 1; k1 < N1; ++k1) a[k1] = fft::cmul(a[k1], tw[n2 * k1]);
#pragma unroll
                for (int k1 = 0; k1 < N1; ++k1) Y[y * RS + N2 * k1 + n2] = a[k1];
            }
            __syncthreads();
            for (int t = tid; t < SR * N1; t += NT)
                if (t % SR < nr) shift_middle<N1, N2>(Y + (t % SR) * RS, 1, t / SR, ph);
            __syncthreads();
            for (int t = tid; t < nr * N2; t += NT) {
                const int y = t / N2, n2 = t % N2;
                const float2* row = X + (r0 + y) * RS;
                float2* o = out + (long long)(2 * (r0 + y) + odd) * N;
                fft::inv_a_store<N1, N2>(Y + y * RS, 1, n2, tw, [&](int n, float2 v) {
                    const float2 e = row[n];
                    const float2 z = make_float2(amplitude(make_float2(e.x + add.x, e.y + add.y)),
                                                 amplitude(make_float2(v.x + mu.x, v.y + mu.y)));
                    o[n] = z;
                    const Sum de = CHIP ? (Sum)z.x : z.x - pivot, dv = CHIP ? (Sum)z.y : z.y - pivot;
                    r1 += de;
                    r2 = fma(de, de, r2);
                    r1 += dv;
                    r2 = fma(dv, dv, r2);
                });
                ++lines;
            }
            __syncthreads();
        }
    };
    const float2 zero = make_float2(0.0f, 0.0f);
    rows(0, mu, zero);
    // S down the columns, in place
    for (int t = tid; t < N * N2; t += NT) fft::fwd_a_minus<N1, N2>(X + t % N, RS, t / N, tw, mu);
    __syncthreads();
    for (int t = tid; t < N * N1; t += NT) shift_middle<N1, N2>(X + t % N, RS, t / N, ph);
    __syncthreads();
    for (int t = tid; t < N * N2; t += NT) fft::inv_a<N1, N2>(X + t % N, RS, t / N, tw);
    __syncthreads();
    rows(1, zero, mu);
    if (!stat) return;
    const double pv = pivot, nr = lines * 2 * N1;
    double sum[3] = {nr * pv + (double)r1, (double)r2 + pv * (2.0 * (double)r1 + nr * pv), (double)r2};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        sum[q] = warp_sum(sum[q]);
        if (lane == 0) red[4 * warp + q] = sum[q];
    }
    __syncthreads();
    if (tid == 0) {
        double s1 = 0.0, s2 = 0.0, about = 0.0;
        for (int w = 0; w < NT / 32; ++w) {
            s1 += red[4 * w];
            s2 += red[4 * w + 1];
            about += red[4 * w + 2];
        }
        // (a window's slack: the FP32 rounding of a thread's sum of squares, at most 100 terms for the
        // windows of up to 80 samples whose norm is used, 6e-6 relative)
        const double n = (double)F * F;
        stat[blockIdx.x] = CHIP ? chip_stat(0.0, s1, s2, n, flat) : window_stat(0.0, s1, s2, n, 1e-5 * about);
    }
}

// compiled tiles: N, N1, N2, threads, rows of a strip, CTAs per SM.  N2 = 16 where it divides: the
// last step's lanes write N2 neighbouring samples of an output row, 128 bytes.
#define AMPCOR_REFINE_TILES(X)   \
    X(16, 2, 8, 64, 16, 8)       \
    X(24, 3, 8, 96, 24, 8)       \
    X(32, 4, 8, 128, 32, 6)      \
    X(40, 5, 8, 160, 40, 5)      \
    X(48, 3, 16, 192, 48, 5)     \
    X(64, 4, 16, 256, 32, 4)     \
    X(80, 5, 16, 256, 32, 3)     \
    X(96, 6, 16, 256, 32, 2)     \
    X(120, 8, 15, 480, 60, 1)    \
    X(128, 8, 16, 512, 64, 1)    \
    X(144, 12, 12, 576, 48, 1)   \
    X(160, 10, 16, 512, 16, 1)

}  // namespace

bool refine_half_radices(int n, int& n1, int& n2)
{
#define AMPCOR_REFINE_CASE(NN, A, B, NT, SR, CTAS) \
    if (n == NN) {                                 \
        n1 = A;                                    \
        n2 = B;                                    \
        return true;                               \
    }
    AMPCOR_REFINE_TILES(AMPCOR_REFINE_CASE)
#undef AMPCOR_REFINE_CASE
    return false;
}

cudaError_t refine_half_set_smem_limits()
{
    cudaError_t e = cudaSuccess;
#define AMPCOR_REFINE_CASE(NN, A, B, NT, SR, CTAS)                                                            \
    for (auto* k : {refine_half_kernel<A, B, NT, SR, CTAS, false, false>,                                     \
                    refine_half_kernel<A, B, NT, SR, CTAS, true, false>,                                      \
                    refine_half_kernel<A, B, NT, SR, CTAS, false, true>,                                      \
                    refine_half_kernel<A, B, NT, SR, CTAS, true, true>})                                      \
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,        \
                                                       HalfGeom<A, B, NT, SR, CTAS>::smem);
    AMPCOR_REFINE_TILES(AMPCOR_REFINE_CASE)
#undef AMPCOR_REFINE_CASE
    return e;
}

cudaError_t launch_refine_half(int n, unsigned blocks, cudaStream_t st, const float2* base, const long long* off,
                               long long stride, const CoarseOut* coarse, long long pair0, long long pairs,
                               const long long* valid, const float2* tab, float* refined, long long refined_stride,
                               long long out_off, bool deramp, double flat, TileStat* stat)
{
#define AMPCOR_REFINE_CASE(NN, A, B, NT, SR, CTAS)                                                             \
    if (n == NN) {                                                                                             \
        auto* kernel = coarse ? deramp ? refine_half_kernel<A, B, NT, SR, CTAS, true, false>                   \
                                       : refine_half_kernel<A, B, NT, SR, CTAS, false, false>                  \
                              : deramp ? refine_half_kernel<A, B, NT, SR, CTAS, true, true>                    \
                                       : refine_half_kernel<A, B, NT, SR, CTAS, false, true>;                  \
        kernel<<<blocks, NT, HalfGeom<A, B, NT, SR, CTAS>::smem, st>>>(base, off, stride, coarse, pair0, pairs, \
                                                                       valid, tab, refined, refined_stride,    \
                                                                       out_off, flat, stat);                   \
        return cudaGetLastError();                                                                             \
    }
    AMPCOR_REFINE_TILES(AMPCOR_REFINE_CASE)
#undef AMPCOR_REFINE_CASE
    return cudaErrorInvalidValue;
}

}  // namespace ampcor_b200

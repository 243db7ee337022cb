// sm_100a kernels over whole rasters, once per job of the spectral form: the amplitudes of both
// rasters, and 1/sigma of every R x R box of the secondary's (the placement statistics of the coarse
// stage, shared by every window that covers a box; tgtStats.cu:88-168 of the reference computes them
// per window from a summed-area table).
//
// The statistics need FP64 sums.  A CTA takes NT columns of a block of box rows: each thread slides the
// sums of its column over R rows down the block, eight rows at a time go through shared memory, where
// a warp per row turns them into prefix sums, and the differences of these are the boxes.  Only the
// amplitudes are read and the statistics written.  The R - 1 columns that neighbouring CTAs share cost a
// quarter of the work at R = 64.
//
// What bounds them: detection, HBM (64 % of its rate) and the latency of the FP64 square roots, against
// which it takes all the warps of a multiprocessor (2 x 4,096^2 samples: 74 us, 125 with two thirds of
// them and both arrays in every thread's loop, 2 x 36 in a launch each); the statistics, instruction
// issue (55 % of the slots) between their barriers: 102 us for 4,096^2 samples at R = 64, 211 with the
// column sums in global memory between two kernels (16 bytes written and read per sample).  Both
// stages, four launches then and two now: 294 -> 184 us, at R = 128 297 -> 198, 512^2 samples and
// R = 32 33 -> 16.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "tile_common.cuh"

namespace ampcor_b200 {

namespace {

constexpr int kBoxRows = 8;  // box rows at a time

constexpr int kDetectCtas = 8;  // per multiprocessor: all its warps, against the square roots' latency

// |z| of the n samples of one array (the first `blocks` CTAs) and of the n2 samples of another
__global__ void __launch_bounds__(256, kDetectCtas)
detect_kernel(const float2* __restrict__ src, long long n, float* __restrict__ dst, const float2* __restrict__ src2,
              long long n2, float* __restrict__ dst2, int blocks)
{
    const bool second = (int)blockIdx.x >= blocks;
    if (second) {
        src = src2;
        dst = dst2;
        n = n2;
    }
    const long long at = ((long long)blockIdx.x - (second ? blocks : 0)) * 256 + threadIdx.x;
    const int step = (second ? (int)gridDim.x - blocks : blocks) * 256;
    src += at;
    dst += at;
    long long left = n - at;  // samples from this thread's on
    for (; left > 3LL * step; left -= 4LL * step) {
        float2 z[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = __ldg(src + k * (long long)step);
#pragma unroll
        for (int k = 0; k < 4; ++k) dst[k * (long long)step] = amp_of(z[k]);
        src += 4LL * step;
        dst += 4LL * step;
    }
    for (; left > 0; left -= step) {
        *dst = amp_of(__ldg(src));
        src += step;
        dst += step;
    }
}

// the same line for line into longer lines, a CTA per line
__global__ void __launch_bounds__(256, kDetectCtas)
detect_lines_kernel(DetectLines a, DetectLines b, int blocks)
{
    const bool second = (int)blockIdx.x >= blocks;
    const DetectLines d = second ? b : a;
    const int first = (int)blockIdx.x - (second ? blocks : 0), step = second ? (int)gridDim.x - blocks : blocks;
    for (long long y = first; y < d.lines; y += step) {
        const float2* src = d.src + y * d.samples;
        float* dst = d.dst + y * d.pitch;
        long long x = threadIdx.x;
        for (; x + 768 < d.samples; x += 1024) {
            float2 z[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) z[k] = __ldg(src + x + 256 * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) dst[x + 256 * k] = amp_of(z[k]);
        }
        for (; x < d.samples; x += 256) dst[x] = amp_of(__ldg(src + x));
    }
}

// element i of a padded row of FP64 sums: 16 neighbours sit in different banks, and so do the first of
// 16 lanes' NT / 32 neighbours (a slot left out every 8 instead costs half of the wavefronts' rate)
__device__ __forceinline__ int padded(int i) { return i + (i >> 4); }

template <int NT>
constexpr int kBoxRow = NT + NT / 16 + 1;  // slots of a row

template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
box_stats_kernel(const float* __restrict__ a, int samples, int pitch, int R, int block_rows, int row_lo, int row_hi,
                 float* __restrict__ inv)
{
    constexpr int kRow = kBoxRow<NT>, kPer = NT / 32;
    extern __shared__ __align__(16) double sums[];  // 2 kBoxRows rows: the sums, then the sums of squares
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cols = NT + 1 - R;  // boxes to a row
    const int x = blockIdx.x * cols + tid;
    const int y0 = (row_lo / block_rows + blockIdx.y) * block_rows;
    const int y1 = min(y0 + block_rows, row_hi);
    // (threads past the raster's last column sum that column again: no box uses it)
    const float* leave = a + (long long)y0 * pitch + min(x, samples - 1);  // row y of this column
    const float* enter = leave;                                              // and row y + R
    double s1 = 0.0, s2 = 0.0;
    auto add = [&](auto rows) {
        constexpr int kN = decltype(rows)::value;
        float v[kN];
#pragma unroll
        for (int k = 0; k < kN; ++k) v[k] = __ldg(enter + k * pitch);
        enter += kN * pitch;
        double c1[2] = {0.0, 0.0}, c2[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < kN; ++k) {
            const double t = v[k];
            c1[k & 1] += t;
            c2[k & 1] += t * t;
        }
        s1 += c1[0] + c1[1];
        s2 += c2[0] + c2[1];
    };
    int i = 0;
    for (; i + 16 <= R; i += 16) add(std::integral_constant<int, 16>{});
    for (; i < R; ++i) add(std::integral_constant<int, 1>{});
    const double per_cell = 1.0 / ((double)R * (double)R);
    float* out = inv + (long long)y0 * pitch + x;
    const bool box = tid < cols && x + R <= samples;
    for (int y = y0; y < y1; y += kBoxRows) {
        float up[kBoxRows], dn[kBoxRows];
        if (y + kBoxRows < y1) {
#pragma unroll
            for (int r = 0; r < kBoxRows; ++r) {
                up[r] = __ldg(leave + r * pitch);
                dn[r] = __ldg(enter + r * pitch);
            }
        } else {
#pragma unroll
            for (int r = 0; r < kBoxRows; ++r) {
                const bool in = y + r + 1 < y1;
                up[r] = in ? __ldg(leave + r * pitch) : 0.0f;
                dn[r] = in ? __ldg(enter + r * pitch) : 0.0f;
            }
        }
        leave += kBoxRows * pitch;
        enter += kBoxRows * pitch;
        double* mine = sums + padded(tid);
#pragma unroll
        for (int r = 0; r < kBoxRows; ++r) {
            mine[r * kRow] = s1;
            mine[(kBoxRows + r) * kRow] = s2;
            const double p = dn[r], q = up[r];
            s1 += p - q;
            s2 += p * p - q * q;
        }
        __syncthreads();
        // exclusive prefix sums, a row to a warp
        for (int t = warp; t < 2 * kBoxRows; t += NT / 32) {
            double* row = sums + t * kRow + lane * kPer + lane * kPer / 16;
            double run = 0.0;
#pragma unroll
            for (int k = 0; k < kPer; ++k) run += row[k + k / 16];
            double incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double below = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += below;
            }
            run = incl - run;
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const double v = row[k + k / 16];
                row[k + k / 16] = run;
                run += v;
            }
            if (lane == 31) sums[t * kRow + padded(NT)] = run;
        }
        __syncthreads();
        if (box) {
            const double* lo = sums + padded(tid);
            const double* hi = sums + padded(tid + R);
            const int first = row_lo - y, last = y1 - y;
#pragma unroll
            for (int r = 0; r < kBoxRows; ++r) {
                const double b1 = hi[r * kRow] - lo[r * kRow], b2 = hi[(kBoxRows + r) * kRow] - lo[(kBoxRows + r) * kRow];
                const float var = (float)(b2 - b1 * b1 * per_cell);
                if (r >= first && r < last) out[r * pitch] = var > 0.0f ? __frsqrt_rn(var) : 0.0f;
            }
        }
        out += kBoxRows * pitch;
        __syncthreads();
    }
}

template <int NT>
constexpr int box_smem()
{
    return 2 * kBoxRows * kBoxRow<NT> * (int)sizeof(double);
}

}  // namespace

cudaError_t raster_set_smem_limits()
{
    return cudaFuncSetAttribute(box_stats_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, box_smem<512>());
}

cudaError_t launch_detect(cudaStream_t st, const float2* src, long long n, float* dst, const float2* src2,
                          long long n2, float* dst2)
{
    // CTAs by the sizes of the arrays, one at least for each that has samples
    const long long total = n + n2, all = std::min<long long>((total + 1023) / 1024 + 1, 148LL * kDetectCtas);
    if (total <= 0) return cudaSuccess;
    long long blocks = (all * n + total / 2) / total;
    blocks = n2 <= 0 ? all : n <= 0 ? 0 : std::min(std::max(blocks, 1LL), all - 1);
    detect_kernel<<<(unsigned)all, 256, 0, st>>>(src, n, dst, src2, n2, dst2, (int)blocks);
    return cudaGetLastError();
}

cudaError_t launch_detect_lines(cudaStream_t st, const DetectLines& a, const DetectLines& b)
{
    const long long la = std::max(a.lines, 0LL), lb = std::max(b.lines, 0LL);
    const long long all = std::min<long long>(la + lb, 148LL * kDetectCtas);
    if (all <= 0) return cudaSuccess;
    long long blocks = (all * la + (la + lb) / 2) / (la + lb);
    blocks = lb == 0 ? all : la == 0 ? 0 : std::min(std::max(blocks, 1LL), all - 1);
    detect_lines_kernel<<<(unsigned)all, 256, 0, st>>>(a, b, (int)blocks);
    return cudaGetLastError();
}

// columns of a CTA: at least twice the box (no chip of the spectral form has more than 160 samples a side)
static int box_threads(int R) { return R <= 96 ? 256 : 512; }

int box_block_rows(long long rows, long long samples, int R, unsigned sms)
{
    const long long cols = box_threads(R) + 1 - R, across = (std::max<long long>(samples - R + 1, 1) + cols - 1) / cols;
    int block = 64;
    while (block > kBoxRows && across * ((rows + block - 1) / block) < 2LL * sms) block /= 2;
    return block;
}

cudaError_t launch_box_stats(cudaStream_t st, const float* a, long long samples, long long pitch, int R,
                             int block_rows, long long row_lo, long long row_hi, float* inv)
{
    const int nt = box_threads(R);
    const long long cols = nt + 1 - R, first = row_lo / block_rows;
    if (R > 256) return cudaErrorInvalidValue;
    if (samples < R || row_hi <= row_lo) return cudaSuccess;
    const dim3 grid((unsigned)((samples - R + cols) / cols), (unsigned)((row_hi + block_rows - 1) / block_rows - first));
    if (nt == 256)
        box_stats_kernel<256><<<grid, 256, box_smem<256>(), st>>>(a, (int)samples, (int)pitch, R, block_rows, (int)row_lo, (int)row_hi, inv);
    else
        box_stats_kernel<512><<<grid, 512, box_smem<512>(), st>>>(a, (int)samples, (int)pitch, R, block_rows, (int)row_lo, (int)row_hi, inv);
    return cudaGetLastError();
}

static __global__ void __launch_bounds__(128)
join_parts_kernel(const CoarseOut* parts, const float* peaks, long long stride, long long pair0, unsigned n,
                  const long long* valid, int C, int Cq, int m, int W, int E, CoarseOut* coarse, float* coarse_peak,
                  const float* part_surfaces, float* surfaces)
{
    const long long p = pair0 + blockIdx.x;
    if (valid[p] < 0) return;
    const int s = C - Cq;
    if (threadIdx.x == 0) {
        // the first maximum in row-major order over all placements (a part without one reports a cell outside)
        float bv = -INFINITY;
        int bi = INT_MAX;
        for (int k = 0; k < 4; ++k) {
            const CoarseOut c = parts[k * stride + p];
            if ((unsigned)c.u < (unsigned)Cq && (unsigned)c.v < (unsigned)Cq)
                better(bv, bi, peaks[k * stride + p], (c.u + (k >> 1) * s) * C + c.v + (k & 1) * s);
        }
        const int u = bi / C, v = bi - u * C;
        coarse[p] = nudged(u, v, E - 2 * m, W, m);
        coarse_peak[p] = bv;
    }
    if (surfaces) {
        for (int i = threadIdx.x; i < C * C; i += 128) {
            const int u = i / C, v = i - u * C, k = (u >= Cq ? 2 : 0) + (v >= Cq ? 1 : 0);
            surfaces[p * C * C + i] = part_surfaces[((long long)k * n + blockIdx.x) * Cq * Cq +
                                                    (u - (k >> 1) * s) * Cq + v - (k & 1) * s];
        }
    }
}

cudaError_t launch_join_parts(cudaStream_t st, const CoarseOut* parts, const float* peaks, long long stride,
                              long long pair0, unsigned n, const long long* valid, int C, int Cq, int m, int W, int E,
                              CoarseOut* coarse, float* coarse_peak, const float* part_surfaces, float* surfaces)
{
    join_parts_kernel<<<n, 128, 0, st>>>(parts, peaks, stride, pair0, n, valid, C, Cq, m, W, E, coarse, coarse_peak,
                                         part_surfaces, surfaces);
    return cudaGetLastError();
}

}  // namespace ampcor_b200

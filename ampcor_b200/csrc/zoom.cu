// Zoom of the refined correlation surfaces (sm_100a, packed FP32): the first maximum of the
// band-limited interpolation of every Cf x Cf surface G by a factor z, and the offsets.
//
// The reference zooms each surface with a zero-padded FFT and takes the first maximum of the
// Z x Z result (Z = z Cf; correlators/kernels.h zoomcor, maxcor).  That interpolation is the
// product Zm = U G U^T with U the Z x Cf Dirichlet interpolation matrix.  Only the cells that can
// hold the maximum are formed, in three steps that rest on two facts about the band-limited
// interpolation f(x) = sum_b D(x - b) g_b of Cf samples (D sums to 1 over b, its squares sum to 1,
// those of D'' to kappa^2):
//   (1) f(x) <= c + |g - c| for any constant c, and |f''(x)| <= kappa |g - c| (Cauchy-Schwarz);
//   (2) between two points h apart f stays below the larger end value + h^2 / 8 sup |f''|, and
//       so does the norm of a vector of such functions.
// Columns: T = G U^T is formed at every s-th column (s = z / 2: half a sample of G).  Its entries
// are cells of Zm; an interval between two of its columns whose norms, by (2) and (1), stay below
// the largest entry is left out.  Rows: the kept columns' cells are formed at every s-th row, and
// the intervals that by (2) stay below the largest cell seen are left out.  Last, the cells of
// the kept rows and columns.  The bounds are widened by more than the sums round.  A correlation
// peak stands over a background of 0.02-0.2, so about 30 of the 264 columns and 20 of the 264 rows
// of the production surface remain; noise keeps everything, at the cost of the whole product, and
// so does NaN (comparisons are written to keep it).
//
// What bounds it: the FP32 pipes and instruction issue.  A team of three warps (nine where
// a multiprocessor has few pairs) walks one pair at a time; the lanes of a warp are 8 rows of U x 4 rows of the other factor, a thread three of the
// former against three of the latter: 18 packed FMAs per six 128-bit shared loads of one
// wavefront each (four rows a thread leave a third of the lanes idle over the 66 sampled rows: 364
// against 317 us below).  The teams of a CTA (one CTA per SM) share U and nothing else, so one
// team's barriers hide behind the others' arithmetic.  Measured on B200, 14,641 surfaces of
// 33 x 33 at z = 8: 317 us.  The whole product on the tensor cores (3xTF32, the Z x Z accumulators
// reduced from tensor memory) took 1,280 us, the kept columns alone on the tensor cores 490 us
// (their waits and operand splits, not the products), both with zoomed maxima 4e-7 off FP64 against
// 1e-7 here.  900 surfaces at z = 16: 68 us against 854 us (the whole product in FP32).
#include <algorithm>

#include "kernels.cuh"
#include "tcgen05.cuh"
#include "tile_common.cuh"

namespace ampcor_b200 {

namespace {

constexpr int kCols = kZoomCols;

template <int TEAM>
__device__ __forceinline__ void team_sync(int team)
{
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(TEAM) : "memory");
}

// acc += a * b on two packed floats
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ float halves(unsigned long long v)
{
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}

constexpr int kNR = 3, kNC = 3;      // rows of U and of the other factor per thread
constexpr int kRows = 8 * kNR;       // rows a warp forms at a time: its lanes are 8 rows x 4 columns
constexpr int kGroup = kZoomTeam / 32;  // warps of a group: they share out the rows
constexpr int kStep = kGroup * kRows;
static_assert(kCols % (4 * kNC) == 0, "a batch is whole blocks of columns");

// out[i][k] = row ra[i] of U times row rb + 4 k of b (rows of kp4 float4, zero past Cf); kp4 is odd,
// so that rows next to each other start in other banks
__device__ __forceinline__ void dots(const float* U, const int (&ra)[kNR], const float* b, int rb, int kp4,
                                     float (&out)[kNR][kNC])
{
    const ulonglong2* u2[kNR];
    const ulonglong2* b2[kNC];
#pragma unroll
    for (int i = 0; i < kNR; ++i) u2[i] = reinterpret_cast<const ulonglong2*>(U) + ra[i] * kp4;
#pragma unroll
    for (int k = 0; k < kNC; ++k) b2[k] = reinterpret_cast<const ulonglong2*>(b) + (rb + 4 * k) * kp4;
    unsigned long long acc[kNR][kNC];
#pragma unroll
    for (int i = 0; i < kNR; ++i)
#pragma unroll
        for (int k = 0; k < kNC; ++k) acc[i][k] = 0ull;
#pragma unroll 3
    for (int c = 0; c < kp4; ++c) {
        ulonglong2 v[kNC];
#pragma unroll
        for (int k = 0; k < kNC; ++k) v[k] = b2[k][c];
#pragma unroll
        for (int i = 0; i < kNR; ++i) {
            const ulonglong2 u = u2[i][c];
#pragma unroll
            for (int k = 0; k < kNC; ++k) {
                fma2(acc[i][k], u.x, v[k].x);
                fma2(acc[i][k], u.y, v[k].y);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kNR; ++i)
#pragma unroll
        for (int k = 0; k < kNC; ++k) out[i][k] = halves(acc[i][k]);
}

struct ZoomTeam {
    float* G;             // g_rows rows of kp4 float4, zero past Cf
    float* T;             // kCols kept columns of T, kp4 float4 each
    float* val;           // J a group: the norms of T's sampled columns, then the maxima of the sampled rows
    float* red;           // a slot per warp, four times (16 or 32 in all), the last one after them
    unsigned* cols;       // Z: the kept columns, index | row of U << 16
    unsigned* rows;       // Z: the kept rows, the same
};

// The indices of the kept intervals into out, in increasing order (every lane of the warp gets
// their number): interval j, [s j, s (j + 1)), is kept unless the larger end value + add stays
// below best.  first: whether the interval's first index (a sample) is listed too.
__device__ __forceinline__ int kept_intervals(const float* val, const ZoomGeomCols& g, float add, float best,
                                              bool first, unsigned* out)
{
    const int lane = threadIdx.x & 31, lo = first ? 0 : 1, per = g.s - lo;
    int n = 0;
    for (int j0 = 0; j0 < g.J; j0 += 32) {
        const int j = j0 + lane, j1 = j + 1 < g.J ? j + 1 : 0;
        const bool keep = j < g.J && (!(val[j] + add < best) || !(val[j1] + add < best));
        const unsigned m = __ballot_sync(kFull, keep);
        const int at = n + __popc(m & ((1u << lane) - 1u)) * per;
        n += __popc(m) * per;
        if (keep)
            for (int k = 0; k < per; ++k)
                if (g.s * j + lo + k < g.Z) out[at + k] = (unsigned)(g.s * j + lo + k) | (unsigned)((lo + k) * g.Jp + j) << 16;
        // (the last interval may be short: nothing follows it)
        const int over = g.s * g.J - g.Z;
        if (over > 0 && j0 + 32 >= g.J && (m >> ((g.J - 1) & 31)) & 1u) n -= min(over, per);
    }
    __syncwarp();
    return n;
}

// the maximum over a team of (value, index), ends with a barrier; every thread gets it
template <int TEAM>
__device__ __forceinline__ void team_argmax(float& bv, int& bi, float* red, int team, int tid)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(kFull, bv, o);
        const int oi = __shfl_xor_sync(kFull, bi, o);
        better(bv, bi, ov, oi);
    }
    constexpr int kWarpsT = TEAM / 32;
    if ((tid & 31) == 0) {
        red[tid >> 5] = bv;
        reinterpret_cast<int*>(red)[kWarpsT + (tid >> 5)] = bi;
    }
    team_sync<TEAM>(team);
#pragma unroll
    for (int w = 0; w < kWarpsT; ++w) better(bv, bi, red[w], reinterpret_cast<int*>(red)[kWarpsT + w]);
    team_sync<TEAM>(team);
}

}  // namespace

// GROUPS groups of three warps to a team: they share out the columns of a product
template <int GROUPS>
__global__ void __launch_bounds__(zoom_teams(GROUPS) * GROUPS * kZoomTeam, 1)
zoom_kernel(const float* gam, long long pair0, long long pairs, const long long* ref_off, ZoomGeomCols g,
            const float* u_g, const CoarseOut* coarse, const float* coarse_peak, const FineOut* fout, int margin,
            int refine_factor, int refine_margin, int ref_compat, float2* offsets, PairDiag* diag,
            unsigned int* err_out, int stall)
{
    extern __shared__ __align__(16) unsigned char zsm[];
    constexpr int kTeam = GROUPS * kZoomTeam, kWarpsT = kTeam / 32, kTotal = 4 * kWarpsT;
    const int team = threadIdx.x / kTeam, tid = threadIdx.x - team * kTeam, teams = blockDim.x / kTeam;
    const int Cf = g.Cf, Z = g.Z, kp4 = g.kp4;
    float* U = reinterpret_cast<float*>(zsm);
    ZoomTeam t;
    unsigned char* own = zsm + g.off_team + team * g.team_bytes;
    t.G = reinterpret_cast<float*>(own);
    t.T = t.G + g.g_rows * 4 * kp4;
    t.val = t.T + kCols * 4 * kp4;
    const int Jv = (g.J + 3) / 4 * 4;
    t.red = t.val + GROUPS * Jv;
    t.cols = reinterpret_cast<unsigned*>(t.red + (kTotal + 4) / 4 * 4);
    t.rows = t.cols + (Z + 3) / 4 * 4;
    const int lane = tid & 31, warp = tid >> 5, rl = lane >> 2, cl = lane & 3;
    const int grp = warp / kGroup, wrow = (warp - grp * kGroup) * kRows;  // this warp's share: columns, rows
    // element tid of a row-major array of Cf columns, and the one kTeam further on
    const int ta0 = tid / Cf, tq0 = tid - ta0 * Cf, da = kTeam / Cf, dq = kTeam - da * Cf;
    auto walk = [&](int& a, int& q) {
        a += da;
        q += dq;
        if (q >= Cf) {
            q -= Cf;
            ++a;
        }
    };

    // a failure-detection test: every thread waits on a barrier that nothing completes; the
    // bounded wait runs out, and the CTA skips its pairs and reports the time-out
    if (stall) {
        uint64_t& never = *reinterpret_cast<uint64_t*>(zsm);
        int& err = *reinterpret_cast<int*>(zsm + 8);
        if (threadIdx.x == 0) {
            err = 0;
            mbar_init(&never, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        mbar_wait(&never, 0u, &err, kStallCycles);
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(err_out, 1u);
        return;
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < g.s * g.Jp * kp4; i += blockDim.x)
        reinterpret_cast<float4*>(U)[i] = __ldg(reinterpret_cast<const float4*>(u_g) + i);
    for (int i = tid; i < (g.g_rows + kCols) * 4 * kp4; i += kTeam) t.G[i] = 0.0f;  // (G and T)
    __syncthreads();

    for (long long b = (long long)blockIdx.x * teams + team; b < pairs; b += (long long)gridDim.x * teams) {
        const long long p = pair0 + b;
        if (ref_off[p] < 0) {
            if (tid == 0) {
                offsets[p] = make_float2(NAN, NAN);
                if (diag) diag[p] = PairDiag{-1, -1, -1, -1, -1, -1, -1, -1, NAN, NAN, NAN, 0.0f};
            }
            continue;
        }
        const float* src = gam + b * Cf * Cf;
        float g1 = 0.0f, g2 = 0.0f;
        {
            // (row, column) of this thread's samples walk along by kTeam; a batch of loads in flight
            constexpr int kLoads = 12 / GROUPS;
            int a = ta0, q = tq0;
            for (int i0 = tid; i0 < Cf * Cf; i0 += kLoads * kTeam) {
                float gv[kLoads];
#pragma unroll
                for (int k = 0; k < kLoads; ++k) gv[k] = i0 + k * kTeam < Cf * Cf ? __ldg(src + i0 + k * kTeam) : 0.0f;
#pragma unroll
                for (int k = 0; k < kLoads; ++k) {
                    if (i0 + k * kTeam < Cf * Cf) {
                        t.G[a * 4 * kp4 + q] = gv[k];
                        g1 += gv[k];
                        g2 = fmaf(gv[k], gv[k], g2);
                    }
                    walk(a, q);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            g1 += __shfl_xor_sync(kFull, g1, o);
            g2 += __shfl_xor_sync(kFull, g2, o);
        }
        if (lane == 0) {
            t.red[warp] = g1;
            t.red[kWarpsT + warp] = g2;
        }
        team_sync<kTeam>(team);
        g1 = g2 = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) {
            g1 += t.red[w];
            g2 += t.red[kWarpsT + w];
        }
        // the constant c, and |G - c| from above (the slack covers the FP32 sums)
        const float c = g1 / (float)(Cf * Cf);
        const float gn = sqrtf(fmaxf(g2 - g1 * c, 0.0f) + 1e-5f * g2);

        // T at every s-th column: the largest entry, the norm of every column
        float best = -INFINITY;
        for (int j0 = wrow; j0 < g.J; j0 += kStep) {
            int q[kNR];
            float nn[kNR];
#pragma unroll
            for (int i = 0; i < kNR; ++i) {
                q[i] = min(j0 + rl + 8 * i, g.J - 1);
                nn[i] = 0.0f;
            }
            for (int a = 4 * kNC * grp; a < Cf; a += 4 * kNC * GROUPS) {
                float v[kNR][kNC];
                dots(U, q, t.G, a + cl, kp4, v);
#pragma unroll
                for (int k = 0; k < kNC; ++k)
                    if (a + cl + 4 * k < Cf)
#pragma unroll
                        for (int i = 0; i < kNR; ++i) {
                            const float d = v[i][k] - c;
                            nn[i] = fmaf(d, d, nn[i]);
                            best = fmaxf(best, v[i][k]);
                        }
            }
#pragma unroll
            for (int i = 0; i < kNR; ++i) {
                nn[i] += __shfl_xor_sync(kFull, nn[i], 1);
                nn[i] += __shfl_xor_sync(kFull, nn[i], 2);
                if (cl == i && j0 + rl + 8 * i < g.J) t.val[grp * Jv + j0 + rl + 8 * i] = GROUPS == 1 ? sqrtf(nn[i]) : nn[i];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(kFull, best, o));
        if (lane == 0) t.red[2 * kWarpsT + warp] = best;
        team_sync<kTeam>(team);
        if constexpr (GROUPS > 1) {
            for (int j = tid; j < g.J; j += kTeam) {
                float n2 = 0.0f;
#pragma unroll
                for (int i = 0; i < GROUPS; ++i) n2 += t.val[i * Jv + j];
                t.val[j] = sqrtf(n2);
            }
            team_sync<kTeam>(team);
        }
        float top = 0.0f;  // the largest norm
        for (int j = lane; j < g.J; j += 32) top = fmaxf(top, t.val[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(kFull, top, o));
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) best = fmaxf(best, t.red[2 * kWarpsT + w]);
        const float slack = 1e-4f * (gn + fabsf(c)) + 1e-6f;
        // (warp 0 writes the list, its length goes through the reduction slots)
        if (warp == 0) {
            const int n = kept_intervals(t.val, g, c + g.curv * gn + slack, best, true, t.cols);
            if (lane == 0) reinterpret_cast<int*>(t.red)[kTotal] = n;
        }
        team_sync<kTeam>(team);
        const int total = reinterpret_cast<int*>(t.red)[kTotal];
        const float rise = g.curv * (top + g.curv * gn) + slack;  // of a kept column between two rows

        float bv = -INFINITY;
        int bi = INT_MAX;
        // cells of rows pa (rows ra of U) and the nb columns in T: this thread's first maximum, and the maximum
        // of each row over the warp's lanes
        auto cells = [&](const int (&ra)[kNR], const int (&pa)[kNR], int c0, int nb, float (&rm)[kNR]) {
#pragma unroll
            for (int i = 0; i < kNR; ++i) rm[i] = -INFINITY;
            for (int s = 4 * kNC * grp; s < nb; s += 4 * kNC * GROUPS) {
                float v[kNR][kNC];
                dots(U, ra, t.T, s + cl, kp4, v);
#pragma unroll
                for (int k = 0; k < kNC; ++k) {
                    const int q = s + cl + 4 * k;
                    if (q < nb)
#pragma unroll
                        for (int i = 0; i < kNR; ++i) {
                            rm[i] = fmaxf(rm[i], v[i][k]);
                            if (v[i][k] >= bv) better(bv, bi, v[i][k], pa[i] * Z + (int)(t.cols[c0 + q] & 0xffffu));
                        }
                }
            }
        };
        for (int c0 = 0; c0 < total; c0 += kCols) {
            const int nb = min(kCols, total - c0), nt = (Cf + 2) / 3;  // (3 nt <= g_rows)
            // the batch's columns of T: a task is one column against three rows of G, nt apart
            for (int i = tid; i < nb * nt; i += kTeam) {
                const int q = i / nt, a = i - q * nt;
                const ulonglong2* u2 = reinterpret_cast<const ulonglong2*>(U) + (t.cols[c0 + q] >> 16) * kp4;
                const ulonglong2* g0 = reinterpret_cast<const ulonglong2*>(t.G) + a * kp4;
                unsigned long long acc[3] = {0ull, 0ull, 0ull};
#pragma unroll 3
                for (int k = 0; k < kp4; ++k) {
                    const ulonglong2 u = u2[k];
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        const ulonglong2 v = g0[r * nt * kp4 + k];
                        fma2(acc[r], u.x, v.x);
                        fma2(acc[r], u.y, v.y);
                    }
                }
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    if (a + r * nt < Cf) t.T[q * 4 * kp4 + a + r * nt] = halves(acc[r]);
            }
            team_sync<kTeam>(team);
            // every s-th row
            for (int j0 = wrow; j0 < g.J; j0 += kStep) {
                int ra[kNR], pa[kNR];
                float rm[kNR];
#pragma unroll
                for (int i = 0; i < kNR; ++i) {
                    ra[i] = min(j0 + rl + 8 * i, g.J - 1);
                    pa[i] = g.s * ra[i];
                }
                cells(ra, pa, c0, nb, rm);
#pragma unroll
                for (int i = 0; i < kNR; ++i) {
                    rm[i] = fmaxf(rm[i], __shfl_xor_sync(kFull, rm[i], 1));
                    rm[i] = fmaxf(rm[i], __shfl_xor_sync(kFull, rm[i], 2));
                    if (cl == i && j0 + rl + 8 * i < g.J) t.val[grp * Jv + j0 + rl + 8 * i] = rm[i];
                }
            }
            team_sync<kTeam>(team);
            if constexpr (GROUPS > 1) {
                for (int j = tid; j < g.J; j += kTeam) {
                    float m = t.val[j];
#pragma unroll
                    for (int i = 1; i < GROUPS; ++i) m = fmaxf(m, t.val[i * Jv + j]);
                    t.val[j] = m;
                }
                team_sync<kTeam>(team);
            }
            // the rows between them that can hold more than the largest cell seen
            if (warp == 0) {
                float seen = best;
                for (int j = lane; j < g.J; j += 32) seen = fmaxf(seen, t.val[j]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) seen = fmaxf(seen, __shfl_xor_sync(kFull, seen, o));
                const int n = kept_intervals(t.val, g, rise, seen, false, t.rows);
                if (lane == 0) reinterpret_cast<int*>(t.red)[kTotal] = n;
            }
            team_sync<kTeam>(team);
            const int nr = reinterpret_cast<int*>(t.red)[kTotal];
            for (int r0 = wrow; r0 < nr; r0 += kStep) {
                int ra[kNR], pa[kNR];
                float rm[kNR];
#pragma unroll
                for (int i = 0; i < kNR; ++i) {
                    const unsigned e = t.rows[min(r0 + rl + 8 * i, nr - 1)];
                    ra[i] = (int)(e >> 16);
                    pa[i] = (int)(e & 0xffffu);
                }
                cells(ra, pa, c0, nb, rm);
            }
            team_sync<kTeam>(team);
        }
        team_argmax<kTeam>(bv, bi, t.red, team, tid);
        if (tid == 0) {
            const CoarseOut co = coarse[p];
            const FineOut fo = fout[p];
            const int fp = bi / Z, fq = bi - fp * Z;
            const float zoom = (float)(refine_factor * g.z);
            float dy, dx;
            if (ref_compat) {
                // offsets.cu:124-125, refine margin subtracted from the nudged corner once more
                dy = ((float)co.top - (float)margin) + ((float)fp / zoom - (float)refine_margin);
                dx = ((float)co.left - (float)margin) + ((float)fq / zoom - (float)refine_margin);
            } else {
                dy = (float)(co.top - margin) + (float)fp / zoom;
                dx = (float)(co.left - margin) + (float)fq / zoom;
            }
            offsets[p] = make_float2(dy, dx);
            if (diag) {
                diag[p] = PairDiag{co.u, co.v, co.top, co.left, fo.u, fo.v, fp, fq, coarse_peak[p],
                                   fo.peak, bv, 0.0f};
            }
        }
    }
}

cudaError_t zoom_set_smem_limits()
{
    const int limit = 227 * 1024;
    cudaError_t e = cudaFuncSetAttribute(zoom_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(zoom_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    return e;
}

cudaError_t launch_zoom_kernel(unsigned sms, cudaStream_t st, const float* gam, long long pair0, unsigned n,
                               const long long* ref_off, const ZoomGeomCols& g, const float* u,
                               const CoarseOut* coarse, const float* coarse_peak, const FineOut* fout, int margin,
                               int refine_factor, int refine_margin, int ref_compat, float2* offsets,
                               PairDiag* diag, unsigned int* err_out, int stall)
{
    // as many teams to a CTA as keep every multiprocessor busy
    const unsigned each = (n + sms - 1) / sms;
    auto launch = [&](auto* kernel, ZoomGeomCols gg, unsigned fit, int threads) {
        const unsigned teams = std::min(fit, each), blocks = std::min<unsigned>((n + teams - 1) / teams, sms);
        kernel<<<blocks, teams * threads, gg.off_team + teams * gg.team_bytes, st>>>(
            gam, pair0, n, ref_off, gg, u, coarse, coarse_peak, fout, margin, refine_factor, refine_margin,
            ref_compat, offsets, diag, err_out, stall);
    };
    // Three groups to a team where a multiprocessor has few pairs: a pair's chain of products is what such
    // a call waits for.  225 surfaces of 33 x 33 at z = 8: 24.2 -> 20.5 us, of noise 127 -> 92 (z = 16: 32.4 ->
    // 24.5, 310 -> 201); 444 surfaces, three to a multiprocessor, 25.9 -> 22.6, but 17 x 17 samples have
    // too few rows for that: 14.3 -> 16.3.
    ZoomGeomCols wide = g;
    wide.team_bytes += 2 * ((g.J + 3) / 4 * 4) * 4 + 96;
    const unsigned fit = (unsigned)std::min<long>(g.J > 48 ? zoom_teams(3) : 2, (227L * 1024 - g.off_team) / wide.team_bytes);
    if (each <= fit)
        launch(zoom_kernel<3>, wide, fit, 3 * kZoomTeam);
    else
        launch(zoom_kernel<1>, g, (unsigned)g.teams, kZoomTeam);
    return cudaGetLastError();
}

}  // namespace ampcor_b200

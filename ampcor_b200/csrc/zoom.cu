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
// the intervals that by (2) stay below the largest cell seen are left out; the second derivative down a
// column is bounded by the column's own norm, the largest of 36 (or 8, 24) neighbours.  Last, the
// cells of the kept rows and columns.  The bounds are widened by more than the sums round.  A
// correlation peak stands over a background of 0.02-0.2, so about 30 of the 264 columns and 20 of the
// 264 rows of the production surface remain.  Noise keeps every column but only a tenth of the rows
// between the sampled ones (a third with a bound from the whole surface's norm).  A surface with a NaN
// sample is NaN in every cell (0 times NaN) and has no maximum.
//
// What bounds it: shared-memory wavefronts and the latency of packed FMAs.  A team of three warps (nine
// where a multiprocessor has two or three pairs, twelve of a kernel of its own where it has one) walks
// one pair at a time; the lanes of a warp are 8 rows of one factor x 4 of the other, a thread three of the
// former against three of the latter: 18 packed FMAs per six 128-bit shared loads (two wavefronts a load
// on the side of 8, four on the side of 4; four rows a thread leave a third of the lanes idle over the
// 66 sampled rows).  The teams of a CTA (one CTA per SM) share U and nothing else, so one team's
// barriers hide behind the others' arithmetic.
//
// Measured on B200, 33 x 33 samples at z = 8, peaks at 10 to -6 dB / noise.  14,641 surfaces: 301 /
// 1,680 us (the whole product on the tensor cores, 3xTF32, with the accumulators reduced from tensor
// memory, 1,280 either way and its maxima 4e-7 off FP64 against 1e-7 here).  225 surfaces: 21 / 57 us, on the
// tensor cores 35; 100 surfaces: 16 / 27, on the tensor cores 20.  At z = 16, 14,641 surfaces: 360 / 3,400 us
// against 12,020 of the whole product in FP32.
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
constexpr int kWide = 4 * kNC;
constexpr int kGroup = 3;            // warps of a group: they share out the sampled columns
constexpr int kStep = kGroup * kRows;
static_assert(kCols % kWide == 0 && kWide == 12 && kRows == 24, "the layout's blocks");

// out[i][k] = row ra[i] of u times row rb[k] of b (rows of kp4 float4, zero past Cf); kp4 is odd,
// so that rows next to each other start in other banks.  The sums' order is that of the columns, whatever
// the block.  AHEAD: the next step's loads are under way during a step's products (for blocks whose loads
// of several steps would not fit the registers).
template <int NR, int NC, bool AHEAD = false>
__device__ __forceinline__ void dots(const float* u, const int (&ra)[NR], const float* b, const int (&rb)[NC],
                                     int kp4, float (&out)[NR][NC])
{
    const ulonglong2* u2[NR];
    const ulonglong2* b2[NC];
#pragma unroll
    for (int i = 0; i < NR; ++i) u2[i] = reinterpret_cast<const ulonglong2*>(u) + ra[i] * kp4;
#pragma unroll
    for (int k = 0; k < NC; ++k) b2[k] = reinterpret_cast<const ulonglong2*>(b) + rb[k] * kp4;
    unsigned long long acc[NR][NC];
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int k = 0; k < NC; ++k) acc[i][k] = 0ull;
    if constexpr (AHEAD) {
        ulonglong2 u[NR], v[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) v[k] = b2[k][0];
#pragma unroll
        for (int i = 0; i < NR; ++i) u[i] = u2[i][0];
#pragma unroll 1
        for (int c = 0; c < kp4; ++c) {
            const int next = c + 1 < kp4 ? c + 1 : c;
            ulonglong2 un[NR], vn[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) vn[k] = b2[k][next];
#pragma unroll
            for (int i = 0; i < NR; ++i) un[i] = u2[i][next];
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    fma2(acc[i][k], u[i].x, v[k].x);
                    fma2(acc[i][k], u[i].y, v[k].y);
                }
#pragma unroll
            for (int k = 0; k < NC; ++k) v[k] = vn[k];
#pragma unroll
            for (int i = 0; i < NR; ++i) u[i] = un[i];
        }
    } else {
#pragma unroll 3
        for (int c = 0; c < kp4; ++c) {
            ulonglong2 v[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) v[k] = b2[k][c];
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const ulonglong2 u = u2[i][c];
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    fma2(acc[i][k], u.x, v[k].x);
                    fma2(acc[i][k], u.y, v[k].y);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int k = 0; k < NC; ++k) out[i][k] = halves(acc[i][k]);
}

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
    constexpr int WARPS = TEAM / 32;
    if ((tid & 31) == 0) {
        red[tid >> 5] = bv;
        reinterpret_cast<int*>(red)[WARPS + (tid >> 5)] = bi;
    }
    team_sync<TEAM>(team);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) better(bv, bi, red[w], reinterpret_cast<int*>(red)[WARPS + w]);
    team_sync<TEAM>(team);
}

// a failure-detection test: every thread waits on a barrier that nothing completes; the
// bounded wait runs out, and the CTA skips its pairs and reports the time-out
__device__ __forceinline__ bool zoom_stalls(unsigned char* zsm, int stall, unsigned int* err_out)
{
    if (!stall) return false;
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
    return true;
}

// the results of a pair without tiles
__device__ __forceinline__ void zoom_none(long long p, float2* offsets, PairDiag* diag)
{
    offsets[p] = make_float2(NAN, NAN);
    if (diag) diag[p] = PairDiag{-1, -1, -1, -1, -1, -1, -1, -1, NAN, NAN, NAN, 0.0f};
}

// the results of pair p from the first maximum bv at cell bi of its zoomed surface
__device__ void zoom_result(long long p, float bv, int bi, int Z, int z, const CoarseOut* coarse,
                            const float* coarse_peak, const FineOut* fout, int margin, int refine_factor,
                            int refine_margin, int ref_compat, float2* offsets, PairDiag* diag)
{
    const CoarseOut co = coarse[p];
    const FineOut fo = fout[p];
    const int fp = bi / Z, fq = bi - fp * Z;
    const float zoom = (float)(refine_factor * z);
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
    if (diag)
        diag[p] = PairDiag{co.u, co.v, co.top, co.left, fo.u, fo.v, fp, fq, coarse_peak[p], fo.peak, bv, 0.0f};
}

// floats as ints in the same order, for a maximum by atomics
__device__ __forceinline__ int ordered(float v)
{
    const int i = __float_as_int(v);
    return i < 0 ? i ^ 0x7fffffff : i;
}
__device__ __forceinline__ float unordered(int i) { return __int_as_float(i < 0 ? i ^ 0x7fffffff : i); }

}  // namespace

// WARPS warps to a team, at most TEAMS teams to a CTA; `sets` sets of kCols columns to a batch
template <int WARPS, int TEAMS>
__global__ void __launch_bounds__(TEAMS * WARPS * 32, 1)
zoom_kernel(const float* gam, long long pair0, long long pairs, const long long* ref_off, ZoomGeomCols g,
            const float* u_g, const CoarseOut* coarse, const float* coarse_peak, const FineOut* fout, int margin,
            int refine_factor, int refine_margin, int ref_compat, float2* offsets, PairDiag* diag,
            unsigned int* err_out, int sets, int stall)
{
    extern __shared__ __align__(16) unsigned char zsm[];
    constexpr int kTeam = WARPS * 32, GROUPS = WARPS / kGroup, kTotal = 3 * WARPS;
    const int team = threadIdx.x / kTeam, tid = threadIdx.x - team * kTeam, teams = blockDim.x / kTeam;
    const int Cf = g.Cf, Z = g.Z, kp4 = g.kp4;
    float* U = reinterpret_cast<float*>(zsm);
    const ZoomTeamLayout at = zoom_team(g, WARPS, sets);
    float* G = reinterpret_cast<float*>(zsm + g.off_team) + team * at.floats;
    float* T = G + at.T;
    float* val = G + at.val;
    float* far = G + at.far;
    float* red = G + at.red;
    int* counts = reinterpret_cast<int*>(red) + kTotal;  // the kept columns; then each set's kept rows
    unsigned* cols = reinterpret_cast<unsigned*>(G + at.cols);
    unsigned* rows = reinterpret_cast<unsigned*>(G + at.rows);
    const int Jv = at.Jv;
    const int lane = tid & 31, warp = tid >> 5, rl = lane >> 2, cl = lane & 3;
    const int grp = warp / kGroup, wrow = (warp - grp * kGroup) * kRows;  // its share of the sampled columns
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

    if (zoom_stalls(zsm, stall, err_out)) return;
#pragma unroll 4
    for (int i = threadIdx.x; i < g.s * g.Jp * kp4; i += blockDim.x)
        reinterpret_cast<float4*>(U)[i] = __ldg(reinterpret_cast<const float4*>(u_g) + i);
    for (int i = tid; i < at.val; i += kTeam) G[i] = 0.0f;  // (G and T)
    __syncthreads();

    for (long long b = (long long)blockIdx.x * teams + team; b < pairs; b += (long long)gridDim.x * teams) {
        const long long p = pair0 + b;
        if (ref_off[p] < 0) {
            if (tid == 0) zoom_none(p, offsets, diag);
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
                        G[a * 4 * kp4 + q] = gv[k];
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
            red[warp] = g1;
            red[WARPS + warp] = g2;
        }
        team_sync<kTeam>(team);
        g1 = g2 = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            g1 += red[w];
            g2 += red[WARPS + w];
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
            for (int a = kWide * grp; a < Cf; a += kWide * GROUPS) {
                float v[kNR][kNC];
                const int ga[kNC] = {a + cl, a + cl + 4, a + cl + 8};
                dots(U, q, G, ga, kp4, v);
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
                if (cl == i && j0 + rl + 8 * i < g.J) val[grp * Jv + j0 + rl + 8 * i] = GROUPS == 1 ? sqrtf(nn[i]) : nn[i];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(kFull, best, o));
        if (lane == 0) red[2 * WARPS + warp] = best;
        team_sync<kTeam>(team);
        if constexpr (GROUPS > 1) {
            for (int j = tid; j < g.J; j += kTeam) {
                float n2 = 0.0f;
#pragma unroll
                for (int i = 0; i < GROUPS; ++i) n2 += val[i * Jv + j];
                val[j] = sqrtf(n2);
            }
            team_sync<kTeam>(team);
        }
#pragma unroll
        for (int w = 0; w < WARPS; ++w) best = fmaxf(best, red[2 * WARPS + w]);
        const float slack = 1e-4f * (gn + fabsf(c)) + 1e-6f;
        // (warp 0 writes the list, its length goes through the reduction slots)
        if (warp == 0) {
            const int n = kept_intervals(val, g, c + g.curv * gn + slack, best, true, cols);
            if (lane == 0) counts[0] = n;
        }
        team_sync<kTeam>(team);
        const int total = counts[0];

        float bv = -INFINITY;
        int bi = INT_MAX;
        // cells of rows pa (rows ra of U) and the columns s .. s + 11 of the nb in T: this thread's first
        // maximum, and the maximum of each row over its columns
        auto cells = [&](const int (&ra)[kNR], const int (&pa)[kNR], int c0, int nb, int s, float (&rm)[kNR]) {
            float v[kNR][kNC];
            const int rt[kNC] = {s + cl, s + cl + 4, s + cl + 8};
            dots(U, ra, T, rt, kp4, v);
            float most = -INFINITY;
#pragma unroll
            for (int i = 0; i < kNR; ++i) {
                float m = -INFINITY;
#pragma unroll
                for (int k = 0; k < kNC; ++k) m = rt[k] < nb ? fmaxf(m, v[i][k]) : m;
                rm[i] = fmaxf(rm[i], m);
                most = fmaxf(most, m);
            }
            // (one test for the block: most hold no new maximum)
            if (most >= bv)
#pragma unroll
                for (int k = 0; k < kNC; ++k)
                    if (rt[k] < nb)
#pragma unroll
                        for (int i = 0; i < kNR; ++i)
                            better(bv, bi, v[i][k], pa[i] * Z + (int)(cols[c0 + rt[k]] & 0xffffu));
        };
        // Batches of columns, whose work goes round the team's warps in blocks: of 12 columns by 24 rows of
        // T; of 24 sampled rows by the 36 columns of a set; a set's list of kept rows to a warp; and of 24
        // kept rows by 12 columns.
        for (int c0 = 0; c0 < total; c0 += kCols * sets) {
            const int nb = min(kCols * sets, total - c0), here = (nb + kCols - 1) / kCols;
            // the batch's columns of T, and the largest |column - c|^2 of each block's share
            for (int u = warp; u < (nb + kWide - 1) / kWide * at.nab; u += WARPS) {
                const int qb = u / at.nab, ab = u - qb * at.nab;
                int q[kNC], uq[kNC], a[kNR];
                float nn[kNC], v[kNR][kNC];
#pragma unroll
                for (int k = 0; k < kNC; ++k) {
                    q[k] = kWide * qb + cl + 4 * k;
                    uq[k] = (int)(cols[c0 + min(q[k], nb - 1)] >> 16);
                    nn[k] = 0.0f;
                }
#pragma unroll
                for (int i = 0; i < kNR; ++i) a[i] = min(kRows * ab + rl + 8 * i, Cf - 1);
                dots(G, a, U, uq, kp4, v);
#pragma unroll
                for (int i = 0; i < kNR; ++i)
                    if (kRows * ab + rl + 8 * i < Cf)
#pragma unroll
                        for (int k = 0; k < kNC; ++k) {
                            if (q[k] < nb) T[q[k] * 4 * kp4 + a[i]] = v[i][k];
                            const float d = v[i][k] - c;
                            nn[k] = fmaf(d, d, nn[k]);
                        }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1)
#pragma unroll
                    for (int k = 0; k < kNC; ++k) nn[k] += __shfl_xor_sync(kFull, nn[k], o);
                float most = fmaxf(nn[0], fmaxf(nn[1], nn[2]));
                most = fmaxf(most, __shfl_xor_sync(kFull, most, 1));
                most = fmaxf(most, __shfl_xor_sync(kFull, most, 2));
                if (lane == 0) far[u] = most;
            }
            team_sync<kTeam>(team);
            // every s-th row
            const int jb = (g.J + kRows - 1) / kRows;
            for (int u = warp; u < here * jb; u += WARPS) {
                const int set = u / jb, j0 = (u - set * jb) * kRows;
                int ra[kNR], pa[kNR];
                float rm[kNR];
#pragma unroll
                for (int i = 0; i < kNR; ++i) {
                    ra[i] = min(j0 + rl + 8 * i, g.J - 1);
                    pa[i] = g.s * ra[i];
                    rm[i] = -INFINITY;
                }
                for (int s = kCols * set; s < min(kCols * set + kCols, nb); s += kWide) cells(ra, pa, c0, nb, s, rm);
#pragma unroll
                for (int i = 0; i < kNR; ++i) {
                    rm[i] = fmaxf(rm[i], __shfl_xor_sync(kFull, rm[i], 1));
                    rm[i] = fmaxf(rm[i], __shfl_xor_sync(kFull, rm[i], 2));
                    if (cl == i && j0 + rl + 8 * i < g.J) val[set * Jv + j0 + rl + 8 * i] = rm[i];
                }
            }
            team_sync<kTeam>(team);
            // the rows between them that can hold more than the largest cell seen
            if (warp < here) {
                float seen = best;
                for (int set = 0; set < here; ++set)
                    for (int j = lane; j < g.J; j += 32) seen = fmaxf(seen, val[set * Jv + j]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) seen = fmaxf(seen, __shfl_xor_sync(kFull, seen, o));
                for (int set = warp; set < here; set += WARPS) {
                    float most = 0.0f;
                    for (int qb = kCols / kWide * set; qb < kCols / kWide * (set + 1) && kWide * qb < nb; ++qb) {
                        float sum = 0.0f;
                        for (int ab = 0; ab < at.nab; ++ab) sum += far[qb * at.nab + ab];
                        most = fmaxf(most, sum);
                    }
                    // (how far a column of the set can rise between two rows)
                    const int n = kept_intervals(val + set * Jv, g, g.curv * sqrtf(most) + slack, seen, false, rows + set * at.Zv);
                    if (lane == 0) counts[1 + set] = n;
                }
            }
            team_sync<kTeam>(team);
            int turn = warp;  // the warp's next block, counted over all sets
            for (int set = 0; set < here; ++set) {
                const int nr = counts[1 + set], wide = (min(kCols, nb - kCols * set) + kWide - 1) / kWide;
                const int units = (nr + kRows - 1) / kRows * wide;
                for (; turn < units; turn += WARPS) {
                    const int r0 = turn / wide * kRows;
                    int ra[kNR], pa[kNR];
                    float rm[kNR];
#pragma unroll
                    for (int i = 0; i < kNR; ++i) {
                        const unsigned e = rows[set * at.Zv + min(r0 + rl + 8 * i, nr - 1)];
                        ra[i] = (int)(e >> 16);
                        pa[i] = (int)(e & 0xffffu);
                        rm[i] = 0.0f;
                    }
                    cells(ra, pa, c0, nb, kCols * set + (turn - turn / wide * wide) * kWide, rm);
                }
                turn -= units;
            }
            team_sync<kTeam>(team);
        }
        team_argmax<kTeam>(bv, bi, red, team, tid);
        if (tid == 0)
            zoom_result(p, bv, bi, Z, g.z, coarse, coarse_peak, fout, margin, refine_factor, refine_margin, ref_compat, offsets,
                        diag);
    }
}

// One pair to a CTA of kWideWarps warps.  Each warp takes sets of 8 NR kept columns through all steps by
// itself - their columns of T, the sampled rows, its list of kept rows and those - with one barrier, before
// the list, so that every warp's largest cell bounds it.  The blocks are 8 NR columns by 4 NC rows, the
// longer side on the 4 lanes whose loads cost two wavefronts (lanes next to each other read 8 rows there:
// four); NC = 9 covers the 33 rows of the production surface at once, NC = 5 those of 17.  Every second sampled row of an
// even zoom is a row of T itself.  Few columns (a peak) go in sets of 8, so that more warps have some.
template <int NR, int NC>
__device__ __forceinline__ void wide_sets(const ZoomGeomCols& g, const float* U, const float* G, float* T, float* val,
                                          const unsigned* cols, unsigned* rows, int* seen_at, int total, float c, float slack,
                                          float& bv, int& bi)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rl = lane & 7, cl = lane >> 3;
    const int Cf = g.Cf, Z = g.Z, kp4 = g.kp4;
    const bool half = g.z == 2 * g.s;
    // the maxima of the rows over the set's columns, and this thread's first maximum: rows p of the surface
    auto row_maxima = [&](const float (&v)[NR][NC], const int (&p)[NC], const int (&col)[NR], float (&rm)[NC]) {
        float most = -INFINITY;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            rm[k] = v[0][k];
#pragma unroll
            for (int i = 1; i < NR; ++i) rm[k] = fmaxf(rm[k], v[i][k]);
            most = fmaxf(most, rm[k]);
        }
        // (one test for the block: most hold no new maximum)
        if (most >= bv)
#pragma unroll
            for (int k = 0; k < NC; ++k)
#pragma unroll
                for (int i = 0; i < NR; ++i) better(bv, bi, v[i][k], p[k] * Z + col[i]);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < NC; ++k) rm[k] = fmaxf(rm[k], __shfl_xor_sync(kFull, rm[k], o));
    };
    for (int first = 0; first < total; first += 8 * NR * kWideWarps) {
        const int c0 = first + 8 * NR * warp, nb = min(8 * NR, total - c0);
        int q[NR], uq[NR], col[NR];  // (lanes past the last column repeat it)
        float rise = 0.0f;           // of a column of the set between two rows
        if (nb > 0) {
            float nn[NR];
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                q[i] = min(rl + 8 * i, nb - 1);
                const unsigned e = cols[c0 + q[i]];
                uq[i] = (int)(e >> 16);
                col[i] = (int)(e & 0xffffu);
                nn[i] = 0.0f;
            }
            for (int a0 = 0; a0 < Cf; a0 += 4 * NC) {
                int a[NC];
                float v[NR][NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) a[k] = min(a0 + cl + 4 * k, Cf - 1);
                dots<NR, NC, true>(U, uq, G, a, kp4, v);
#pragma unroll
                for (int k = 0; k < NC; ++k)
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        const float d = v[i][k] - c;
                        if (a0 + cl + 4 * k < Cf) nn[i] = fmaf(d, d, nn[i]);
                        T[q[i] * 4 * kp4 + a[k]] = v[i][k];
                    }
                if (half) {
                    int p[NC];
                    float rm[NC];
#pragma unroll
                    for (int k = 0; k < NC; ++k) p[k] = a[k] * g.z;
                    row_maxima(v, p, col, rm);
#pragma unroll
                    for (int k = 0; k < NC; ++k)
                        if (rl == 0) val[2 * a[k]] = rm[k];
                }
            }
            float far = 0.0f;  // the largest |column - c|^2
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                nn[i] += __shfl_xor_sync(kFull, nn[i], 8);
                nn[i] += __shfl_xor_sync(kFull, nn[i], 16);
                far = fmaxf(far, nn[i]);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) far = fmaxf(far, __shfl_xor_sync(kFull, far, o));
            rise = g.curv * sqrtf(far) + slack;
            __syncwarp();
            // the sampled rows (but those of T)
            const int n = half ? Cf : g.J;
            for (int r0 = 0; r0 < n; r0 += 4 * NC) {
                int j[NC], p[NC];
                float v[NR][NC], rm[NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const int r = min(r0 + cl + 4 * k, n - 1);
                    j[k] = half ? 2 * r + 1 : r;
                    p[k] = g.s * j[k];
                }
                dots<NR, NC, true>(T, q, U, j, kp4, v);
                row_maxima(v, p, col, rm);
#pragma unroll
                for (int k = 0; k < NC; ++k)
                    if (rl == 0) val[j[k]] = rm[k];
            }
            __syncwarp();
            float seen = -INFINITY;
            for (int j = lane; j < g.J; j += 32) seen = fmaxf(seen, val[j]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) seen = fmaxf(seen, __shfl_xor_sync(kFull, seen, o));
            if (lane == 0) atomicMax(seen_at, ordered(seen));
        }
        __syncthreads();
        if (nb <= 0) continue;
        // the rows between them that can hold more than the largest cell that any warp has seen
        const int nr = kept_intervals(val, g, rise, unordered(*const_cast<volatile int*>(seen_at)), false, rows);
        constexpr int kRowsK = NC < 3 ? NC : 3;
        for (int r0 = 0; r0 < nr; r0 += 4 * kRowsK) {
            int ru[kRowsK], p[kRowsK];
            float v[NR][kRowsK];
#pragma unroll
            for (int k = 0; k < kRowsK; ++k) {
                const unsigned e = rows[min(r0 + cl + 4 * k, nr - 1)];
                ru[k] = (int)(e >> 16);
                p[k] = (int)(e & 0xffffu);
            }
            dots<NR, kRowsK>(T, q, U, ru, kp4, v);
            float most = -INFINITY;
#pragma unroll
            for (int k = 0; k < kRowsK; ++k)
#pragma unroll
                for (int i = 0; i < NR; ++i) most = fmaxf(most, v[i][k]);
            if (most >= bv)
#pragma unroll
                for (int k = 0; k < kRowsK; ++k)
#pragma unroll
                    for (int i = 0; i < NR; ++i) better(bv, bi, v[i][k], p[k] * Z + col[i]);
        }
        __syncwarp();
    }
}

template <int NC>
__global__ void __launch_bounds__(kWideWarps * 32, 1)
zoom_wide_kernel(const float* gam, long long pair0, const long long* ref_off, ZoomGeomCols g,
                 const float* u_g, const CoarseOut* coarse, const float* coarse_peak, const FineOut* fout, int margin,
                 int refine_factor, int refine_margin, int ref_compat, float2* offsets, PairDiag* diag,
                 unsigned int* err_out, int stall)
{
    extern __shared__ __align__(16) unsigned char zsm[];
    constexpr int kTeam = kWideWarps * 32, W = kWideWarps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rl = lane & 7, cl = lane >> 3;
    const int Cf = g.Cf, Z = g.Z, kp4 = g.kp4;
    const ZoomWideLayout at = zoom_wide(g);
    float* U = reinterpret_cast<float*>(zsm);
    float* G = reinterpret_cast<float*>(zsm + g.off_team);
    float* norm = G + at.norm;
    float* red = G + at.red;
    int* counts = reinterpret_cast<int*>(red) + 3 * W;
    unsigned* cols = reinterpret_cast<unsigned*>(G + at.cols);
    float* own = G + at.own + warp * at.warp;
    if (zoom_stalls(zsm, stall, err_out)) return;
    const long long b = blockIdx.x, p = pair0 + b;
    if (ref_off[p] < 0) {
        if (tid == 0) zoom_none(p, offsets, diag);
        return;
    }
    // (the surface's loads are under way while U is copied)
    constexpr int kLoads = 3;
    const float* src = gam + b * Cf * Cf;
    float gv[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) gv[k] = tid + k * kTeam < Cf * Cf ? __ldg(src + tid + k * kTeam) : 0.0f;
#pragma unroll 4
    for (int i = tid; i < g.s * g.Jp * kp4; i += kTeam)
        reinterpret_cast<float4*>(U)[i] = __ldg(reinterpret_cast<const float4*>(u_g) + i);
    // zero past Cf: what one of the two factors' rows holds there is multiplied by the other's
    for (int i = tid; i < Cf; i += kTeam)
        for (int k = Cf; k < 4 * kp4; ++k) G[i * 4 * kp4 + k] = 0.0f;
    if (lane < 24)
        for (int k = Cf; k < 4 * kp4; ++k) own[lane * 4 * kp4 + k] = 0.0f;
    float g1 = 0.0f, g2 = 0.0f;
    for (int i0 = tid; i0 < Cf * Cf; i0 += kLoads * kTeam) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const int i = i0 + k * kTeam, a = i / Cf;
            if (i >= Cf * Cf) break;
            const float v = i0 == tid ? gv[k] : __ldg(src + i);
            G[a * 4 * kp4 + i - a * Cf] = v;
            g1 += v;
            g2 = fmaf(v, v, g2);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g1 += __shfl_xor_sync(kFull, g1, o);
        g2 += __shfl_xor_sync(kFull, g2, o);
    }
    if (lane == 0) {
        red[warp] = g1;
        red[W + warp] = g2;
    }
    __syncthreads();
    g1 = g2 = 0.0f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        g1 += red[w];
        g2 += red[W + w];
    }
    const float c = g1 / (float)(Cf * Cf);
    const float gn = sqrtf(fmaxf(g2 - g1 * c, 0.0f) + 1e-5f * g2);
    // T at every s-th column, a block of eight to a warp: the largest entry, the norm of every column
    float best = -INFINITY;
    for (int j0 = 8 * warp; j0 < g.J; j0 += 8 * W) {
        const int q[1] = {min(j0 + rl, g.J - 1)};
        float nn = 0.0f;
        for (int a0 = 0; a0 < Cf; a0 += 4 * NC) {
            int a[NC];
            float v[1][NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) a[k] = min(a0 + cl + 4 * k, Cf - 1);
            dots<1, NC>(U, q, G, a, kp4, v);
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const float d = v[0][k] - c;
                if (a0 + cl + 4 * k < Cf) nn = fmaf(d, d, nn);
                best = fmaxf(best, v[0][k]);
            }
        }
        nn += __shfl_xor_sync(kFull, nn, 8);
        nn += __shfl_xor_sync(kFull, nn, 16);
        if (cl == 0) norm[q[0]] = sqrtf(nn);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(kFull, best, o));
    if (lane == 0) red[2 * W + warp] = best;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < W; ++w) best = fmaxf(best, red[2 * W + w]);
    const float slack = 1e-4f * (gn + fabsf(c)) + 1e-6f;
    if (warp == 0) {
        const int n = kept_intervals(norm, g, c + g.curv * gn + slack, best, true, cols);
        if (lane == 0) {
            counts[0] = n;
            counts[1] = ordered(best);
        }
    }
    __syncthreads();
    const int total = counts[0];
    float bv = -INFINITY;
    int bi = INT_MAX;
    float* T = own;
    float* val = own + 24 * 4 * kp4;
    unsigned* rows = reinterpret_cast<unsigned*>(val + at.Jv);
    if (total <= 8 * W)
        wide_sets<1, NC>(g, U, G, T, val, cols, rows, counts + 1, total, c, slack, bv, bi);
    else
        wide_sets<3, NC>(g, U, G, T, val, cols, rows, counts + 1, total, c, slack, bv, bi);
    team_argmax<kTeam>(bv, bi, red, 0, tid);
    if (tid == 0)
        zoom_result(p, bv, bi, Z, g.z, coarse, coarse_peak, fout, margin, refine_factor, refine_margin, ref_compat, offsets,
                    diag);
}

cudaError_t zoom_set_smem_limits()
{
    const int limit = 227 * 1024;
    cudaError_t e = cudaSuccess;
    for (auto* k : {zoom_wide_kernel<5>, zoom_wide_kernel<6>, zoom_wide_kernel<9>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    for (auto* k : {zoom_kernel<3, kZoomTeams>, zoom_kernel<9, 3>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
    return e;
}

cudaError_t launch_zoom_kernel(unsigned sms, cudaStream_t st, const float* gam, long long pair0, unsigned n,
                               const long long* ref_off, const ZoomGeomCols& g, const float* u,
                               const CoarseOut* coarse, const float* coarse_peak, const FineOut* fout, int margin,
                               int refine_factor, int refine_margin, int ref_compat, float2* offsets,
                               PairDiag* diag, unsigned int* err_out, int stall)
{
    const unsigned each = (n + sms - 1) / sms;
    const long room = 227L * 1024 - g.off_team;
    // as many teams to a CTA as keep every multiprocessor busy, and as many sets of columns to a batch as fit
    // beside each other, `most` at most
    auto launch = [&](auto* kernel, int warps, unsigned teams, int most) {
        int sets = std::max(1, std::min(most, (g.Z + kCols - 1) / kCols));
        while (sets > 1 && 4L * teams * zoom_team(g, warps, sets).floats > room) --sets;
        const unsigned blocks = std::min<unsigned>((n + teams - 1) / teams, sms);
        kernel<<<blocks, teams * warps * 32, g.off_team + 4 * teams * zoom_team(g, warps, sets).floats, st>>>(
            gam, pair0, n, ref_off, g, u, coarse, coarse_peak, fout, margin, refine_factor, refine_margin, ref_compat,
            offsets, diag, err_out, sets, stall);
    };
    auto fit = [&](int warps, int teams) { return (unsigned)std::min<long>(teams, room / (4L * zoom_team(g, warps, 1).floats)); };
    // One pair to a multiprocessor: the pair's chain of products is all that such a call waits for, and
    // twelve warps shorten it most (100 surfaces of 33 x 33 at z = 8, peaks / noise: 16 / 27 us, 18 / 41 with
    // a team of nine warps; at z = 16 17 / 43, 25 / 74; 17 x 17 samples at z = 8 12 / 16, 14 / 20).  Two or three:
    // teams of nine side by side (225 surfaces 21 / 57 us; the twelve warps would take the pairs one after the
    // other, 400 surfaces 37 / 63 against 25 / 70), but 17 x 17 samples have too few rows for three of them
    // (444 surfaces 16.3 us, 14.3 with teams of three).  More: teams of three, which wait for each other least,
    // and two sets of columns to a batch (noise 1,680 us against 1,747 with one, peaks the same).
    if (each == 1 && 4L * zoom_wide(g).floats <= room) {
        // (blocks of 20, 24 or 36 rows: those that reach past Cf least)
        auto past = [&](int nc) { return (g.Cf + 4 * nc - 1) / (4 * nc) * nc; };
        auto* kernel = past(9) <= std::min(past(5), past(6)) ? zoom_wide_kernel<9>
                       : past(6) <= past(5)                  ? zoom_wide_kernel<6>
                                                             : zoom_wide_kernel<5>;
        kernel<<<n, kWideWarps * 32, g.off_team + 4 * zoom_wide(g).floats, st>>>(
            gam, pair0, ref_off, g, u, coarse, coarse_peak, fout, margin, refine_factor, refine_margin, ref_compat,
            offsets, diag, err_out, stall);
    } else if (each <= fit(9, g.J > 48 ? 3 : 2)) {
        launch(zoom_kernel<9, 3>, 9, each, 64);
    } else {
        launch(zoom_kernel<3, kZoomTeams>, 3, std::min(fit(3, kZoomTeams), each), 2);
    }
    return cudaGetLastError();
}

}  // namespace ampcor_b200

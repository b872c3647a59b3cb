/*
 * tp_disparity.cuh - residual disparity of each tile from its pair
 * correlations (the consumer of correlate2D).
 *
 * The reference stops at the correlation tiles (src/TileProcessor.cuh:
 * 1176-1443) and leaves the disparity fit to its Java caller, which is not
 * part of it; this is the plain fit the library defines.  Pair p = (i, j) of a
 * tile correlates with its peak at rho * b_p, b_p = port_offsets[j] -
 * port_offsets[i] (pairs as src/TileProcessor.cuh:484-490) and rho the
 * residual disparity (true minus task disparity).  The tile's profile is
 *   S(k) = sum over its listed pairs in pair_mask of C_p(k * b_p),
 * k = -r..r, C_p sampled bilinearly in the centred (2r+1)^2 tile; a k whose
 * sample of any contributing pair leaves the tile is not used.  rho is the
 * sub-pixel maximum of S around its first integer argmax k* (double
 * precision):
 *   mode 0: parabola through S(k*-1), S(k*), S(k*+1);
 *   mode 1: least-squares parabola through the valid S(k*-2 .. k*+2);
 *   mode 2: centroid of S - min over k*-1 .. k*+1.
 * The sub-pixel offset is kept within [-1, 1]; a fit without a maximum gives
 * k*.  strength = the fitted peak value / number of pairs.
 *
 * A warp takes `win` consecutive entries (a power of two up to 32, by the
 * list's length: see list_window), finds the first entries of the tiles'
 * runs among them (entries of one tile adjacent in the list) and fits two
 * tiles at a time, one per half warp, lane k evaluating S(k - r).  Where each
 * lane samples each pair's tile does not depend on the tile, so it is worked
 * out once per block; the samples of a run are all in flight at once.  A warp
 * per entry, five of six of which only looked at two list entries, with the
 * samples one after another, took 0.219 ms for a 2592x1936 frame, this form
 * 0.060 (six blocks per SM; 0.065 at four).  Bound by the latency of a run:
 * list entries, samples, maximum, fit.
 */
#pragma once
#include "tp_common.cuh"

namespace tp {

/* sub-pixel step on s[t + 2] = S(k* + t), t = -2..2 (ok[]: usable) */
__device__ __forceinline__ void fit_peak(const double s[5], const bool ok[5], int mode, double *off_out,
                                         double *peak_out)
{
    double off = 0.0, pk = s[2];
    if (mode == 0) {
        if (ok[1] && ok[3]) {
            const double a = s[1], b = s[2], c = s[3];
            const double den = a - 2.0 * b + c;
            if (den < 0.0) {
                off = fmin(1.0, fmax(-1.0, 0.5 * (a - c) / den));
                pk = b - 0.25 * (a - c) * off;
            }
        }
    } else if (mode == 1) {
        /* normal equations of y = a + b t + c t^2 over the usable points */
        double m0 = 0, m1 = 0, m2 = 0, m3 = 0, m4 = 0, z0 = 0, z1 = 0, z2 = 0;
        int cnt = 0;
#pragma unroll
        for (int i = 0; i < 5; i++) {
            if (!ok[i]) continue;
            const double t = i - 2, t2 = t * t;
            m0 += 1.0; m1 += t; m2 += t2; m3 += t2 * t; m4 += t2 * t2;
            z0 += s[i]; z1 += t * s[i]; z2 += t2 * s[i];
            cnt++;
        }
        if (cnt >= 3) {
            /* Cramer's rule on [m0 m1 m2; m1 m2 m3; m2 m3 m4] */
            const double c00 = m2 * m4 - m3 * m3, c01 = m1 * m4 - m3 * m2, c02 = m1 * m3 - m2 * m2;
            const double det = m0 * c00 - m1 * c01 + m2 * c02;
            if (det != 0.0) {
                const double a = (z0 * c00 - m1 * (z1 * m4 - m3 * z2) + m2 * (z1 * m3 - m2 * z2)) / det;
                const double b = (m0 * (z1 * m4 - z2 * m3) - z0 * c01 + m2 * (m1 * z2 - z1 * m2)) / det;
                const double c = (m0 * (m2 * z2 - m3 * z1) - m1 * (m1 * z2 - m3 * z0) + z0 * c02) / det;
                if (c < 0.0) {
                    off = fmin(1.0, fmax(-1.0, -b / (2.0 * c)));
                    pk = a + b * off + c * off * off;
                }
            }
        }
    } else {
        if (ok[1] && ok[3]) {
            const double a = s[1], b = s[2], c = s[3];
            const double m = fmin(a, fmin(b, c));
            const double w = (a - m) + (b - m) + (c - m);
            if (w > 0.0) off = ((c - m) - (a - m)) / w;
        }
    }
    *off_out = off;
    *peak_out = pk;
}

/* Where lane k samples pair p's centred (2r+1)^2 tile: the offset of the
 * sample's corner (-1: outside the tile) and the bilinear fractions. */
struct FitSample {
    int off;
    float fx, fy;
};

__device__ __forceinline__ FitSample fit_sample_at(int r, float x, float y)
{
    const float fx0 = floorf(x), fy0 = floorf(y);
    const int ix = (int)fx0, iy = (int)fy0;
    FitSample s{-1, x - fx0, y - fy0};
    if (ix < -r || iy < -r || ix > r || iy > r) return s;
    if ((s.fx > 0.0f && ix + 1 > r) || (s.fy > 0.0f && iy + 1 > r)) return s;
    s.off = (iy + r) * (2 * r + 1) + ix + r;
    return s;
}

/* bilinear sample of tile c at s (s.off >= 0), n = 2r + 1 */
__device__ __forceinline__ float fit_sample(const float *__restrict__ c, const FitSample &s, int n)
{
    const float *p = c + s.off;
    float v = (1.0f - s.fx) * (1.0f - s.fy) * __ldg(p);
    if (s.fx > 0.0f) v = __fmaf_rn(s.fx * (1.0f - s.fy), __ldg(p + 1), v);
    if (s.fy > 0.0f) v = __fmaf_rn((1.0f - s.fx) * s.fy, __ldg(p + n), v);
    if (s.fx > 0.0f && s.fy > 0.0f) v = __fmaf_rn(s.fx * s.fy, __ldg(p + n + 1), v);
    return v;
}

__global__ void __launch_bounds__(256, 6) k_disparity_fit(int ntiles, const float *__restrict__ corrs,
                                                       size_t corr_stride, int r, long long num,
                                                       const int *__restrict__ idx,
                                                       const float *__restrict__ port_offsets, int pair_mask,
                                                       int mode, int win, float *__restrict__ disparity,
                                                       float *__restrict__ strength)
{
    __shared__ FitSample s_at[6][16];
    __shared__ int s_whole[6]; /* every sample of the pair is a grid point */
    const int n = 2 * r + 1; /* at most 15 */
    if (threadIdx.x < 96) {
        const int p = threadIdx.x >> 4, k = (threadIdx.x & 15) - r;
        const int i = c_pairs[p][0], j = c_pairs[p][1];
        const float bx = __ldg(&port_offsets[2 * j]) - __ldg(&port_offsets[2 * i]);
        const float by = __ldg(&port_offsets[2 * j + 1]) - __ldg(&port_offsets[2 * i + 1]);
        FitSample at = fit_sample_at(r, (float)k * bx, (float)k * by);
        if (k > r) at = FitSample{-1, 0.0f, 0.0f};
        s_at[p][threadIdx.x & 15] = at;
        const unsigned whole = __ballot_sync(0xffffffffu, at.fx == 0.0f && at.fy == 0.0f);
        if ((threadIdx.x & 15) == 0) s_whole[p] = ((whole >> (threadIdx.x & 16)) & 0xffffu) == 0xffffu;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, hl = lane & 15, half = lane >> 4;
    const unsigned hm = 0xffffu << (16 * half);
    const long long step = (long long)gridDim.x * (blockDim.x >> 5) * win;
    for (long long e0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * win; e0 < num; e0 += step) {
        /* the runs that start in this window */
        const long long my = e0 + lane;
        const int mytile = my < num ? __ldg(&idx[my]) >> 8 : -1;
        const int before = __shfl_up_sync(0xffffffffu, mytile, 1);
        bool first = lane < win && my < num && mytile >= 0 && mytile < ntiles;
        if (first) first = lane ? before != mytile : (my == 0 || (__ldg(&idx[my - 1]) >> 8) != mytile);
        unsigned starts = __ballot_sync(0xffffffffu, first);
        while (starts) {
            /* the first half warp takes the lowest start, the second the next */
            const unsigned rest = starts & (starts - 1);
            const unsigned mine = half ? rest : starts;
            starts = rest & (rest - 1);
            if (!mine) break; /* only the second half: the first one's run was the last */
            const long long e = e0 + __ffs(mine) - 1;
            const int tile = __ldg(&idx[e]) >> 8;
            /* the first 8 entries of the run in one load, lane j holding e + j */
            const int mycode = (hl < 8 && e + hl < num) ? __ldg(&idx[e + hl]) : -1;
            const unsigned same = __ballot_sync(hm, hl < 8 && e + hl < num && (mycode >> 8) == tile) >> (16 * half);
            const int m = __ffs(~same) - 1; /* run length within the first 8 */
            float v[8];
            bool valid = hl < n;
            int npairs = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int p = __shfl_sync(hm, mycode, j, 16) & 0xff;
                v[j] = 0.0f;
                if (j >= m || p > 5 || !((pair_mask >> p) & 1)) continue;
                npairs++;
                const FitSample at = s_at[p][hl];
                const float *c = corrs + (size_t)(e + j) * corr_stride;
                if (at.off < 0)
                    valid = false;
                else
                    v[j] = s_whole[p] ? __ldg(c + at.off) : fit_sample(c, at, n);
            }
            float S = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; j++) S += v[j];
            /* runs longer than 8 (repeated pairs) */
            for (long long e2 = e + 8; m == 8 && e2 < num; e2++) {
                const int code = __ldg(&idx[e2]);
                if ((code >> 8) != tile) break;
                const int p = code & 0xff;
                if (p > 5 || !((pair_mask >> p) & 1)) continue;
                npairs++;
                const FitSample at = s_at[p][hl];
                if (at.off < 0)
                    valid = false;
                else
                    S += fit_sample(corrs + (size_t)e2 * corr_stride, at, n);
            }
            if (!npairs) continue;
            /* first (lowest k) maximum over the usable lanes */
            float best = valid ? S : -INFINITY;
            int bk = valid ? hl : 64;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const float ob = __shfl_down_sync(hm, best, o, 16);
                const int ok = __shfl_down_sync(hm, bk, o, 16);
                if (ok < 64 && (bk == 64 || ob > best || (ob == best && ok < bk))) { best = ob; bk = ok; }
            }
            const int km = __shfl_sync(hm, bk, 0, 16);
            if (km == 64) continue; /* no usable k */
            double s5[5];
            bool ok5[5];
            const unsigned usable = __ballot_sync(hm, valid) >> (16 * half);
#pragma unroll
            for (int t = -2; t <= 2; t++) {
                const int src = km + t;
                const int srcc = src < 0 ? 0 : (src > 15 ? 15 : src);
                s5[t + 2] = (double)__shfl_sync(hm, S, srcc, 16);
                ok5[t + 2] = src >= 0 && src < n && ((usable >> srcc) & 1);
            }
            if (hl == 0) {
                double off, pk;
                fit_peak(s5, ok5, mode, &off, &pk);
                disparity[tile] = (float)((double)(km - r) + off);
                strength[tile] = (float)(pk / npairs);
            }
        }
        __syncwarp();
    }
}

} /* namespace tp */

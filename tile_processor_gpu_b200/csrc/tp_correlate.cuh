/*
 * tp_correlate.cuh - pairwise phase correlation (the drop-in for the
 * reference's correlate2D, src/TileProcessor.cuh:1176-1443, with its helpers
 * correlateAccumulateTiles :2829-2890, normalizeTileAmplitude :2915-2942 and
 * corrUnfoldTile :2950-3008).
 *
 * One 8-lane group per (tile, pair) entry of the index list.  Lane l holds
 * row l of the four accumulated quadrants, loaded 32 bytes at a time; the
 * color accumulation, the two LPFs and the amplitude normalisation are per
 * coefficient, on pairs of them; the pixel-domain transforms run on pairs of
 * quadrants, (q0, q2) and (q1, q3): the horizontal DCT-II / DST-II on the held
 * row, one 16-byte transpose per coefficient, the vertical pass on the held
 * column, and the unfold into the (2r+1)^2 output, stored straight from
 * registers.
 *
 * What bounds it is the latency of the three colours' loads at 16 warps per SM
 * (the sums of a row and one colour of both tiles are 96 registers) and the L1
 * (91% busy before, 57% now): 256-bit loads halve the passes over the loaded
 * lines, which 16-byte loads at a 32-byte lane stride touch twice.  A
 * 2592x1936 frame's 470,448 pairs went from 0.385 to 0.314 ms (3.61 to 4.42
 * TB/s of 1.39 GB).  Tried and slower: staging four tiles for one bulk store
 * (0.328), L2 prefetch of the next entry (+5%), 20 and 24 warps (spills).
 */
#pragma once
#include "tp_common.cuh"

namespace tp {

/* per-group buffer: 8 rows of 9 quadruples (one value per quadrant), so that
 * 16-byte accesses along rows and columns are conflict-free */
constexpr int kCorrBuf = 8 * 9 * 4 + 8;

/* 8 consecutive floats at p (16-byte aligned when al16) */
__device__ __forceinline__ void load_row8(const float *p, bool al16, float v[8])
{
    if (al16) {
        const float4 x = *reinterpret_cast<const float4 *>(p), y = *reinterpret_cast<const float4 *>(p + 4);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = p[k];
    }
}

/* The normalised, low-pass-filtered CLT-domain product of one (tile, pair)
 * entry without its last scale: row l of the four quadrants in acc, as pairs,
 * and the factor of each coefficient (1 / amplitude times the final LPF) in
 * scale.  a, b: the two cameras' CLT of the tile, colour c at a + c * cstride
 * (4 x 64 floats, row stride 8).  GLOBAL: in global memory, rows in one
 * 256-bit load each where both lie on 32-byte boundaries; else in shared
 * memory, half a row at a time (half the registers). */
template <bool GLOBAL>
__device__ __forceinline__ void corr_product(const float *a, const float *b, int cstride, int colors, float scale0,
                                             float scale1, float scale2, float fat_zero, int l, float2 acc[4][4],
                                             float2 scale[4])
{
    const uintptr_t al = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                         (uintptr_t)(cstride * sizeof(float));
    const bool al32 = GLOBAL && !(al & 31), al16 = !(al & 15);
    constexpr int KC = GLOBAL ? 4 : 2; /* pairs of a row at a time */
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[q][k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int color = 0; color < colors; color++) {
        const float2 s = dup2(color == 0 ? scale0 : color == 1 ? scale1 : scale2);
        const float *pa = a + color * cstride + l * 8, *pb = b + color * cstride + l * 8;
#pragma unroll
        for (int k0 = 0; k0 < 4; k0 += KC) {
            float A[4][2 * KC], B[4][2 * KC];
            if constexpr (GLOBAL) {
                if (al32) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        ld8_l1(pa + q * 64, A[q]);
                        ld8_l1(pb + q * 64, B[q]);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        load_row8(pa + q * 64, al16, A[q]);
                        load_row8(pb + q * 64, al16, B[q]);
                    }
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 x = *reinterpret_cast<const float4 *>(pa + q * 64 + 2 * k0);
                    const float4 y = *reinterpret_cast<const float4 *>(pb + q * 64 + 2 * k0);
                    A[q][0] = x.x; A[q][1] = x.y; A[q][2] = x.z; A[q][3] = x.w;
                    B[q][0] = y.x; B[q][1] = y.y; B[q][2] = y.z; B[q][3] = y.w;
                }
            }
#pragma unroll
            for (int kk = 0; kk < KC; kk++) {
                const int k = k0 + kk;
                float2 x[4], y[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    x[q] = make_float2(A[q][2 * kk], A[q][2 * kk + 1]);
                    y[q] = make_float2(B[q][2 * kk], B[q][2 * kk + 1]);
                }
                /* CLT-domain correlation of the two tiles */
                const float2 r0 = fma2(x[3], y[3], fma2(x[2], y[2], fma2(x[1], y[1], mul2(x[0], y[0]))));
                const float2 r1 = sub2(fma2(x[2], y[3], mul2(x[0], y[1])), fma2(x[3], y[2], mul2(x[1], y[0])));
                const float2 r2 = sub2(fma2(x[1], y[3], mul2(x[0], y[2])), fma2(x[3], y[1], mul2(x[2], y[0])));
                const float2 r3 = sub2(fma2(x[0], y[3], mul2(x[3], y[0])), fma2(x[2], y[1], mul2(x[1], y[2])));
                acc[0][k] = fma2(s, r0, acc[0][k]);
                acc[1][k] = fma2(s, r1, acc[1][k]);
                acc[2][k] = fma2(s, r2, acc[2][k]);
                acc[3][k] = fma2(s, r3, acc[3][k]);
            }
        }
        if (color == 1) { /* LPF after red and blue */
            float f[8];
            load_row8s(&d_lpf[4][l * 8], f);
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q][k] = mul2(acc[q][k], make_float2(f[2 * k], f[2 * k + 1]));
        }
    }
    /* amplitude normalisation with fat zero and the final LPF */
    float f[8];
    load_row8s(&d_lpf[5][l * 8], f);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float2 s2 = dup2(fat_zero * fat_zero);
#pragma unroll
        for (int q = 0; q < 4; q++) s2 = fma2(acc[q][k], acc[q][k], s2);
        scale[k] = mul2(make_float2(rsqrtf(s2.x), rsqrtf(s2.y)), make_float2(f[2 * k], f[2 * k + 1]));
    }
}

/* One (tile, pair) correlation on an 8-lane group (arguments as corr_product).
 * tb: kCorrBuf floats of this group, 16-byte aligned.  dst: (2r+1)^2 floats,
 * written element by element. */
template <bool GLOBAL>
__device__ __forceinline__ void corr_job(const float *a, const float *b, int cstride, int colors, float scale0,
                                         float scale1, float scale2, float fat_zero, int r, float *tb,
                                         float *__restrict__ dst, int l, unsigned gm)
{
    const int sz = 2 * r + 1;
    float2 x02[8], x13[8], y02[8], y13[8];
    {
        float2 acc[4][4], scale[4];
        corr_product<GLOBAL>(a, b, cstride, colors, scale0, scale1, scale2, fat_zero, l, acc, scale);
        /* the pairs (q0, q2) and (q1, q3), with the unfold's factor 1/4, the
         * alternating signs of the horizontal DST-II's input (q1, q3: along
         * the row) and of the vertical one's (q2, q3: down the column, so one
         * sign per lane) */
        const float sl = (l & 1) ? -0.25f : 0.25f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float sc = (k & 1) ? scale[k >> 1].y : scale[k >> 1].x;
            const float s0 = 0.25f * sc, s2 = sl * sc;
            const float q0 = (k & 1) ? acc[0][k >> 1].y : acc[0][k >> 1].x;
            const float q1 = (k & 1) ? acc[1][k >> 1].y : acc[1][k >> 1].x;
            const float q2 = (k & 1) ? acc[2][k >> 1].y : acc[2][k >> 1].x;
            const float q3 = (k & 1) ? acc[3][k >> 1].y : acc[3][k >> 1].x;
            x02[k] = make_float2(q0 * s0, q2 * s2);
            x13[k] = (k & 1) ? make_float2(-q1 * s0, -q3 * s2) : make_float2(q1 * s0, q3 * s2);
        }
    }
    /* pixel domain: horizontal DCT-II (q0, q2) / DST-II (q1, q3) on the held
     * row, transpose, vertical DCT-II (q0, q1) / DST-II (q2, q3) on the held
     * column.  Lane j reads column j of q0 and q2 and column j - 1 of q1 and q3
     * (zeros for j = 0), as the unfold adds them. */
    dct2_pair(x02, y02);
    dct2_pair(x13, y13);
    float4 *t4 = reinterpret_cast<float4 *>(tb);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        /* DST_{k-1} of q1 and q3 is output 8 - k */
        const float2 o = k ? y13[8 - k] : make_float2(0.0f, 0.0f);
        t4[l * 9 + k] = make_float4(y02[k].x, y02[k].y, o.x, o.y);
    }
    __syncwarp(gm);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float4 t = t4[k * 9 + l];
        x02[k] = make_float2(t.x, t.y);
        x13[k] = make_float2(t.z, t.w);
    }
    __syncwarp(gm); /* the transpose buffer free for the group's next job */
    dct2_pair(x02, y02);
    dct2_pair(x13, y13);
    /* unfold, lane j = columns r +- j: R[+-i][+-j] from q0[i][j], q1[i][j-1],
     * q2[i-1][j], q3[i-1][j-1]; row i of q0 and q1 is output i, row i - 1 of q2
     * and q3 output 8 - i */
    float2 S[8], D[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        S[k] = add2(y02[k], y13[k]);
        D[k] = sub2(y02[k], y13[k]);
    }
    if (l <= r) {
        const int j = l;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (i > r) break;
            const float se = S[i].x, de = D[i].x;
            const float so = i ? S[8 - i].y : 0.0f, od = i ? D[8 - i].y : 0.0f;
            /* where i or j is 0 the stores to one element carry the same value
             * but for the sign of a zero; the later one stays */
            float *up = dst + (r + i) * sz + r, *dn = dst + (r - i) * sz + r;
            up[j] = se + so;
            up[-j] = de + od;
            dn[j] = se - so;
            dn[-j] = de - od;
        }
    }
}

constexpr int kCorrThreads = 128;

/* SLOTS: entry n is pair n % 6 of task n / 6, whose CLT lies in the frame's workspace by task (FrameSlots) */
template <bool SLOTS>
__global__ void __launch_bounds__(kCorrThreads, 4) k_correlate2D(Geom g, float *const *clt, int colors,
                                                                 float scale0, float scale1, float scale2,
                                                                 float fat_zero, long long num_corr_tiles,
                                                                 const int *__restrict__ corr_indices,
                                                                 size_t corr_stride, int corr_radius,
                                                                 float *__restrict__ corrs,
                                                                 const tp_task *__restrict__ tasks,
                                                                 const float *slot_clt)
{
    __shared__ __align__(16) float tbuf[kCorrThreads / 8][kCorrBuf];
    const int l = threadIdx.x & 7;
    const int grp = threadIdx.x >> 3;
    const unsigned gm = group_mask();
    const long long groups_total = (long long)gridDim.x * (blockDim.x >> 3);
    const int ntiles = g.TX * g.TY;
    /* a programmatic dependent of the forward transform; only once that is complete
     * the frame's textures, which read its CLT and lists too, may fill the SM
     * slots this grid frees */
    if (SLOTS) {
        grid_dependency_wait();
        grid_dependents_launch();
    }
    for (long long n = (long long)blockIdx.x * (blockDim.x >> 3) + grp; n < num_corr_tiles; n += groups_total) {
        const float *ta, *tb2;
        if (SLOTS) {
            const int slot = (int)(n / 6), pair = (int)n - 6 * slot;
            const int task = __ldg(&tasks[slot].task), txy = __ldg(&tasks[slot].txy);
            const int tx = txy & 0xffff, ty = txy >> 16;
            if (!((task >> (TP_TASK_CORR_BITS + pair)) & 1) || tx >= g.TX || ty < 0 || ty >= g.TY) continue;
            ta = slot_clt + (size_t)slot * (4 * 768) + c_pairs[pair][0] * 768;
            tb2 = slot_clt + (size_t)slot * (4 * 768) + c_pairs[pair][1] * 768;
        } else {
            const int code = corr_indices[n];
            const int tile = code >> 8, pair = code & 0xff;
            if (pair >= 6 || tile < 0 || tile >= ntiles) continue;
            ta = clt[c_pairs[pair][0]] + (size_t)tile * 768;
            tb2 = clt[c_pairs[pair][1]] + (size_t)tile * 768;
        }
        corr_job<true>(ta, tb2, 256, colors, scale0, scale1, scale2, fat_zero, corr_radius, tbuf[grp],
                       corrs + (size_t)n * corr_stride, l, gm);
    }
}

} /* namespace tp */

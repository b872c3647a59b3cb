/*
 * tp_texture.cuh - texture tiles (the drop-in for the reference's
 * textures_accumulate, src/TileProcessor.cuh:2207-2579, with imclt8threads
 * :3847-4017, debayer_shot / debayer :4019-4199 and tile_combine_rgba
 * :4202-4665).
 *
 * One 128-thread block per listed tile (mono: up to four tiles at a time),
 * grid-stride.
 * The CLT is read straight from global memory by the inverse transform; the
 * next tile's CLT and the RGBA rows it will update are prefetched into L2 while
 * the block works on the current tile.  Per (camera, colour) job one 8-lane
 * group, working only with __syncwarp on its
 * own buffers:
 *   1. low-pass filter and invert the CLT tile (horizontal DCT-IV/DST-IV on
 *      the held rows, transpose, vertical pass on the held column) and unfold
 *      it into the un-windowed tile T (colour) or the windowed tile M (mono);
 *   2. debayer T with the 3x3 stencil (walked down each column), apply the
 *      shot-noise square root and re-window into D (a lane owns two columns).
 * After one block barrier every thread fuses the four cameras at its pixel
 * pairs (stage 3; the plain windowed tile is T times the squared window) and
 * writes them out itself (stage 4): as non-overlapping 16x16 tiles and/or
 * faded by the neighbour mask and added into the overlapped RGBA image.
 *
 * The kernel is bound by issue slots and by the latency of each tile's chain of
 * steps (DRAM 16-27%), so all of it runs on packed pairs of FP32 values
 * (add2 / mul2 / fma2): two quadrants per pair in the transforms, two rows of
 * a column per pair from the unfold on.  The RGBA-only colour form takes 4776
 * warp instructions a tile (7238 in scalar form); the four passes of a
 * 2592x1936 frame with their list and clear went from 0.787 to 0.607 ms.
 * Seven blocks of four warps share an SM; three-warp blocks (no idle warp
 * in the transforms, but two turns of the fusion for one warp) took 0.671.
 * Tiles in shared memory hold pairs of rows: pair (rp, c) = rows 2 rp and 2 rp + 1 of column c at float2 16 rp + c,
 * so a warp of the fusion reads two row pairs of 16 columns in 64-bit loads
 * without a bank conflict and its RGBA accesses stay whole 64-byte rows.
 */
#pragma once
#include "tp_common.cuh"
#include "tp_correlate.cuh"

namespace tp {

struct TextureParams {
    int colors;
    float min_shot, scale_shot, diff_sigma;
    float w0, w1, w2;
    int dust_remove, keep_weights;
};

/* floats per job tile (16 x 16), padded: 272 % 32 == 16 puts the two groups of
 * a half-warp, whose 64-bit accesses cover 64 bytes each, on distinct banks */
constexpr int kJob = 272;
/* floats per group of transpose buffer: 8 rows of 9 quadruples, one per
 * quadrant (16-byte accesses along rows and columns are conflict-free);
 * 304 % 32 == 16 where job tiles overlay it */
constexpr int kXb = 304;
/* float2 index of the pair (rows 2 rp, 2 rp + 1) of column c in a job tile */
#define JT2(rp, c) ((rp) * 16 + (c))

/* Per-pixel factors of the unfold, [16][17]:
 *   tfac[r][c] = (0.25 / w[c]) / w[r]     un-windowed tile T = d * tfac
 *   mfac[r][c] = (0.5 w[r]) (0.5 w[c])    windowed tile M = mfac * d
 * with w the half-sine window, as read-only tables in global memory for the
 * tensor-core inverse stage's epilogue (values bit-identical to the float
 * expressions, generated by gen_tables.py); and the squared window at each
 * of the 256 pixels with its reciprocal for the camera fusion. */
constexpr int kFac = 16 * 17;
__device__ float d_tex_tfac[kFac] = TP_TEX_TFAC_INIT;
__device__ float d_tex_mfac[kFac] = TP_TEX_MFAC_INIT;
__device__ float d_tex_wnd2[256] = TP_TEX_WND2_INIT;
__device__ float d_tex_wi[256] = TP_TEX_WI_INIT;

/* Lane l's rows of a job's CLT tile: row l of quadrants 0 and 1, row 7 - l of 2
 * and 3 (see imclt_pairs); one 256-bit load each from global memory where the
 * tile lies on a 32-byte boundary, else 16-byte or scalar loads (GLOBAL false:
 * shared memory) */
template <bool GLOBAL>
__device__ __forceinline__ void load_clt_rows(const float *src, float raw[4][8], int l)
{
    if (GLOBAL && !(reinterpret_cast<uintptr_t>(src) & 31)) {
#pragma unroll
        for (int q = 0; q < 4; q++) ld8_global(src + q * 64 + (q < 2 ? l : 7 - l) * 8, raw[q]);
    } else {
        const bool al16 = !(reinterpret_cast<uintptr_t>(src) & 15);
#pragma unroll
        for (int q = 0; q < 4; q++) load_row8(src + q * 64 + (q < 2 ? l : 7 - l) * 8, al16, raw[q]);
    }
}

/* The four quadrants of one CLT tile to the pixel domain on an 8-lane group
 * (imclt8threads, :3847-4017).  Lane l holds coefficient row l of quadrants 0
 * and 1 and row 7 - l of 2 and 3 (load_clt_rows), times the low-pass filter
 * (NULL: none); the horizontal pass runs on the pairs (q0, q2) (DCT-IV) and
 * (q1, q3) (DST-IV), one 16-byte transpose per coefficient moves both pairs,
 * and the vertical pass runs on the same pairs, whose second halves (DST-IV)
 * arrive in the reverse row order the sine transform wants.  Lane l ends with
 * pixel-domain column l, a02[u] = (q0, q2), a13[u] = (q1, q3), except for the
 * signs dct4_pair leaves out: a02[u].y and a13[u].y are negated for odd u, and
 * a13 is negated as a whole for odd l. */
__device__ __forceinline__ void imclt_pairs(const float raw[4][8], const float *lpf, float4 *tb, float2 a02[8],
                                            float2 a13[8], int l, unsigned gm)
{
    float2 x[8], y02[8], y13[8];
    float f[8], g[8]; /* rows l and 7 - l of the low-pass filter */
    if (lpf) {
        load_row8(lpf + l * 8, true, f);
        load_row8(lpf + (7 - l) * 8, true, g);
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) f[k] = g[k] = 1.0f;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = make_float2(raw[0][k] * f[k], raw[2][k] * g[k]);
    dct4_pair(x, y02);
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = make_float2(raw[1][7 - k] * f[7 - k], raw[3][7 - k] * g[7 - k]);
    dct4_pair(x, y13);
#pragma unroll
    for (int k = 0; k < 8; k++) tb[l * 9 + k] = make_float4(y02[k].x, y02[k].y, y13[k].x, y13[k].y);
    __syncwarp(gm);
    float2 z[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const float4 t = tb[r * 9 + l];
        x[r] = make_float2(t.x, t.y);
        z[r] = make_float2(t.z, t.w);
    }
    dct4_pair(x, a02);
    dct4_pair(z, a13);
}

/* output column h (0, 1) of a lane: the two window columns that fold onto l */
__device__ __forceinline__ int unfold_col(int l, int h) { return h ? ((l < 4) ? l + 12 : l - 4) : 11 - l; }

/* Unfold of output column c of lane l into row pairs t[8], from the pairs of
 * imclt_pairs: the quadrant signs of idct_signs (:399-420) are a sign pair
 * per column (columns 0-3: (+,+); 4-11: (-,+); 12-15: (-,-) on the (even,
 * odd) quadrants) and compile-time signs per row; cf, the column's window
 * factor, rides on the column's signs, as do the signs imclt_pairs left out;
 * kr[r] is the row's factor (UNIT: 1 for every row). */
template <bool UNIT = false>
__device__ __forceinline__ void unfold_column(const float2 a02[8], const float2 a13[8], int l, int c, float cf,
                                              const float (&kr)[16], float2 t[8])
{
    const int cq = c >> 2;
    const float s0 = (cq == 0) ? cf : -cf, s1 = ((cq == 3) != ((l & 1) != 0)) ? -cf : cf;
    const float2 s0e = dup2(s0), s0o = make_float2(s0, -s0), s1e = dup2(s1), s1o = make_float2(s1, -s1);
    float2 e[8]; /* the even and odd vertical quadrants' sums */
#pragma unroll
    for (int u = 0; u < 8; u++) e[u] = fma2((u & 1) ? s0o : s0e, a02[u], mul2((u & 1) ? s1o : s1e, a13[u]));
#pragma unroll
    for (int rp = 0; rp < 8; rp++) {
        float d[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = 2 * rp + i, rq = r >> 2;
            const int u = (r < 4) ? r + 4 : (r < 12) ? 11 - r : r - 12;
            /* vertical signs: rows 0-3 (+,+); 4-11 (-,+); 12-15 (-,-) */
            d[i] = ((rq != 0) ? -e[u].x : e[u].x) + ((rq == 3) ? -e[u].y : e[u].y);
        }
        t[rp] = make_float2(d[0], d[1]);
        if (!UNIT) t[rp] = mul2(t[rp], make_float2(kr[2 * rp], kr[2 * rp + 1]));
    }
}

/* Inverse CLT of one job (raw: load_clt_rows), unfolded into the job tile `out` (row pairs): the
 * un-windowed tile T = d / (4 sin r sin c) (the windowed one with the squared
 * window removed, formed directly from the signed sum d) or, MONO, the
 * windowed M = (w_r / 2) (w_c / 2) d.  t: the lane's two columns, for the
 * debayer.  out may be the memory of tb, or the one raw was loaded from. */
template <bool MONO>
__device__ __forceinline__ void imclt_unfold_job(const float raw[4][8], const float *lpf, float *tb, float *out,
                                                 float2 t[2][8], int l, unsigned gm)
{
    constexpr float kHwin[16] = TP_HWIN_INIT;
    constexpr float kRow[16] = {
        MONO ? 0.5f * kHwin[0] : 1.0f / kHwin[0],   MONO ? 0.5f * kHwin[1] : 1.0f / kHwin[1],
        MONO ? 0.5f * kHwin[2] : 1.0f / kHwin[2],   MONO ? 0.5f * kHwin[3] : 1.0f / kHwin[3],
        MONO ? 0.5f * kHwin[4] : 1.0f / kHwin[4],   MONO ? 0.5f * kHwin[5] : 1.0f / kHwin[5],
        MONO ? 0.5f * kHwin[6] : 1.0f / kHwin[6],   MONO ? 0.5f * kHwin[7] : 1.0f / kHwin[7],
        MONO ? 0.5f * kHwin[8] : 1.0f / kHwin[8],   MONO ? 0.5f * kHwin[9] : 1.0f / kHwin[9],
        MONO ? 0.5f * kHwin[10] : 1.0f / kHwin[10], MONO ? 0.5f * kHwin[11] : 1.0f / kHwin[11],
        MONO ? 0.5f * kHwin[12] : 1.0f / kHwin[12], MONO ? 0.5f * kHwin[13] : 1.0f / kHwin[13],
        MONO ? 0.5f * kHwin[14] : 1.0f / kHwin[14], MONO ? 0.5f * kHwin[15] : 1.0f / kHwin[15]};
    float2 a02[8], a13[8]; /* pixel-domain column l of the quadrants */
    imclt_pairs(raw, lpf, reinterpret_cast<float4 *>(tb), a02, a13, l, gm);
    __syncwarp(gm);
    float2 *o2 = reinterpret_cast<float2 *>(out);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = unfold_col(l, h);
        const float wc = __ldg(&d_hwin[c]);
        unfold_column(a02, a13, l, c, MONO ? 0.5f * wc : 0.25f / wc, kRow, t[h]);
#pragma unroll
        for (int rp = 0; rp < 8; rp++) o2[JT2(rp, c)] = t[h][rp];
    }
}

/* 1 / sqrt(x) from the hardware's reciprocal square root (PTX
 * rsqrt.approx.ftz; x must be a normal float or zero) */
__device__ __forceinline__ float rsqrt_hw(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* 1 / x from the hardware's reciprocal (PTX rcp.approx.ftz, within one ulp
 * of the correctly rounded value for normal x) */
__device__ __forceinline__ float rcp_hw(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* 3x3 debayer of the un-windowed tile T (interior 14x14; border copied),
 * shot-noise square root, squared window re-applied: T -> D
 * (debayer_shot / debayer, :4019-4199).  Lane l owns the two columns it
 * unfolded (in t), as row pairs; the neighbouring columns come from the job
 * tile.  The stencil's horizontal sum t[r][c-1] + t[r][c+1] is formed once
 * per row and shared by the three rows that use it; red/blue (rb_mode) and
 * green take one branch-free form (the diagonal term's weight is 0 for
 * green), so the groups of a warp, which hold different colours, do not
 * diverge; the border columns (copied unchanged) take the same form with
 * stencil weights 0, 0 and 1.
 * WINDOWED = false stores D without the shot scale and the window factors
 * (the camera fusion of the RGBA-only path measures distances in D wi sqrt(w)
 * scale_shot, where the squared window cancels against wi = 1 / wnd2: it
 * takes scale_shot with its colour factors instead).  SHOT: scale_shot > 0,
 * the shot-noise step applies. */
template <bool WINDOWED, bool SHOT>
__device__ __forceinline__ void debayer_tile(const float2 t[2][8], const float *tile, float *d, int rb_mode,
                                             float min_shot, float scale_shot, int l, unsigned gm)
{
    /* the window as compile-time constants (the values of c_hwin) */
    constexpr float kHwin[16] = TP_HWIN_INIT;
    const float2 *t2 = reinterpret_cast<const float2 *>(tile);
    float2 *d2 = reinterpret_cast<float2 *>(d);
    __syncwarp(gm);
    const float kdiag = rb_mode ? 0.0625f : 0.0f, kcenter = rb_mode ? 0.25f : 0.5f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = unfold_col(l, h);
        const bool cborder = h && ((c == 0) || (c == 15)); /* columns 4..11 for h = 0 */
        const int cm = cborder ? c : c - 1, cp = cborder ? c : c + 1;
        /* per-lane stencil weights: diagonal, orthogonal, centre */
        const float2 kd = dup2(cborder ? 0.0f : kdiag), ko = dup2(cborder ? 0.0f : 0.125f);
        const float2 kc = dup2(cborder ? 1.0f : kcenter);
        const float hcc = __ldg(&d_hwin[c]);
        const float swx = (SHOT ? scale_shot : 1.0f) * (hcc * hcc);
        float2 hp = make_float2(0.0f, 0.0f), hs = add2(t2[JT2(0, cm)], t2[JT2(0, cp)]);
#pragma unroll
        for (int rp = 0; rp < 8; rp++) {
            float2 hn = make_float2(0.0f, 0.0f);
            if (rp < 7) hn = add2(t2[JT2(rp + 1, cm)], t2[JT2(rp + 1, cp)]);
            const float up = rp > 0 ? t[h][rp - 1].y : 0.0f, dn = rp < 7 ? t[h][rp + 1].x : 0.0f;
            const float2 me = t[h][rp];
            const float2 orth = add2(make_float2(up + me.y, me.x + dn), hs);
            const float2 diag = make_float2(hp.y + hs.y, hs.x + hn.x);
            float2 v = fma2(kd, diag, fma2(ko, orth, mul2(kc, me)));
            if (rp == 0) v.x = me.x;
            if (rp == 7) v.y = me.y;
            hp = hs;
            hs = hn;
            /* shot-noise square root above min_shot, v / sqrt(min_shot) at or
             * below it: both are v * rsqrt(max(v, min_shot)) (min_shot is a
             * normal float > 0 whenever the transform applies), from the
             * hardware reciprocal square root (within 3e-7 of sqrtf) */
            if (SHOT) v = mul2(v, make_float2(rsqrt_hw(fmaxf(v.x, min_shot)), rsqrt_hw(fmaxf(v.y, min_shot))));
            if (WINDOWED)
                v = mul2(v, mul2(dup2(swx), make_float2(kHwin[2 * rp] * kHwin[2 * rp],
                                                        kHwin[2 * rp + 1] * kHwin[2 * rp + 1])));
            d2[JT2(rp, c)] = v;
        }
    }
    __syncwarp(gm);
}

/* debayer_tile with the shot-noise step compiled in (scale_shot > 0) or out:
 * one switch per job, outside the unrolled stencil */
template <bool WINDOWED>
__device__ __forceinline__ void debayer_job(const float2 t[2][8], const float *tile, float *d, int rb_mode,
                                            float min_shot, float scale_shot, int l, unsigned gm)
{
    if (scale_shot > 0.0f)
        debayer_tile<WINDOWED, true>(t, tile, d, rb_mode, min_shot, scale_shot, l, gm);
    else
        debayer_tile<WINDOWED, false>(t, tile, d, rb_mode, min_shot, scale_shot, l, gm);
}

/* log2(e): e^x = 2^(x log2 e) */
constexpr float kLog2e = 1.4426950408889634f;

/* 2^x from the hardware's base-2 exponential (PTX ex2.approx.ftz; results
 * below the smallest normal float flush to zero) */
__device__ __forceinline__ float exp2_hw(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* a >= b as 1.0 / 0.0, on both halves of pairs */
__device__ __forceinline__ float2 ge2(float2 a, float2 b)
{
    float2 r;
    asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(r.x) : "f"(a.x), "f"(b.x));
    asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(r.y) : "f"(a.y), "f"(b.y));
    return r;
}

/* exp2 plus the 1e-4 weight floor, added in double and rounded once to float
 * (see combine_pair) */
__device__ __forceinline__ float weight_hw(float x) { return __double2float_rn((double)exp2_hw(x) + 1e-4); }

/* The best two of four weights (first of equals; a NaN is never the greater
 * one) by comparison: a mask of two cameras. */
__device__ __forceinline__ int best_two_of(float w0, float w1, float w2, float w3)
{
    const float w[4] = {w0, w1, w2, w3};
    int b1 = 0;
    float p1 = w0;
#pragma unroll
    for (int cam = 1; cam < 4; cam++)
        if (w[cam] > p1) { b1 = cam; p1 = w[cam]; }
    int b2 = b1 == 0 ? 1 : 0;
    float p2 = b1 == 0 ? w1 : w0;
#pragma unroll
    for (int cam = 1; cam < 4; cam++)
        if (cam > b2 && cam != b1 && w[cam] > p2) { b2 = cam; p2 = w[cam]; }
    return 1 << b1 | 1 << b2;
}

/* combine_pair's average of the best two cameras by selection, from the values
 * in its scaled space: only the chosen cameras' count.  For the rare pair with
 * an infinite or NaN value, and a call: inlined, its registers spill the
 * ordinary pairs' (RGBA image of 2592x1936 0.699 ms, 0.615 this way, 0.613
 * without the test for such pairs). */
template <int COLORS>
struct CameraValues {
    float2 d[4][COLORS];
};
template <int COLORS>
struct CameraAverage {
    float2 a[COLORS];
};
template <int COLORS>
__device__ __noinline__ CameraAverage<COLORS> best_two(CameraValues<COLORS> in, const float *npd2r)
{
    CameraAverage<COLORS> r;
    const auto &D = in.d;
    float2 w[4] = {};
    int k = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = i + 1; j < 4; j++) {
            float2 d = dup2(0.0f);
#pragma unroll
            for (int col = 0; col < COLORS; col++) {
                const float2 dc = sub2(D[i][col], D[j][col]);
                d = fma2(dc, dc, d);
            }
            d = mul2(d, dup2(npd2r[k++]));
            const float2 x = make_float2(weight_hw(d.x), weight_hw(d.y));
            w[i] = add2(w[i], x);
            w[j] = add2(w[j], x);
        }
    const int mx = best_two_of(w[0].x, w[1].x, w[2].x, w[3].x), my = best_two_of(w[0].y, w[1].y, w[2].y, w[3].y);
    float2 sum = dup2(0.0f);
#pragma unroll
    for (int cam = 0; cam < 4; cam++) {
        w[cam] = make_float2(mx >> cam & 1 ? w[cam].x : 0.0f, my >> cam & 1 ? w[cam].y : 0.0f);
        sum = add2(sum, w[cam]);
    }
    const float2 inv = make_float2(rcp_hw(sum.x), rcp_hw(sum.y));
#pragma unroll
    for (int col = 0; col < COLORS; col++) {
        float2 a = dup2(0.0f);
#pragma unroll
        for (int cam = 0; cam < 4; cam++)
            a = fma2(mul2(w[cam], inv),
                     make_float2(mx >> cam & 1 ? D[cam][col].x : 0.0f, my >> cam & 1 ? D[cam][col].y : 0.0f), a);
        r.a[col] = a;
    }
    return r;
}

/* Fuse the four cameras at a pair of pixels, rows 2 rp and 2 rp + 1 of one
 * column (tile_combine_rgba, two pixels).
 * sd: debayered tiles D; sm: the plain (not debayered) tiles, scaled by
 * m_scale (the plain tile is the un-windowed one times the squared window);
 * both [job = cam * colors + color] with the given strides in float2, pair
 * index e.
 * chw: the colour weights; chws: their square roots, times scale_shot when
 * the D tiles come without the window and the shot scale (D_WINDOWED false;
 * wi is then not applied to them).  npd2r (the six pairs'
 * -1 / (2 sigma^2 |offset|^2)) and nksigma (-1 / (2 sigma^2)) come multiplied
 * by log2(e): each weight exp(-k d) is evaluated as 2^(-(k log2 e) d).
 * o: colours, alpha, 4 port weights and (keep_weights) colors + 1 rms.
 * The colour distances sum_col chw[col] ((X[col] - Y[col]) wi)^2 are formed
 * as sum_col (X'[col] - Y'[col])^2 in the scaled space X' = X wi sqrt(chw),
 * the same quantity with fewer operations per camera pair. */
template <int COLORS, bool D_WINDOWED = true>
__device__ __forceinline__ void combine_pair(const float2 *sd, int sd_stride, const float2 *sm, int sm_stride,
                                             float2 m_scale, int e, const float *npd2r, float nksigma,
                                             const float *chw, const float *chws, float2 wnd2, float2 wi,
                                             int dust_remove, int keep_weights, float2 *o)
{
    float2 D[4][COLORS];
#pragma unroll
    for (int cam = 0; cam < 4; cam++)
#pragma unroll
        for (int col = 0; col < COLORS; col++) D[cam][col] = sd[(cam * COLORS + col) * sd_stride + e];
    if (keep_weights) {
        float2 sw = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int col = 0; col < COLORS; col++) {
            /* variance of the four cameras, two-pass (the one-pass form of
             * the reference loses digits where the cameras agree) */
            const float2 mean = mul2(add2(add2(D[0][col], D[1][col]), add2(D[2][col], D[3][col])), dup2(0.25f));
            float2 ss = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int cam = 0; cam < 4; cam++) {
                const float2 dv = sub2(D[cam][col], mean);
                ss = fma2(dv, dv, ss);
            }
            const float2 mse = mul2(ss, dup2(0.25f));
            o[COLORS + 5 + col] = make_float2(sqrtf(mse.x), sqrtf(mse.y));
            sw = fma2(dup2(chw[col]), mse, sw);
        }
        o[COLORS + 5 + COLORS] = make_float2(sqrtf(sw.x), sqrtf(sw.y));
    }
    /* D in the scaled space */
#pragma unroll
    for (int col = 0; col < COLORS; col++) {
        const float2 sc = D_WINDOWED ? mul2(wi, dup2(chws[col])) : dup2(chws[col]);
#pragma unroll
        for (int cam = 0; cam < 4; cam++) D[cam][col] = mul2(D[cam][col], sc);
    }
    /* wi = 1 / wnd2 correctly rounded (the reference forms it in double).
     * A weight is exp(...) plus the 1e-4 floor added in double and rounded
     * once to float, as the reference's double floor constant makes it: the
     * floor sum decides the best and worst cameras where every exponential
     * is tiny (high-contrast or high-dynamic-range tiles), and a float sum
     * with 1e-4f can land one ulp lower and break such ties the other way
     * (splitting the floor into two floats still rounds 1 in 2e6 tiny sums
     * differently).  The exponential is the hardware's base-2 one with the
     * log2(e) factor folded into npd2r and nksigma: its relative error (about
     * 2^-22) is under what float32 inputs already move a weight by, and a
     * flushed subnormal weight is lost in the 1e-4 floor. */
    float2 pw[4];
    {
        int k = 0;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = i + 1; j < 4; j++) {
                float2 d;
#pragma unroll
                for (int col = 0; col < COLORS; col++) {
                    const float2 dc = sub2(D[i][col], D[j][col]);
                    d = col ? fma2(dc, dc, d) : mul2(dc, dc);
                }
                d = mul2(d, dup2(npd2r[k]));
                const float2 x = make_float2(weight_hw(d.x), weight_hw(d.y));
                pw[i] = (i == 0 && j == 1) ? x : add2(pw[i], x);
                pw[j] = (i == 0) ? x : add2(pw[j], x);
                k++;
            }
    }
    /* the average of the best two cameras (first of equals) in proportion to
     * their weights.  Camera i beats a later camera j when w_i >= w_j; the two
     * best are those that beat at least two of the others, whichever of them
     * is first.  Six comparisons as 1.0 / 0.0 and a saturated sum of each
     * camera's wins (1 where there are two or three) choose them without a
     * branch or a select */
    {
        const float2 c01 = ge2(pw[0], pw[1]), c02 = ge2(pw[0], pw[2]), c03 = ge2(pw[0], pw[3]);
        const float2 c12 = ge2(pw[1], pw[2]), c13 = ge2(pw[1], pw[3]), c23 = ge2(pw[2], pw[3]);
        const float2 one = dup2(1.0f);
        /* wins - 1: camera 1 loses c01, 2 loses c02 and c12, 3 loses c03, c13 and c23 */
        const float2 n0 = sub2(add2(c01, c02), one), n1 = sub2(c12, c01), n2 = sub2(sub2(one, c02), c12);
        const float2 n3 = sub2(sub2(dup2(2.0f), c03), c13);
        pw[0] = mul2(pw[0], make_float2(__saturatef(n0.x + c03.x), __saturatef(n0.y + c03.y)));
        pw[1] = mul2(pw[1], make_float2(__saturatef(n1.x + c13.x), __saturatef(n1.y + c13.y)));
        pw[2] = mul2(pw[2], make_float2(__saturatef(n2.x + c23.x), __saturatef(n2.y + c23.y)));
        pw[3] = mul2(pw[3], make_float2(__saturatef(n3.x - c23.x), __saturatef(n3.y - c23.y)));
    }
    const float2 best = add2(add2(pw[0], pw[1]), add2(pw[2], pw[3])); /* two of the four are 0 */
    const float2 binv = make_float2(rcp_hw(best.x), rcp_hw(best.y));
    float2 avg[COLORS];
#pragma unroll
    for (int cam = 0; cam < 4; cam++) {
        const float2 sh = mul2(pw[cam], binv);
#pragma unroll
        for (int col = 0; col < COLORS; col++)
            avg[col] = cam ? fma2(sh, D[cam][col], avg[col]) : mul2(sh, D[cam][col]);
    }
    /* A camera left out enters as 0 * D, and one whose weight is a NaN (it and
     * another have the same infinite value) neither wins nor is left out: either
     * way the average is a NaN, which finite values never give */
    {
        float2 any = avg[0];
#pragma unroll
        for (int col = 1; col < COLORS; col++) any = add2(any, avg[col]);
        if (isnan(any.x + any.y)) {
            CameraValues<COLORS> in;
#pragma unroll
            for (int cam = 0; cam < 4; cam++)
#pragma unroll
                for (int col = 0; col < COLORS; col++) in.d[cam][col] = D[cam][col];
            const CameraAverage<COLORS> r = best_two<COLORS>(in, npd2r);
#pragma unroll
            for (int col = 0; col < COLORS; col++) avg[col] = r.a[col];
        }
    }
#pragma unroll
    for (int cam = 0; cam < 4; cam++) {
        float2 d;
#pragma unroll
        for (int col = 0; col < COLORS; col++) {
            const float2 dc = sub2(D[cam][col], avg[col]);
            d = col ? fma2(dc, dc, d) : mul2(dc, dc);
        }
        d = mul2(d, dup2(nksigma));
        pw[cam] = make_float2(weight_hw(d.x), weight_hw(d.y));
    }
    if (dust_remove) {
        const float2 wv = make_float2(fminf(fminf(pw[0].x, pw[1].x), fminf(pw[2].x, pw[3].x)),
                                      fminf(fminf(pw[0].y, pw[1].y), fminf(pw[2].y, pw[3].y)));
        float2 a = sub2(pw[0], wv);
#pragma unroll
        for (int cam = 1; cam < 4; cam++) a = add2(a, pw[cam]);
        a = mul2(a, dup2(1.0f / 3.0f));
        const float2 ra = make_float2(rcp_hw(a.x), rcp_hw(a.y));
        const float2 scale =
            fma2(mul2(mul2(wv, sub2(a, wv)), mul2(ra, ra)), dup2(1.0f / 3.0f), dup2(1.0f));
        const float2 fw = mul2(wv, ra);
        /* the worst camera (first of equals) */
        bool fx = true, fy = true;
#pragma unroll
        for (int cam = 0; cam < 4; cam++) {
            const bool ex = fx && pw[cam].x == wv.x, ey = fy && pw[cam].y == wv.y;
            pw[cam] = mul2(pw[cam], make_float2(ex ? fw.x : scale.x, ey ? fw.y : scale.y));
            fx = fx && !ex;
            fy = fy && !ey;
        }
    }
    float2 ksum = pw[0];
#pragma unroll
    for (int cam = 1; cam < 4; cam++) ksum = add2(ksum, pw[cam]);
    const float2 kinv = make_float2(rcp_hw(ksum.x), rcp_hw(ksum.y));
    float2 kw[4];
#pragma unroll
    for (int cam = 0; cam < 4; cam++) kw[cam] = mul2(kinv, pw[cam]);
#pragma unroll
    for (int col = 0; col < COLORS; col++) {
        float2 v;
#pragma unroll
        for (int cam = 0; cam < 4; cam++) {
            const float2 m = sm[(cam * COLORS + col) * sm_stride + e];
            v = cam ? fma2(kw[cam], m, v) : mul2(kw[cam], m);
        }
        o[col] = mul2(v, m_scale);
    }
    o[COLORS] = mul2(mul2(wnd2, ksum), dup2(0.25f));
#pragma unroll
    for (int cam = 0; cam < 4; cam++) o[COLORS + 1 + cam] = pw[cam];
}

/* k_textures block: four warps, so that the fusion of a tile's 128 pixel pairs
 * takes each of them one turn; one 8-lane group per (camera, colour) job of
 * the block's tiles (colour: one tile of 12 jobs on three warps, the fourth
 * prefetches; mono: four tiles of four jobs) */
constexpr int kTexThreads = 128;
__host__ __device__ constexpr int tex_tiles(int colors) { return colors == 1 ? kTexThreads / 32 : 1; }
/* dynamic shared memory of k_textures: per job its un-windowed tile T, then its
 * debayered tile D (mono: the windowed tile M alone); the transposes of the
 * inverse run over both.  26.3 KB a block: seven blocks, 28 warps, share an SM */
__host__ __device__ constexpr int tex_job(int colors) { return colors == 1 ? kXb : 560; } /* floats; % 32 == 16 as kJob */
constexpr int kTexD = kJob; /* D's offset in a job */
static_assert(kTexD + 256 <= tex_job(3) && 8 * 9 * 4 <= tex_job(1), "a job's tiles and its transposes");
constexpr size_t kTexSmemBytes = sizeof(float) * 12 * tex_job(3);
static_assert(sizeof(float) * 16 * tex_job(1) <= kTexSmemBytes, "mono fits the same block");

/* FROM_T: `clt` holds the jobs' pixel tiles instead of their CLT, as
 * k_tc_stage<InvTcStage> writes them (the un-windowed T for colour, the
 * windowed M for mono, [16][16] row-major at the job's CLT offset): stage 1
 * copies the tile into shared memory instead of inverting the CLT.
 * ALL: the texture-tile outputs and the keep-weights statistics are built
 * (false: the RGBA image only).  COLORS: the colour count, 1 or 3 (p.colors;
 * a compile-time count lets each form keep only its own colour path).  SLOTS: the
 * CLT and the list lie in the frame's workspace (FrameSlots; one parity a launch). */
template <bool FROM_T, bool ALL, int COLORS, bool SLOTS = false>
__global__ void __launch_bounds__(kTexThreads, 7) k_textures(
    Geom g, const int *__restrict__ woi, float *const *clt, int num_texture_tiles,
    const int *__restrict__ list, const int *__restrict__ dev_counts, int count_slot, int list_cap,
    int border_quarter, const float *__restrict__ port_offsets, TextureParams p,
    size_t texture_rbg_stride, float *__restrict__ texture_rbg, size_t texture_stride,
    float *__restrict__ texture_tiles, FrameSlots slots)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ float *s_cp[4];
    __shared__ float s_npd2r[6], s_chw[3], s_chws[3];

    const int tid = threadIdx.x;
    const int l = tid & 7, grp = tid >> 3;
    const unsigned gm = group_mask();
    static_assert(COLORS == 1 || COLORS == 3, "colour count");
    constexpr int colors = COLORS, kTiles = tex_tiles(COLORS), kJobs = 4 * COLORS, kTexJob = tex_job(COLORS);
    /* this group's job: tile `sub` of the block's (kTiles: none), camera, colour */
    const int sub = grp / kJobs, job = grp - sub * kJobs;
    const int cam = job / colors, color = job - cam * colors;
    /* -1 / (2 sigma^2) times log2(e): the fusion's weights are powers of two */
    const float nksigma = -((float)(1.0 / (2.0 * (double)p.diff_sigma * (double)p.diff_sigma)) * kLog2e);
    if (tid < 4) s_cp[tid] = SLOTS ? slots.clt + tid * 768 : clt[tid];
    if (tid == 0) {
        int k = 0;
        for (int i = 0; i < 4; i++)
            for (int j = i + 1; j < 4; j++) {
                const float dx = port_offsets[2 * j] - port_offsets[2 * i];
                const float dy = port_offsets[2 * j + 1] - port_offsets[2 * i + 1];
                s_npd2r[k++] = nksigma / (dx * dx + dy * dy);
            }
        s_chw[0] = p.w0; s_chw[1] = p.w1; s_chw[2] = p.w2;
        /* the RGBA-only colour path debayers without the window (see
         * debayer_job): its distance factors carry the shot scale */
        const float dsc = (!ALL && COLORS == 3 && p.scale_shot > 0.0f) ? p.scale_shot : 1.0f;
        for (int c = 0; c < 3; c++) s_chws[c] = sqrtf(s_chw[c]) * dsc;
    }
    /* D tiles come with the window and the shot scale in the ALL form and
     * for mono (the keep-weights statistics and mono need them as the
     * reference forms them); the RGBA-only colour form debayers without them */

    int count = num_texture_tiles;
    const int *lst = list;
    /* entries at or past `split` sit `gap` further on in the list */
    int split = 0x7fffffff, gap = 0;
    if (dev_counts) {
        /* sub-list length from the list builder, kept inside its quarter */
        count = dev_counts[count_slot];
        count = count < 0 ? 0 : (count > list_cap ? list_cap : count);
        if (border_quarter > 0) {
            /* the border sub-list alone: it grows down from the quarter's end */
            lst = list + (border_quarter - count);
        } else if (border_quarter < 0) {
            /* inner (count_slot) then border (count_slot + 1) sub-lists of one
             * quarter of -border_quarter entries in one pass: tiles of one
             * parity never overlap, so their RGBA updates need no ordering */
            const int q = -border_quarter, ci = count;
            int cb = dev_counts[count_slot + 1];
            cb = cb < 0 ? 0 : (cb > q - ci ? q - ci : cb);
            split = ci;
            gap = q - cb - ci;
            count += cb;
        }
    }
    const bool want_rbg = texture_rbg && texture_rbg_stride;
    const bool want_tiles = ALL && texture_tiles && texture_stride;
    const int keep_weights = ALL ? p.keep_weights : 0;
    const int ns_tiles = (colors == 3) ? (p.keep_weights ? 12 : 4) : (p.keep_weights ? 8 : 2);
    int wx0 = 0, wy0 = 0, wh = 0;
    if (want_rbg) { wx0 = woi[0]; wy0 = woi[1]; wh = woi[3]; }
    const size_t slice_stride = texture_rbg_stride * (size_t)(wh + 1) * 8;
    __syncthreads();
    const int ntiles = g.TX * g.TY;
    /* entry n of this pass: its code, or 0 when there is none or it is not a
     * texture tile */
    auto entry = [&](int n, int &at) -> int {
        if (n >= count) return 0;
        if (SLOTS) {
            const int2 e = slots.list[n];
            at = e.x;
            return e.y;
        }
        const int code = lst[n + (n >= split ? gap : 0)], tile = code >> 8;
        return ((code & (1 << 7)) && tile >= 0 && tile < ntiles) ? code : 0;
    };
    /* window position of a tile's top-left pixel.  The row comes from a float
     * quotient (tiles < 2^24 are exact, the quotient within one of the row)
     * and one correction either way. */
    const float tx_inv = 1.0f / (float)g.TX;
    auto rgba_origin = [&](int tile, int *gy0, int *gx0) {
        int ty = (int)((float)tile * tx_inv), tx = tile - ty * g.TX;
        if (tx < 0) { ty--; tx += g.TX; }
        if (tx >= g.TX) { ty++; tx -= g.TX; }
        *gy0 = (ty - wy0) * 8;
        *gx0 = (tx - wx0) * 8;
    };
    /* RGBA address of pixel (r, c) (slice 0) of the tile at (gy0, gx0), or
     * NULL when it lies left of / above the window (gy0 and gx0 are multiples
     * of 8, so both rows of a pair lie on the same side) */
    auto rgba_at = [&](int gy0, int gx0, int r, int c) -> float * {
        const int gy = gy0 + r, gx = gx0 + c;
        if (gy < 0 || gx < 0) return nullptr;
        return texture_rbg + (size_t)gy * texture_rbg_stride + (size_t)gx;
    };
    /* The next tiles' inputs are prefetched into L2 while the block works on
     * the current ones: their CLT (one 128-byte line per thread: 24 lines of
     * 768 floats per camera, mono 8 lines of 256) and, after the fusion, the
     * RGBA rows their pixels update (both ends of each 16-pixel row of each
     * slice; the previous pass, which writes them, has completed by then). */
    constexpr int kTileStride = SLOTS ? kSlot : 768;
    constexpr int kLines = colors == 3 ? 24 : 8;
    auto prefetch_clt = [&](const int *codes, const int *ats) {
        const int t = colors == 3 ? 0 : tid >> 5, k = colors == 3 ? tid : tid & 31;
        if (k >= 4 * kLines) return;
        int code = 0, at = 0;
#pragma unroll
        for (int i = 0; i < kTiles; i++)
            if (t == i) {
                code = codes[i];
                if (SLOTS) at = ats[i];
            }
        if (!code) return;
        const int pcam = k / kLines, line = k - pcam * kLines;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(s_cp[pcam] + (size_t)(SLOTS ? at : code >> 8) * kTileStride + line * 32));
    };
    auto prefetch_rgba = [&](int code, int gy0, int gx0) {
        /* row r of slice sl */
        const int r = tid & 15, sl = colors == 3 ? tid >> 4 : (tid >> 4) & 1;
        if (!want_rbg || !(code & TP_TASK_TEXTURE_BITS) || sl > colors) return;
        const float *b = rgba_at(gy0, gx0, r, 0);
        if (b) {
            b += (size_t)sl * slice_stride;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(b));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(b + 15));
        }
    };
    /* this group's entry of a block's codes or places (0: none) */
    auto pick = [&](const int *codes) -> int {
        int code = 0;
#pragma unroll
        for (int i = 0; i < kTiles; i++)
            if (sub == i) code = codes[i];
        return code;
    };
    auto job_clt = [&](int code, int at) -> const float * {
        return s_cp[cam] + ((size_t)(SLOTS ? at : code >> 8) * (kTileStride / 256) + color) * 256;
    };

    /* the next tile-parity pass may be scheduled on the SM slots this grid
     * frees as its blocks finish */
    grid_dependents_launch();
    /* A pass launched as a programmatic dependent of the launch before it (the
     * RGBA clear, the correlations of the frame in stages, or the previous
     * tile-parity pass) waits for it before its first access to the RGBA image,
     * which that launch or one before it writes; the inverse transform and
     * debayer of its first tiles run before that wait.  So a launch may be the
     * predecessor of a dependent pass only if everything those steps read (the
     * list and its counts, the window, the CLT or the pixel tiles, the port
     * offsets) was complete before it let the pass start.  The tensor-core
     * inverse transform (FROM_T), which writes the pixel tiles, is not: the
     * first pass after it is an ordinary launch. */
    bool waited = false;
    /* A list that fits the blocks in one turn is spread over them, a block's
     * entries a grid apart, so that a short mono list takes as many blocks as it
     * has entries (300 mono tiles: 8.3 us, 10.3 with four neighbours a block); the
     * entries of a longer one are neighbours, so that its last turn takes few
     * blocks (5120: 22.6 us, 24.6 spread). */
    const int grid = (int)gridDim.x;
    const bool spread = kTiles == 1 || count <= grid * kTiles;
    const int slot_step = spread ? grid : 1, first = (int)blockIdx.x * (spread ? 1 : kTiles);
    int codes[kTiles], ats[kTiles] = {}, gy0 = 0, gx0 = 0;
#pragma unroll
    for (int i = 0; i < kTiles; i++) codes[i] = entry(first + i * slot_step, ats[i]);
    int mine = pick(codes), mine_at = pick(ats);
    if (colors == 3 && want_rbg) rgba_origin(codes[0] >> 8, &gy0, &gx0);

    for (int n = first; n < count; n += grid * kTiles) {
        int next[kTiles], next_at[kTiles] = {};
#pragma unroll
        for (int i = 0; i < kTiles; i++) next[i] = entry(n + grid * kTiles + i * slot_step, next_at[i]);

        /* ---- stages 1-2: per (tile, camera, color) group ---- */
        if (mine) {
            /* T (mono: M), then D; the transposes use the whole job */
            float *tj = smem + grp * kTexJob, *dj = tj + kTexD;
            float2 t[2][8];
            if (FROM_T) {
                /* lane l: columns 2 l and 2 l + 1 of every row pair (a row of the
                 * group's loads is 64 bytes, its stores 16 bytes a lane) */
                const float *src = job_clt(mine, mine_at) + 2 * l;
                const bool al8 = !(reinterpret_cast<uintptr_t>(src) & 7);
                float4 *t4 = reinterpret_cast<float4 *>(tj);
                float2 v[8][2];
#pragma unroll
                for (int rp = 0; rp < 8; rp++)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const float *p = src + (2 * rp + i) * 16;
                        v[rp][i] = al8 ? *reinterpret_cast<const float2 *>(p) : make_float2(p[0], p[1]);
                    }
#pragma unroll
                for (int rp = 0; rp < 8; rp++)
                    t4[rp * 8 + l] = make_float4(v[rp][0].x, v[rp][1].x, v[rp][0].y, v[rp][1].y);
                if (colors > 1) {
                    __syncwarp(gm);
                    const float2 *t2 = reinterpret_cast<const float2 *>(tj);
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int rp = 0; rp < 8; rp++) t[h][rp] = t2[JT2(rp, unfold_col(l, h))];
                }
            } else {
                float raw[4][8];
                load_clt_rows<true>(job_clt(mine, mine_at), raw, l);
                imclt_unfold_job<COLORS == 1>(raw, d_lpf[colors > 1 ? color : 3], tj, tj, t, l, gm);
            }
            if (colors > 1) debayer_job<ALL>(t, tj, dj, color < 2, p.min_shot, p.scale_shot, l, gm);
        }
        __syncthreads();
        prefetch_clt(next, next_at);
        if (!waited) {
            grid_dependency_wait();
            waited = true;
        }

        /* ---- stages 3-4: fuse the four cameras at the thread's pixel pairs
         * and write them out ---- */
#pragma unroll 1
        for (int i = tid; i < 128 * kTiles; i += kTexThreads) {
            const int k = kTiles > 1 ? i >> 7 : 0; /* uniform in a warp */
            int code = codes[0];
#pragma unroll
            for (int j = 1; j < kTiles; j++)
                if (k == j) code = codes[j];
            if (!code) continue;
            const int e = i & 127, r = (e >> 4) * 2, c = e & 15;
            const int px = r * 16 + c;
            const int nbr = code & TP_TASK_TEXTURE_BITS;
            const float2 wnd2 = make_float2(__ldg(&d_tex_wnd2[px]), __ldg(&d_tex_wnd2[px + 16]));
            float2 wi = wnd2;
            if (ALL || colors == 1) wi = make_float2(__ldg(&d_tex_wi[px]), __ldg(&d_tex_wi[px + 16]));
            /* the pixels' RGBA values are loaded before the fusion, whose
             * arithmetic then covers their latency */
            float2 old[4];
            float *b = nullptr;
            if (want_rbg && nbr) {
                if (colors == 1) rgba_origin(code >> 8, &gy0, &gx0);
                b = rgba_at(gy0, gx0, r, c);
            }
            if (b) {
#pragma unroll
                for (int sl = 0; sl <= colors; sl++)
                    old[sl] = make_float2(__ldcg(b + (size_t)sl * slice_stride),
                                          __ldcg(b + (size_t)sl * slice_stride + texture_rbg_stride));
            }
            float2 o[12];
            const float2 *t2 = reinterpret_cast<const float2 *>(smem + k * kJobs * kTexJob);
            if (colors == 3)
                combine_pair<3, ALL>(t2 + kTexD / 2, kTexJob / 2, t2, kTexJob / 2, wnd2, e, s_npd2r, nksigma, s_chw,
                                     s_chws, wnd2, wi, p.dust_remove, keep_weights, o);
            else
                combine_pair<1>(t2, kTexJob / 2, t2, kTexJob / 2, dup2(1.0f), e, s_npd2r, nksigma, s_chw, s_chws,
                                wnd2, wi, p.dust_remove, keep_weights, o);
            if (want_tiles) {
                float *dst = texture_tiles + (size_t)(n + k * slot_step) * texture_stride + px;
#pragma unroll
                for (int sl = 0; sl < 12; sl++)
                    if (sl < ns_tiles) {
                        dst[sl * 256] = o[sl].x;
                        dst[sl * 256 + 16] = o[sl].y;
                    }
            }
            if (b) {
                float2 f = dup2(1.0f);
                if (nbr != TP_TASK_TEXTURE_BITS)
                    f = make_float2(__ldg(&d_alpha_fade[nbr][px]), __ldg(&d_alpha_fade[nbr][px + 16]));
#pragma unroll
                for (int sl = 0; sl <= colors; sl++) {
                    const float2 v = add2(old[sl], mul2(o[sl], f));
                    b[(size_t)sl * slice_stride] = v.x;
                    b[(size_t)sl * slice_stride + texture_rbg_stride] = v.y;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kTiles; i++) codes[i] = next[i];
        mine = pick(codes);
        mine_at = pick(next_at);
        if (want_rbg) {
            if (colors == 3) {
                rgba_origin(codes[0] >> 8, &gy0, &gx0);
                prefetch_rgba(codes[0], gy0, gx0);
            } else {
                int code = 0;
#pragma unroll
                for (int i = 0; i < kTiles; i++)
                    if ((tid >> 5) == i) code = codes[i];
                int y, x;
                rgba_origin(code >> 8, &y, &x);
                prefetch_rgba(code, y, x);
            }
        }
        __syncthreads(); /* the tiles' buffers free */
    }
    /* a block without a tile waits too: a grid has completed only once the
     * launches before it have */
    if (!waited) grid_dependency_wait();
}

} /* namespace tp */

/*
 * tp_convert.cuh - forward CLT with aberration correction (the drop-in for the
 * reference's convert_correct_tiles, src/TileProcessor.cuh:1859-1937 and
 * convertCorrectTile :3106-3635).
 *
 * One 8-lane group per (tile, camera, color) job; a warp holds four jobs of the
 * same camera and color for four consecutive tasks, so the green jobs (two
 * Bayer phases and a DST pass) never share a warp with the cheaper red/blue
 * ones.  Per job:
 *   lane v gathers DTT column v of the folded, windowed Bayer samples (8
 *   same-color pixels of one image column; the group's 8 loads of one row are
 *   one 64-byte run), applies the column DCT-IV, transposes through shared
 *   memory and applies the row DCT-IV (green: also the row DST-IV of the
 *   sine-windowed fold), ending with row v of CC (and SC);
 *   the remaining quadrants come from the Bayer mirror symmetries, within the
 *   row or from the opposite row; the CLT-domain kernel, the two
 *   residual-shift rotations and the optional LPF are per coefficient, run on
 *   pairs of coefficients (mul2 / fma2) and end in rows of 32 bytes, the width
 *   of one load of the kernel tile and one store of the result.
 *
 * Lanes that hold rows make every access of the kernel tile and the CLT a
 * whole 32-byte sector; holding columns (the transposed order of the two
 * passes) took eight times as many load and store instructions and kept the L1
 * busy 79% of the time at 55% issue.  815 warp instructions a job (1232
 * before); a 2592x1936 frame went from 0.454 to 0.351 ms (2.87 to 3.71 TB/s of
 * its 1.30 GB).  What bounds it now is the latency of a job's steps at 15 warps
 * per SM: the samples, the kernel rows and the result of a job are 48 to 80
 * registers, and more warps spill them (256 threads at 80 registers 0.448 ms,
 * 192 at 96 0.451, 128 at 158 0.358).
 */
#pragma once
#include "tp_common.cuh"

namespace tp {

/* Clamp of the integer tile corner (src/TileProcessor.cuh:3188-3193,
 * :3246-3252); `n` is the image size along the axis. */
__device__ __forceinline__ int corner_clamp(int itl, int n, bool horizontal, int mode)
{
    if (itl < 0) itl &= 1;
    if (itl >= n - 8) {
        if (mode == TP_BORDER_REFERENCE && horizontal)
            itl = itl & (1 + (n - 8 - 2)); /* the reference's `itlx & 1 +(W-10)` */
        else
            itl = (itl & 1) + (n - 8 - 2);
    }
    return itl;
}

__device__ __forceinline__ int pair_clamp(int idx, int n)
{
    if (idx < 0) return idx & 1;
    if (idx >= n) return (n - 2) + (idx & 1);
    return idx;
}

/* Where a job's window sits and how its kernel tile and shifts follow from
 * the task's tile centre (float32, as the reference computes them:
 * src/TileProcessor.cuh:3129-3255). */
struct JobGeometry {
    size_t kidx;    /* kernel tile (x, y, colour) index into the table   */
    int itlx, itly; /* integer corner of the 16x16 window                */
    float shx, shy; /* residual shifts                                   */
};

__device__ __forceinline__ JobGeometry job_geometry(const Geom &g, const float *__restrict__ extra_tab, float cx,
                                                    float cy, int color, const float *pre_ex)
{
    JobGeometry j;
    const float step_inv = __int_as_float((127 - g.ls) << 23);
    int ktx = __float2int_rn(__fmaf_rn(cx, step_inv, 1.0f));
    int kty = __float2int_rn(__fmaf_rn(cy, step_inv, 1.0f));
    ktx = min(g.KH - 1, max(0, ktx));
    kty = min(g.KV - 1, max(0, kty));
    const float kdx = (cx - (float)(ktx << g.ls)) + (float)(1 << (g.ls - 1));
    const float kdy = (cy - (float)(kty << g.ls)) + (float)(1 << (g.ls - 1));
    j.kidx = ((size_t)ktx + (size_t)kty * g.KH) * 3 + color;
    /* the kernel tile's offsets: prefetched by the caller (pre_ex[6]) or here */
    const float *ex = extra_tab + j.kidx * 8;
    const float data_x = pre_ex ? pre_ex[0] : __ldg(ex + 0), data_y = pre_ex ? pre_ex[1] : __ldg(ex + 1);
    const float dxc_dx = pre_ex ? pre_ex[2] : __ldg(ex + 4), dxc_dy = pre_ex ? pre_ex[3] : __ldg(ex + 5);
    const float dyc_dx = pre_ex ? pre_ex[4] : __ldg(ex + 6), dyc_dy = pre_ex ? pre_ex[5] : __ldg(ex + 7);
    const float px = (cx - 8.0f) - __fmaf_rn(dxc_dy, kdy, __fmaf_rn(dxc_dx, kdx, data_x));
    const float py = (cy - 8.0f) - __fmaf_rn(dyc_dy, kdy, __fmaf_rn(dyc_dx, kdx, data_y));
    j.itlx = corner_clamp(__float2int_rd(px + 0.5f), g.W, true, g.border_mode);
    j.itly = corner_clamp(__float2int_rd(py + 0.5f), g.H, false, g.border_mode);
    j.shx = (float)j.itlx - px;
    j.shy = (float)j.itly - py;
    return j;
}

/* A job's window staged in shared memory (the TMA-fed convert kernel): 16
 * rows of 20 floats from the 16-byte boundary at or left of the corner */
constexpr int kCvWinW = 20, kCvWinH = 16;

/* (cos, sin) of a lane's residual-shift rotations: column l horizontally, row
 * l vertically, pi s (2l + 1) / 16.  Lane 0's are the rotations of the shifted
 * windows. */
struct JobAngles {
    float ch, sh, cv, sv;
};

__device__ __forceinline__ JobAngles job_angles(const JobGeometry &j, int l)
{
    JobAngles a;
    sincospif((j.shx * (float)(2 * l + 1)) * 0.0625f, &a.sh, &a.ch);
    sincospif((j.shy * (float)(2 * l + 1)) * 0.0625f, &a.sv, &a.cv);
    return a;
}

/* Floats of a group's shared buffer: the shifted windows (vertical, horizontal
 * cosine and sine fold: [2 parities][8 DTT indices] each), the horizontal
 * rotations (8 cosines, 8 sines), then two 8x8 transposes with rows of 12
 * (16-byte reads along rows and 4-byte writes down columns are conflict-free)
 * or the mirror exchange with rows of 20.  264 % 32 == 8 keeps the four groups
 * of a warp on distinct banks. */
constexpr int kCvRot = 48, kCvTr = 64, kCvTrRow = 12, kCvMirRow = 20;
constexpr int kCvBuf = 264;
static_assert(kCvTr + 2 * 8 * kCvTrRow <= kCvBuf && kCvTr + 8 * kCvMirRow <= kCvBuf, "group buffer");

/* 8 consecutive floats (16-byte aligned) as pairs */
__device__ __forceinline__ void lds_row(const float *p, float2 v[4])
{
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = make_float2(a.x, a.y);
    v[1] = make_float2(a.z, a.w);
    v[2] = make_float2(b.x, b.y);
    v[3] = make_float2(b.z, b.w);
}

/* The job's Bayer samples of DTT column l: pix[gp][u] = the sample of Bayer
 * phase gp (green has two) that folds onto DTT row u, from image addresses as
 * src/TileProcessor.cuh:3257-3416.  win (may be NULL): the job's window in
 * shared memory, used for windows inside the image (the same samples). */
__device__ __forceinline__ void load_pixels(const Geom &g, size_t dstride, const float *__restrict__ img,
                                            const JobGeometry &j, int color, int l, float pix[2][8],
                                            const float *win = nullptr, int win_dx = 0)
{
    const int itlx = j.itlx, itly = j.itly;
    const int c0 = color & 1, c1 = (color >> 1) & 1;
    const bool fast = (itlx >= 0) && (itlx < g.W - 16) && (itly >= 0) && (itly < g.H - 16);
    const long long last = (long long)g.image_rows * (long long)dstride - 1;
#pragma unroll
    for (int gp = 0; gp < 2; gp++) {
        if (gp > c1) break;
        const int colp = (itlx & 1) ^ (1 ^ c0 ^ c1 ^ gp);
        const int rowp = (itly & 1) ^ (c0 ^ gp);
        const int lc = fold_sample(l, colp);
        /* row i of the phase (rowp + 2i) at pix[u(i)]: the DTT rows of i at rowp
         * 0; at rowp 1 neighbours 2k and 2k + 1 change places (fold_phase) */
        constexpr int kI[8] = {6, 5, 7, 4, 0, 3, 1, 2};
        if (fast && win) {
            /* the window staged in shared memory: rows of kCvWinW floats from
             * column itlx - win_dx */
            const float *w = win + rowp * kCvWinW + win_dx + lc;
#pragma unroll
            for (int u = 0; u < 8; u++) pix[gp][u] = w[2 * kI[u] * kCvWinW];
        } else if (fast) {
            const float *w = img + (size_t)(itly + rowp) * dstride + (itlx + lc);
#pragma unroll
            for (int u = 0; u < 8; u++) pix[gp][u] = __ldg(w + kI[u] * (2 * dstride));
        } else if (g.border_mode == TP_BORDER_CLAMP) {
            const float *w = img + pair_clamp(itlx + lc, g.W);
#pragma unroll
            for (int u = 0; u < 8; u++)
                pix[gp][u] = __ldg(w + (size_t)pair_clamp(itly + rowp + 2 * kI[u], g.H) * dstride);
        } else {
            /* src/TileProcessor.cuh:3328-3361: columns clamped by IMG_HEIGHT/2,
             * rows by IMG_WIDTH/2, row offset `rowp` added once */
            const int cp = min(g.H / 2 - 1, max(0, itlx >> 1));
            const int col = (cp << 1) + (itlx & 1) + lc;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int rp = min(g.W / 2 - 1, max(0, (itly >> 1) + kI[u]));
                long long a = (long long)(rowp + (rp << 1) + (itly & 1)) * (long long)dstride + col;
                a = a > last ? last : (a < 0 ? 0 : a);
                pix[gp][u] = __ldg(img + a);
            }
        }
    }
}

/* The fold by columns: lane l builds DTT column l (P[k] = rows 2k, 2k + 1; Q
 * for green) of the folded, windowed Bayer samples of load_pixels, both Bayer
 * phases of green summed.  Leaves the group's rotations in buf. */
__device__ __forceinline__ void fold_cols(const JobGeometry &j, const JobAngles &ang, int color, int l, unsigned gm,
                                          float *buf, const float pix[2][8], float2 P[4], float2 Q[4])
{
    const int itlx = j.itlx, itly = j.itly;
    const int c0 = color & 1, c1 = (color >> 1) & 1;
    const float hc = __shfl_sync(gm, ang.ch, 0, 8), hs = __shfl_sync(gm, ang.sh, 0, 8);
    const float vc = __shfl_sync(gm, ang.cv, 0, 8), vs = __shfl_sync(gm, ang.sv, 0, 8);
    /* the lane's two of the 16 window samples, n = l and l + 8, at their
     * parity and DTT index, with the signs of the fold branches (cosine: + for
     * n < 4; sine: + for n < 12) */
    {
        const float s0 = l < 4 ? 1.0f : -1.0f;
        const int i0 = (l & 1) * 8 + (l < 4 ? l + 4 : 11 - l), i1 = (l & 1) * 8 + (l < 4 ? 3 - l : l - 4);
        const float h0 = shifted_window_lane(l, hc, hs), h1 = shifted_window_lane(l + 8, hc, hs);
        buf[i0] = s0 * shifted_window_lane(l, vc, vs);
        buf[i1] = -shifted_window_lane(l + 8, vc, vs);
        buf[16 + i0] = s0 * h0;
        buf[16 + i1] = -h1;
        buf[32 + i0] = h0;
        buf[32 + i1] = s0 * h1;
        buf[kCvRot + l] = ang.ch;
        buf[kCvRot + 8 + l] = ang.sh;
    }
    __syncwarp(gm);
#pragma unroll
    for (int gp = 0; gp < 2; gp++) {
        if (gp > c1) break;
        const int colp = (itlx & 1) ^ (1 ^ c0 ^ c1 ^ gp);
        const int rowp = (itly & 1) ^ (c0 ^ gp);
        float2 wv[4];
        lds_row(buf + rowp * 8, wv);
        const float2 whc = dup2(buf[16 + colp * 8 + l]);
        const float2 whs = c1 ? dup2(buf[32 + colp * 8 + l]) : whc;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float x = pix[gp][2 * k], y = pix[gp][2 * k + 1];
            const float2 d = mul2(make_float2(rowp ? y : x, rowp ? x : y), wv[k]);
            P[k] = gp ? fma2(d, whc, P[k]) : mul2(d, whc);
            if (c1) Q[k] = gp ? fma2(d, whs, Q[k]) : mul2(d, whs);
        }
    }
}

/* Lane l's part of the four quadrants of a kernel tile, read-only for the whole
 * launch.  True: row l, one 256-bit load each where the tile lies on a 32-byte
 * boundary, two of 16 bytes on a 16-byte one.  Else column l (a load of the
 * group is a run of 32 bytes), which kernel_rows turns into row l when the rows
 * are needed. */
__device__ __forceinline__ bool load_kernel(const float *tile, int l, float2 v[4][4])
{
    const float *p = tile + l * 8;
    if (!(reinterpret_cast<uintptr_t>(tile) & 31)) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(v[q][0].x), "=f"(v[q][0].y), "=f"(v[q][1].x), "=f"(v[q][1].y), "=f"(v[q][2].x),
                           "=f"(v[q][2].y), "=f"(v[q][3].x), "=f"(v[q][3].y)
                         : "l"(p + q * 64));
        return true;
    }
    if (!(reinterpret_cast<uintptr_t>(tile) & 15)) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(p + q * 64) + k);
                v[q][2 * k] = make_float2(x.x, x.y);
                v[q][2 * k + 1] = make_float2(x.z, x.w);
            }
        return true;
    }
    p = tile + l;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int k = 0; k < 4; k++)
            v[q][k] = make_float2(__ldg(p + q * 64 + 16 * k), __ldg(p + q * 64 + 16 * k + 8));
    return false;
}

/* columns of load_kernel to rows, through tr (200 floats of the group's) */
__device__ __forceinline__ void kernel_rows(float2 v[4][4], float *tr, int l, unsigned gm)
{
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
        __syncwarp(gm);
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                tr[(8 * h + 2 * k) * kCvTrRow + l] = v[q + h][k].x;
                tr[(8 * h + 2 * k + 1) * kCvTrRow + l] = v[q + h][k].y;
            }
        __syncwarp(gm);
#pragma unroll
        for (int h = 0; h < 2; h++) lds_row(tr + (8 * h + l) * kCvTrRow, v[q + h]);
    }
}

/* Row l of the four quadrants of a result at out.  STREAM:
 * global memory, evict-first (the kernel writes 963 MB of CLT for a full quad
 * frame, far more than L2 holds, and later kernels read it back; retaining the
 * stores in L2 would only evict the kernel tiles and Bayer rows that
 * neighbouring jobs of this kernel still read): 32 bytes a lane where the tile
 * lies on a 32-byte boundary, two times 16 on a 16-byte one, else through tr
 * (200 floats of the group's), so that a store of the group is a run of 32
 * bytes; !STREAM: shared memory, 16-byte aligned.  A 2592x1936 frame (0.326 ms
 * aligned) with kernel tables and CLT 16 / 8 / 4 bytes off such a boundary takes
 * 0.386 / 0.496 / 0.496 ms; 0.699 / 0.666 / 0.649 with a lane's row moved value
 * by value in both directions. */
template <bool STREAM>
__device__ __forceinline__ void store_rows(float *out, const float2 v[4][4], float *tr, int l, unsigned gm)
{
    float *p = out + l * 8;
    if (!STREAM) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int k = 0; k < 2; k++)
                reinterpret_cast<float4 *>(p + q * 64)[k] =
                    make_float4(v[q][2 * k].x, v[q][2 * k].y, v[q][2 * k + 1].x, v[q][2 * k + 1].y);
    } else if (!(reinterpret_cast<uintptr_t>(p) & 31)) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + q * 64),
                         "f"(v[q][0].x), "f"(v[q][0].y), "f"(v[q][1].x), "f"(v[q][1].y), "f"(v[q][2].x),
                         "f"(v[q][2].y), "f"(v[q][3].x), "f"(v[q][3].y)
                         : "memory");
    } else if (!(reinterpret_cast<uintptr_t>(p) & 15)) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int k = 0; k < 2; k++)
                __stcs(reinterpret_cast<float4 *>(p + q * 64) + k,
                       make_float4(v[q][2 * k].x, v[q][2 * k].y, v[q][2 * k + 1].x, v[q][2 * k + 1].y));
    } else {
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            __syncwarp(gm);
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int k = 0; k < 2; k++)
                    reinterpret_cast<float4 *>(tr + (8 * h + l) * kCvTrRow)[k] =
                        make_float4(v[q + h][2 * k].x, v[q + h][2 * k].y, v[q + h][2 * k + 1].x, v[q + h][2 * k + 1].y);
            __syncwarp(gm);
#pragma unroll
            for (int r = 0; r < 16; r++) __stcs(out + q * 64 + r * 8 + l, tr[r * kCvTrRow + l]);
        }
    }
}

/* The rest of a job after its fold (fold_cols: P, Q, the rotations in buf; kq,
 * rows: its kernel tile as load_kernel leaves it): 2-D transform, CLT-domain convolution with the kernel tile, residual
 * shifts, LPF, store. */
template <bool STREAM>
__device__ __forceinline__ void convert_finish(const JobGeometry &jg, const JobAngles &ang, int color, int lpf_mask, float *__restrict__ out,
                                               float *buf, int l, unsigned gm, float2 kq[4][4], bool rows,
                                               const float2 P[4], const float2 Q[4])
{
    const int itlx = jg.itlx, itly = jg.itly;
    const int c1 = (color >> 1) & 1;
    float *tr = buf + kCvTr;
    /* ---- 2-D transform: columns (registers), transpose, rows; a[q]: row l
     * of the four quadrants as pairs ---- */
    float2 a[4][4];
    {
        float cc[8], row[8];
        if (c1) {
            /* the cosine and the sine-windowed fold side by side */
            float2 x[8], y[8];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                x[2 * k] = make_float2(P[k].x, Q[k].x);
                x[2 * k + 1] = make_float2(P[k].y, Q[k].y);
            }
            dct4_pair(x, y);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                tr[k * kCvTrRow + l] = y[k].x;
                tr[(8 + k) * kCvTrRow + l] = y[k].y;
            }
        } else {
            const float x[8] = {P[0].x, P[0].y, P[1].x, P[1].y, P[2].x, P[2].y, P[3].x, P[3].y};
            float y[8];
            dtt8<0>(x, y);
#pragma unroll
            for (int k = 0; k < 8; k++) tr[k * kCvTrRow + l] = y[k];
        }
        __syncwarp(gm);
        load_row8s(tr + l * kCvTrRow, row);
        dtt8<0>(row, cc); /* row l of CC */
        float sc[8];
        if (c1) {
            load_row8s(tr + (8 + l) * kCvTrRow, row);
            dtt8<1>(row, sc); /* row l of SC */
        } else {
            /* R, B: SC[i][7-j] = +-CC[i][j] (src/TileProcessor.cuh:3459-3475) */
            const float neg1 = 1.0f - 2.0f * (float)((itlx & 1) ^ (1 ^ color));
#pragma unroll
            for (int m = 0; m < 8; m++) sc[m] = neg1 * cc[7 - m];
        }
        __syncwarp(gm); /* the transposes read */
        /* SS[7-i][7-j] = +-CC[i][j], CS[7-i][7-j] = +-SC[i][j] (:3486-3504):
         * from the opposite row, reversed */
        float *mir = tr + l * kCvMirRow;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            reinterpret_cast<float4 *>(mir)[k] =
                make_float4(cc[7 - 4 * k], cc[6 - 4 * k], cc[5 - 4 * k], cc[4 - 4 * k]);
            reinterpret_cast<float4 *>(mir + 8)[k] =
                make_float4(sc[7 - 4 * k], sc[6 - 4 * k], sc[5 - 4 * k], sc[4 - 4 * k]);
        }
        __syncwarp(gm);
        const float2 neg2 = dup2(1.0f - 2.0f * (float)((itlx & 1) ^ (itly & 1) ^ 1 ^ c1));
        lds_row(tr + (7 - l) * kCvMirRow, a[3]);
        lds_row(tr + (7 - l) * kCvMirRow + 8, a[2]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            a[0][k] = make_float2(cc[2 * k], cc[2 * k + 1]);
            a[1][k] = make_float2(sc[2 * k], sc[2 * k + 1]);
            a[2][k] = mul2(neg2, a[2][k]);
            a[3][k] = mul2(neg2, a[3][k]);
        }
    }

    /* ---- CLT-domain convolution (src/TileProcessor.cuh:2778-2827), then the
     * residual shift: horizontal (per column, shared across the group), then
     * vertical (this lane's row) (:2715-2776) ---- */
    if (!rows) kernel_rows(kq, tr, l, gm);
    float2 ch[4], sh[4];
    lds_row(buf + kCvRot, ch);
    lds_row(buf + kCvRot + 8, sh);
    const float2 cv = dup2(ang.cv), sv = dup2(ang.sv), nsv = dup2(-ang.sv);
    float2 o[4][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 a0 = a[0][k], a1 = a[1][k], a2 = a[2][k], a3 = a[3][k];
        const float2 k0 = kq[0][k], k1 = kq[1][k], k2 = kq[2][k], k3 = kq[3][k];
        const float2 x0 = sub2(fma2(a3, k3, mul2(a0, k0)), fma2(a2, k2, mul2(a1, k1)));
        const float2 x1 = sub2(fma2(a0, k1, mul2(a1, k0)), fma2(a3, k2, mul2(a2, k3)));
        const float2 x2 = sub2(fma2(a0, k2, mul2(a2, k0)), fma2(a3, k1, mul2(a1, k3)));
        const float2 x3 = fma2(a0, k3, fma2(a1, k2, fma2(a2, k1, mul2(a3, k0))));
        const float2 nsh = make_float2(-sh[k].x, -sh[k].y);
        const float2 y0 = fma2(x0, ch[k], mul2(x1, nsh)), y1 = fma2(x0, sh[k], mul2(x1, ch[k]));
        const float2 y2 = fma2(x2, ch[k], mul2(x3, nsh)), y3 = fma2(x2, sh[k], mul2(x3, ch[k]));
        o[0][k] = fma2(y0, cv, mul2(y2, nsv));
        o[2][k] = fma2(y0, sv, mul2(y2, cv));
        o[1][k] = fma2(y1, cv, mul2(y3, nsv));
        o[3][k] = fma2(y1, sv, mul2(y3, cv));
    }
    if ((lpf_mask >> color) & 1) { /* optional LPF (:3572-3593) */
        float2 f[4];
        lds_row(&d_lpf[color][l * 8], f);
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int k = 0; k < 4; k++) o[q][k] = mul2(o[q][k], f[k]);
    }
    store_rows<STREAM>(out, o, tr, l, gm);
    __syncwarp(gm); /* buf free for the group's next job */
}

template <bool STREAM = false>
__device__ __forceinline__ void convert_job(const Geom &g, size_t dstride,
                                            const float *__restrict__ extra_tab,
                                            const float *__restrict__ kern_tab,
                                            const float *__restrict__ img, float cx, float cy,
                                            int color, int lpf_mask, float *__restrict__ out,
                                            float *buf, int l, unsigned gm, const float *pre_ex = nullptr)
{
    const JobGeometry jg = job_geometry(g, extra_tab, cx, cy, color, pre_ex);
    /* the samples and the kernel tile's rows in flight together, while the
     * angles and windows are computed */
    float pix[2][8];
    load_pixels(g, dstride, img, jg, color, l, pix);
    float2 kq[4][4];
    const bool rows = load_kernel(kern_tab + jg.kidx * 256, l, kq);
    const JobAngles ang = job_angles(jg, l);
    float2 P[4], Q[4];
    fold_cols(jg, ang, color, l, gm, buf, pix, P, Q);
    convert_finish<STREAM>(jg, ang, color, lpf_mask, out, buf, l, gm, kq, rows, P, Q);
}

/* A warp's item of the grid-stride loop is four consecutive tasks of one camera
 * with PER colours: 3, one job after another (the tasks' fields and kernel tile
 * are then found once for three jobs, and the warp keeps its camera's tables),
 * or 1 (item % 12 = colour * 4 + camera), which spreads a small list over
 * three times as many warps.  The host takes PER 1 as long as its items fit
 * the resident warps in one turn: past that the shared work is worth more
 * (2592x1936 frame: 0.351 ms, 0.374 with PER 1).
 * The fields of the next item's tasks are read an item ahead, the offsets of
 * the next job's kernel tile a job ahead, and the kernel tile itself is
 * prefetched into L2 an item ahead (lane l: bytes 128 l .. 128 l + 127 of the
 * 1 KB tile).
 * SLOTS: the CLT goes to the frame's workspace by task, and each textured task
 * into the list of its parity (FrameSlots; the order within a list does not matter). */
constexpr int kConvertThreads = 160;
template <int PER, bool SLOTS = false>
__global__ void __launch_bounds__(kConvertThreads, 3) k_convert_correct_tiles(
    Geom g, size_t dstride, float *const *kernel_offsets, float *const *kernels,
    float *const *images, const tp_task *__restrict__ tasks, float *const *clt, int num_tiles,
    int lpf_mask, FrameSlots slots)
{
    static_assert(PER == 1 || PER == 3, "colours per item");
    __shared__ __align__(16) float cbuf[kConvertThreads / 8][kCvBuf];
    const int l = threadIdx.x & 7;
    const int grp = threadIdx.x >> 3;
    const unsigned gm = group_mask();
    /* a programmatic dependent of the RGBA clear (or of the part before, whose
     * workspace it takes over); the correlations may be scheduled behind it */
    if (SLOTS) {
        grid_dependency_wait();
        grid_dependents_launch();
    }
    const int step = gridDim.x * (blockDim.x >> 5);
    const int items = ((num_tiles + 3) >> 2) * (12 / PER);
    /* a task of the list as this group sees it: its tile (-1: none) and centre */
    struct Task {
        int tile;
        float cx, cy;
        int ktile; /* kernel tile x + y * KH, times 3 */
    };
    auto fetch = [&](int w) -> Task {
        Task t = {-1, 0.0f, 0.0f, 0};
        if (w >= items) return t;
        const int chunk = PER == 3 ? w >> 2 : w / 12, cam = PER == 3 ? w & 3 : (w - chunk * 12) & 3;
        const int n = chunk * 4 + (grp & 3);
        if (n >= num_tiles) return t;
        const tp_task *p = tasks + n;
        const int task = __ldg(&p->task), txy = __ldg(&p->txy);
        const int tx = txy & (SLOTS ? 0xffff : 0xfff), ty = txy >> 16;
        t.cx = __ldg(&p->xy[cam][0]);
        t.cy = __ldg(&p->xy[cam][1]);
        if (!task || tx >= g.TX || ty < 0 || ty >= g.TY) return t;
        t.tile = SLOTS ? n : ty * g.TX + tx;
        if (SLOTS && cam == 0 && l == 0 && (PER == 3 || (w % 12) >> 2 == 0) && (task & TP_TASK_TEXTURE_BITS)) {
            /* its entry in the texture list of its parity */
            const int parity = (tx & 1) | ((ty & 1) << 1);
            const int k = atomicAdd(&slots.counts[parity], 1);
            slots.list[(size_t)parity * num_tiles + k] =
                make_int2(n, ((ty * g.TX + tx) << 8) | (1 << 7) | (task & TP_TASK_TEXTURE_BITS));
        }
        /* the kernel tile (as job_geometry chooses it) */
        const float step_inv = __int_as_float((127 - g.ls) << 23);
        const int ktx = min(g.KH - 1, max(0, __float2int_rn(__fmaf_rn(t.cx, step_inv, 1.0f))));
        const int kty = min(g.KV - 1, max(0, __float2int_rn(__fmaf_rn(t.cy, step_inv, 1.0f))));
        t.ktile = (ktx + kty * g.KH) * 3;
        return t;
    };
    auto fetch_extra = [&](const float *extra, int ktile, int color, float ex[6]) {
        const float *e = extra + (size_t)(ktile + color) * 8;
        ex[0] = __ldg(e + 0); ex[1] = __ldg(e + 1);
        ex[2] = __ldg(e + 4); ex[3] = __ldg(e + 5);
        ex[4] = __ldg(e + 6); ex[5] = __ldg(e + 7);
    };
    int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    /* PER 3: the grid, and so the step, is a multiple of 4: a warp keeps its camera */
    int cam = PER == 3 ? w & 3 : (w % 12) & 3;
    const float *kern = kernels[cam], *extra = kernel_offsets[cam], *img = images[cam];
    float *out = SLOTS ? slots.clt + cam * 768 : clt[cam];
    Task next = fetch(w);
    float nex[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (next.tile >= 0) fetch_extra(extra, next.ktile, PER == 3 ? 0 : (w % 12) >> 2, nex);
    for (; w < items; w += step) {
        const Task t = next;
        const int color0 = PER == 3 ? 0 : (w % 12) >> 2;
        next = fetch(w + step);
        const float *kern_n = kern, *extra_n = extra, *img_n = img;
        float *out_n = out;
        const int color_n = PER == 3 ? 0 : ((w + step) % 12) >> 2;
        if (PER == 1) {
            const int c = ((w + step) % 12) & 3;
            kern_n = kernels[c];
            extra_n = kernel_offsets[c];
            img_n = images[c];
            out_n = SLOTS ? slots.clt + c * 768 : clt[c];
        }
#pragma unroll 1
        for (int i = 0; i < PER; i++) {
            const int color = color0 + i;
            float ex[6];
#pragma unroll
            for (int k = 0; k < 6; k++) ex[k] = nex[k];
            if (i + 1 < PER) {
                if (t.tile >= 0) fetch_extra(extra, t.ktile, color + 1, nex);
            } else if (next.tile >= 0) {
                fetch_extra(extra_n, next.ktile, color_n, nex);
            }
            if (next.tile >= 0)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(kern_n + (size_t)(next.ktile + color_n + i) * 256 + l * 32));
            if (t.tile < 0) continue;
            convert_job<true>(g, dstride, extra, kern, img, t.cx, t.cy, color, lpf_mask,
                                out + (size_t)t.tile * (SLOTS ? kSlot : 768) + color * 256, cbuf[grp], l, gm, ex);
        }
        if (PER == 1) {
            kern = kern_n;
            extra = extra_n;
            img = img_n;
            out = out_n;
        }
    }
}

} /* namespace tp */

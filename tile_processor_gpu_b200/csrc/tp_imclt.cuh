/*
 * tp_imclt.cuh - inverse CLT of color planes into an image by overlap-add
 * (the drop-in for the reference's imclt_rbg, src/TileProcessor.cuh:2588-2710,
 * with imclt :3700-3835).
 *
 * One 8-lane group per tile: it inverts the four quadrants on packed pairs
 * (imclt_pairs) and leaves the signed unfolded 16x16 tile d in shared memory
 * as row pairs.  A pixel accumulates its (up to four) tiles in the order of
 * the reference's four parity passes with the reference's round-down fused
 * multiply-add, w * d + previous, w the product of the half-sine windows;
 * pass (0, 0) overwrites the image.
 *
 * k_imclt_rbg is one parity pass: each tile is added into the image in memory.
 * k_imclt_rbg_all is the whole image of all three colors: a block walks down a
 * strip of kImclTiles tile columns, keeps the tile row above in shared memory,
 * and writes each pixel once, its four contributions added in pass order.
 * The twelve passes read and wrote every pixel four times in twelve launches
 * of a latency-bound kernel: a 2592x1936 image took 0.284 ms, now 0.108 (2.8
 * TB/s of its 0.30 GB; five blocks per SM at 96 registers: four 0.128, six
 * spill, 0.143).  What bounds it is the chain load - transform - barrier -
 * write of a tile row.
 */
#pragma once
#include "tp_common.cuh"
#include "tp_texture.cuh"

namespace tp {

/* (w * d + v) on both halves, rounded down */
__device__ __forceinline__ float2 fma2_rd(float2 w, float2 d, float2 v)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rm.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(w.x), "f"(w.y), "f"(d.x), "f"(d.y), "f"(v.x), "f"(v.y));
    return r;
}

/* the signed unfolded tile of raw (load_clt_rows) as row pairs in `tile`, whose
 * memory the transposes use first (kXb floats) */
__device__ __forceinline__ void imclt_tile(const float raw[4][8], float *tile, int l, unsigned gm)
{
    constexpr float kOne[16] = {};
    float2 a02[8], a13[8], t[8];
    imclt_pairs(raw, nullptr, reinterpret_cast<float4 *>(tile), a02, a13, l, gm);
    __syncwarp(gm);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = unfold_col(l, h);
        unfold_column<true>(a02, a13, l, c, 1.0f, kOne, t);
#pragma unroll
        for (int rp = 0; rp < 8; rp++) reinterpret_cast<float2 *>(tile)[JT2(rp, c)] = t[rp];
    }
}

__global__ void __launch_bounds__(256) k_imclt_rbg(Geom g, const float *__restrict__ clt,
                                                   float *__restrict__ rbg, int color, int v_offset,
                                                   int h_offset, size_t dstride)
{
    __shared__ __align__(16) float tbuf[256 / 8][kXb];
    const int l = threadIdx.x & 7;
    const int grp = threadIdx.x >> 3;
    const unsigned gm = group_mask();
    const float2 *t2 = reinterpret_cast<const float2 *>(tbuf[grp]);
    const int txh = (g.TX + (h_offset ^ 1)) >> 1;
    const int tyh = (g.TY + (v_offset ^ 1)) >> 1;
    const long long ntl = (long long)txh * tyh;
    const long long groups_total = (long long)gridDim.x * (blockDim.x >> 3);
    const int pass = (v_offset << 1) + h_offset;
    float *plane = rbg + dstride * (size_t)(g.H + 8) * color;
    for (long long n = (long long)blockIdx.x * (blockDim.x >> 3) + grp; n < ntl; n += groups_total) {
        const int ty = 2 * (int)(n / txh) + v_offset;
        const int tx = 2 * (int)(n % txh) + h_offset;
        float raw[4][8];
        load_clt_rows<true>(clt + (((size_t)ty * g.TX + tx) * 3 + color) * 256, raw, l);
        imclt_tile(raw, tbuf[grp], l, gm);
        __syncwarp(gm);
        float *top = plane + (size_t)ty * 8 * dstride + (size_t)tx * 8;
        const bool mark0 = g.debug_marks && tx == 0 && ty == 0;
        const bool mark2 = g.debug_marks && tx == 161 && ty == 111;
#pragma unroll
        for (int hc = 0; hc < 2; hc++) {
            const int c = l + 8 * hc;
            const float wc = 0.5f * __ldg(&d_hwin[c]);
            for (int r = 0; r < 16; r++) {
                const float w = (0.5f * c_hwin[r]) * wc;
                float *px = top + (size_t)r * dstride + c;
                const float prev = pass ? *px : 0.0f;
                const float2 d = t2[JT2(r >> 1, c)];
                float val = __fmaf_rd(w, (r & 1) ? d.y : d.x, prev);
                if (mark0) val = 100.0f;
                else if (mark2) val *= 2.0f;
                *px = val;
            }
        }
        __syncwarp(gm);
    }
}

/* tile columns a block inverts per row (one per group); they complete
 * kImclTiles - 1 columns of 8x8 cells, cell (cy, cx) lying under tiles cy - 1
 * and cy, cx - 1 and cx */
constexpr int kImclTiles = 16, kImclThreads = 8 * kImclTiles, kImclCells = kImclTiles - 1;
constexpr int kImclBlocksPerSm = 5;

/* Block (x, y, z): cells x * kImclCells .. of rows y * seg_rows .. +
 * seg_rows - 1 of color z.  A row's next tiles are loaded while the row before
 * is written. */
__global__ void __launch_bounds__(kImclThreads, kImclBlocksPerSm) k_imclt_rbg_all(
    Geom g, const float *__restrict__ clt, float *__restrict__ rbg, size_t dstride, int seg_rows)
{
    __shared__ __align__(16) float tiles[2][kImclTiles][kXb];
    const int tid = threadIdx.x, l = tid & 7, grp = tid >> 3;
    const unsigned gm = group_mask();
    const int color = blockIdx.z, cx0 = blockIdx.x * kImclCells;
    const int cy0 = blockIdx.y * seg_rows, cy1 = min(cy0 + seg_rows, g.TY + 1);
    if (cy0 >= cy1) return;
    float *plane = rbg + dstride * (size_t)(g.H + 8) * color;
    /* this group's tile column and, for the output, this thread's pixel column */
    const int tx = cx0 - 1 + grp;
    const bool col_ok = tx >= 0 && tx < g.TX;
    const float *src = clt + ((size_t)(col_ok ? tx : 0) * 3 + color) * 256;
    const size_t row_step = (size_t)g.TX * 768;
    const int cell = tid >> 3, cx = cx0 + cell, c = tid & 7;
    const bool out_ok = cell < kImclCells && cx <= g.TX;
    /* the even and the odd tile column over this cell: its slot, the pixel's
     * column in it, and whether it exists */
    const int te = cx & 1 ? cx - 1 : cx, to = cx & 1 ? cx : cx - 1;
    const bool e_ok = te >= 0 && te < g.TX, o_ok = to >= 0 && to < g.TX;
    const int ce = cx & 1 ? c + 8 : c, co = cx & 1 ? c : c + 8;
    const float we = 0.5f * __ldg(&d_hwin[ce]), wo = 0.5f * __ldg(&d_hwin[co]);

    float raw[4][8];
    int ty = cy0 - 1;
    bool have = col_ok && ty >= 0;
    if (have) load_clt_rows<true>(src + (size_t)ty * row_step, raw, l);
    for (; ty < cy1; ty++) {
        if (have) imclt_tile(raw, tiles[ty & 1][grp], l, gm);
        have = col_ok && ty + 1 < cy1 && ty + 1 < g.TY;
        if (have) load_clt_rows<true>(src + (size_t)(ty + 1) * row_step, raw, l);
        __syncthreads();
        if (ty >= cy0 && out_ok) {
            /* cell row ty: the lower half of tile row ty - 1, the upper of ty */
            float *px = plane + (size_t)ty * 8 * dstride + (size_t)cx * 8 + c;
            const int rows[2] = {ty & 1 ? ty - 1 : ty, ty & 1 ? ty : ty - 1}; /* even, odd */
            const bool covered = rows[0] >= 0 && rows[0] < g.TY && e_ok;      /* by pass (0, 0) */
#pragma unroll
            for (int rp = 0; rp < 4; rp++) {
                float2 v = make_float2(0.0f, 0.0f);
                if (!covered)
                    v = make_float2(px[(size_t)(2 * rp) * dstride], px[(size_t)(2 * rp + 1) * dstride]);
#pragma unroll
                for (int vp = 0; vp < 2; vp++) {
                    const int row = rows[vp], rl = row == ty ? rp : rp + 4; /* row pair in that tile */
                    if (row < 0 || row >= g.TY) continue;
                    const float2 wr = make_float2(0.5f * c_hwin[2 * rl], 0.5f * c_hwin[2 * rl + 1]);
#pragma unroll
                    for (int hp = 0; hp < 2; hp++) {
                        if (!(hp ? o_ok : e_ok)) continue;
                        const int t = hp ? to : te;
                        const float2 d = reinterpret_cast<const float2 *>(
                            tiles[row & 1][t - cx0 + 1])[JT2(rl, hp ? co : ce)];
                        v = fma2_rd(mul2(wr, dup2(hp ? wo : we)), d, v);
                        if (g.debug_marks) {
                            if (t == 0 && row == 0) v = dup2(100.0f);
                            else if (t == 161 && row == 111) v = mul2(v, dup2(2.0f));
                        }
                    }
                }
                px[(size_t)(2 * rp) * dstride] = v.x;
                px[(size_t)(2 * rp + 1) * dstride] = v.y;
            }
        }
        __syncthreads(); /* the older tile row's slots free */
    }
}

} /* namespace tp */

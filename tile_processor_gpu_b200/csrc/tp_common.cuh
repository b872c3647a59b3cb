/*
 * tp_common.cuh - shared device code of the B200 tile processor.
 *
 * Work decomposition used by every kernel: one 8x8 transform job (one tile,
 * camera and color) is owned by a group of 8 consecutive lanes of a warp.
 * Lane l of the group holds one row or one column of each 8x8 quadrant in
 * registers, so the 8-point transforms along the held direction are
 * butterflies in registers (dct4_fast, dct2_fast); the other direction goes
 * through one 8x9 shared-memory
 * transpose per quadrant, padded so that both the row writes and the column
 * reads are bank-conflict free.  Groups never wait on each other: the only
 * synchronisation is __syncwarp on the group's 8-lane mask, so a block has no
 * block-wide barrier and groups of a warp may take different paths.
 */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/tp_b200.h"
#include "tp_tables.inc"

namespace tp {

/* ---- constant tables (generated by gen_tables.py) -------------------------- */
__device__ __constant__ float c_hwin[16] = TP_HWIN_INIT;
/* Tables that lanes index by their own row / column live in global memory
 * and are read through the read-only data cache: the lanes of a warp then
 * fetch distinct words in one pass, where the constant cache would serialise
 * them.  Runtime-settable low-pass filters: lpf_data[0..3], lpf_rb_corr,
 * lpf_corr. */
__device__ __align__(32) float d_lpf[6][64] = TP_LPF_DEFAULT_INIT;
__device__ float d_alpha_fade[16][256] = TP_ALPHA_FADE_INIT;
__device__ float d_hwin[16] = TP_HWIN_INIT;
__device__ float d_hwinc[16] = TP_HWINC_INIT;
/* camera pairs (src/TileProcessor.cuh:484-490) */
__device__ __constant__ int c_pairs[6][2] = {{0, 1}, {2, 3}, {0, 2}, {1, 3}, {0, 3}, {2, 1}};

/* Geometry as kernels see it. */
struct Geom {
    int W, H;        /* image size                                  */
    int TX, TY, TYA; /* tiles                                       */
    int KH, KV, ls;  /* kernel table grid and log2 step             */
    int image_rows;  /* rows allocated per source image             */
    int border_mode;
    int debug_marks;
};

__device__ __forceinline__ unsigned group_mask() { return 0xffu << (threadIdx.x & 24); }

/* Asynchronous global -> shared copies (LDGSTS).  Completion is awaited with
 * cp_async_wait_all() by the issuing thread; other threads see the data after
 * a following block barrier. */
__device__ __forceinline__ void cp_async4(void *sdst, const void *gsrc)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

/* Programmatic dependent launch.  A kernel launched with programmatic stream
 * serialisation may start while the launch before it on the stream is still
 * running: grid_dependency_wait() blocks the calling thread until that grid
 * has completed and its memory operations are visible (a no-op for an
 * ordinary launch), and grid_dependents_launch() lets such a dependent grid
 * be scheduled once every block of this grid has issued it. */
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

/* 8-point DCT-IV (SINE false) or DST-IV (SINE true) with the tables' scale,
 * y[k] = 0.5 sum_n x[n] cos|sin(pi (2k+1)(2n+1) / 32), through a 4-point
 * complex transform: with a_m = x[2m], b_m = x[7-2m] (swapped for the sine,
 * as DST-IV x = (-1)^k DCT-IV of x reversed), z_m = (a_m - i b_m)
 * e^{i pi m / 8}, Z_p = sum_m z_m i^{mp} and Y_p = 0.5 e^{i pi (4p+1) / 32}
 * Z_p: y[2p] = Re Y_p, y[7-2p] = Im Y_p (negated for the sine).  44
 * operations against the 64 multiply-adds of the matrix product. */
template <bool SINE>
__host__ __device__ __forceinline__ void dct4_fast(const float x[8], float y[8])
{
    constexpr float pre[4][2] = TP_DCT4_PRE_INIT;
    constexpr float post[4][2] = TP_DCT4_POST_INIT;
    float zr[4], zi[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const float a = SINE ? x[7 - 2 * m] : x[2 * m];
        const float b = SINE ? x[2 * m] : x[7 - 2 * m];
        if (m == 0) {
            zr[0] = a;
            zi[0] = -b;
        } else {
            zr[m] = fmaf(a, pre[m][0], b * pre[m][1]);
            zi[m] = fmaf(a, pre[m][1], -(b * pre[m][0]));
        }
    }
    const float s02r = zr[0] + zr[2], s02i = zi[0] + zi[2], d02r = zr[0] - zr[2], d02i = zi[0] - zi[2];
    const float s13r = zr[1] + zr[3], s13i = zi[1] + zi[3], d13r = zr[1] - zr[3], d13i = zi[1] - zi[3];
    const float Zr[4] = {s02r + s13r, d02r - d13i, s02r - s13r, d02r + d13i};
    const float Zi[4] = {s02i + s13i, d02i + d13r, s02i - s13i, d02i - d13r};
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const float yr = fmaf(Zr[p], post[p][0], -(Zi[p] * post[p][1]));
        const float yi = fmaf(Zr[p], post[p][1], Zi[p] * post[p][0]);
        y[2 * p] = yr;
        y[7 - 2 * p] = SINE ? -yi : yi;
    }
}

/* 8-point DCT-II (SINE false) or DST-II (SINE true) with the tables' scale,
 * y[k] = 0.5 sum_n x[n] cos(pi (2n+1) k / 16) | sin(pi (2n+1) (k+1) / 16):
 * the even outputs are the 4-point DCT-II of u_n = x_n + x_{7-n}, the odd
 * ones the 4-point DCT-IV of v_n = x_n - x_{7-n} (through a 2-point complex
 * transform, as in dct4_fast); the DST-II is the DCT-II of (-1)^n x_n with
 * the outputs in reverse order.  36 operations against 64. */
template <bool SINE>
__host__ __device__ __forceinline__ void dct2_fast(const float xin[8], float y[8])
{
    constexpr float K[8] = TP_DCT2_FAST_INIT;
    float x[8];
#pragma unroll
    for (int n = 0; n < 8; n++) x[n] = (SINE && (n & 1)) ? -xin[n] : xin[n];
    const float u0 = x[0] + x[7], u1 = x[1] + x[6], u2 = x[2] + x[5], u3 = x[3] + x[4];
    const float v0 = x[0] - x[7], v1 = x[1] - x[6], v2 = x[2] - x[5], v3 = x[3] - x[4];
    const float w0 = u0 + u3, w1 = u1 + u2, d0 = u0 - u3, d1 = u1 - u2;
    float r[8];
    r[0] = 0.5f * (w0 + w1);
    r[4] = K[0] * (w0 - w1);
    r[2] = fmaf(d0, K[1], d1 * K[2]);
    r[6] = fmaf(d0, K[2], -(d1 * K[1]));
    /* 4-point DCT-IV of v: z0 = v0 - i v3, z1 = (v2 - i v1) e^{i pi / 4} */
    const float z1r = K[3] * (v2 + v1), z1i = K[3] * (v2 - v1);
    const float p0r = v0 + z1r, p0i = z1i - v3; /* Z_0 = z0 + z1 */
    const float p1r = v0 - z1r, p1i = -v3 - z1i; /* Z_1 = z0 - z1 */
    r[1] = fmaf(p0r, K[4], -(p0i * K[5]));
    r[7] = fmaf(p0r, K[5], p0i * K[4]);
    r[5] = fmaf(p1r, K[6], -(p1i * K[7]));
    r[3] = fmaf(p1r, K[7], p1i * K[6]);
#pragma unroll
    for (int k = 0; k < 8; k++) y[k] = SINE ? r[7 - k] : r[k];
}

/* Two independent FP32 values in one 64-bit register pair (add/mul/fma.f32x2:
 * one issue slot for two operations, each rounded as its scalar form).  The
 * stage kernels are bound by issue slots, not by the FP32 units, so their
 * transforms, stencils and camera fusion run on pairs. */
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
#if !defined(__CUDA_ARCH__) || __CUDA_ARCH__ >= 1000
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

/* dct4_fast on both halves of pairs: y[2p] = Re Y_p, y[7-2p] = Im Y_p.  A
 * DST-IV half takes its input in reverse order (x[7-n] at n) and leaves the
 * sign of its odd outputs to the caller, who carries it in a later factor;
 * one sequence then serves cosine and sine halves alike.  Bit-identical to
 * dct4_fast. */
__device__ __forceinline__ void dct4_pair(const float2 x[8], float2 y[8])
{
    constexpr float pre[4][2] = TP_DCT4_PRE_INIT;
    constexpr float post[4][2] = TP_DCT4_POST_INIT;
    float2 zr[4], zi[4];
    zr[0] = x[0];
#pragma unroll
    for (int m = 1; m < 4; m++) {
        const float2 a = x[2 * m], b = x[7 - 2 * m];
        zr[m] = fma2(a, dup2(pre[m][0]), mul2(b, dup2(pre[m][1])));
        zi[m] = fma2(a, dup2(pre[m][1]), mul2(b, dup2(-pre[m][0])));
    }
    const float2 b0 = x[7]; /* zi[0] = -b0 */
    const float2 s02r = add2(zr[0], zr[2]), d02r = sub2(zr[0], zr[2]);
    const float2 s02i = sub2(zi[2], b0), n02i = add2(b0, zi[2]); /* n02i = -d02i */
    const float2 s13r = add2(zr[1], zr[3]), d13r = sub2(zr[1], zr[3]);
    const float2 s13i = add2(zi[1], zi[3]), d13i = sub2(zi[1], zi[3]);
    const float2 Zr[4] = {add2(s02r, s13r), sub2(d02r, d13i), sub2(s02r, s13r), add2(d02r, d13i)};
    const float2 Zi[3] = {add2(s02i, s13i), sub2(d13r, n02i), sub2(s02i, s13i)};
    const float2 n3 = add2(n02i, d13r); /* -Z_3's imaginary part */
#pragma unroll
    for (int p = 0; p < 3; p++) {
        y[2 * p] = fma2(Zr[p], dup2(post[p][0]), mul2(Zi[p], dup2(-post[p][1])));
        y[7 - 2 * p] = fma2(Zr[p], dup2(post[p][1]), mul2(Zi[p], dup2(post[p][0])));
    }
    y[6] = fma2(Zr[3], dup2(post[3][0]), mul2(n3, dup2(post[3][1])));
    y[1] = fma2(Zr[3], dup2(post[3][1]), mul2(n3, dup2(-post[3][0])));
}

/* dct2_fast<false> on both halves of pairs.  A DST-II half takes its input
 * with alternating signs ((-1)^n x[n]) and finds its outputs in reverse order
 * (DST_k at 7-k).  Bit-identical to dct2_fast. */
__device__ __forceinline__ void dct2_pair(const float2 x[8], float2 r[8])
{
    constexpr float K[8] = TP_DCT2_FAST_INIT;
    const float2 u0 = add2(x[0], x[7]), u1 = add2(x[1], x[6]), u2 = add2(x[2], x[5]), u3 = add2(x[3], x[4]);
    const float2 v0 = sub2(x[0], x[7]), v1 = sub2(x[1], x[6]), v2 = sub2(x[2], x[5]), v3 = sub2(x[3], x[4]);
    const float2 w0 = add2(u0, u3), w1 = add2(u1, u2), d0 = sub2(u0, u3), d1 = sub2(u1, u2);
    r[0] = mul2(dup2(0.5f), add2(w0, w1));
    r[4] = mul2(dup2(K[0]), sub2(w0, w1));
    r[2] = fma2(d0, dup2(K[1]), mul2(d1, dup2(K[2])));
    r[6] = fma2(d0, dup2(K[2]), mul2(d1, dup2(-K[1])));
    const float2 z1r = mul2(dup2(K[3]), add2(v2, v1)), z1i = mul2(dup2(K[3]), sub2(v2, v1));
    const float2 p0r = add2(v0, z1r), p0i = sub2(z1i, v3);
    const float2 p1r = sub2(v0, z1r), n1i = add2(v3, z1i); /* n1i = -p1i */
    r[1] = fma2(p0r, dup2(K[4]), mul2(p0i, dup2(-K[5])));
    r[7] = fma2(p0r, dup2(K[5]), mul2(p0i, dup2(K[4])));
    r[5] = fma2(p1r, dup2(K[6]), mul2(n1i, dup2(K[7])));
    r[3] = fma2(p1r, dup2(K[7]), mul2(n1i, dup2(-K[6])));
}
#endif

/* 8 consecutive floats of shared memory (16-byte aligned) */
__device__ __forceinline__ void load_row8s(const float *p, float v[8])
{
    const float4 x = *reinterpret_cast<const float4 *>(p), y = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
}

/* 8 consecutive floats of global memory (32-byte aligned): one 256-bit access.  ld8_global is for rows that
   the SM reads once (CLT tiles of the textures and the inverse transform, deconvolution kernel rows): it leaves
   L1 to what is read again.  With plain loads the tensor-core inverse's tables were evicted by the tiles that
   pass: the three tensor-core stages of 1024x768 took 436 us in FP16, 418 this way; the RGBA image of 2592x1936
   611 and 608.  ld8_l1 is for the correlation, whose pairs share a tile's rows. */
__device__ __forceinline__ void ld8_global(const float *p, float v[8])
{
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld8_l1(const float *p, float v[8])
{
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void st8_global(float *p, const float v[8])
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

/* y[k] = sum_n M[k][n] x[n] for the four 8-point transforms of the tables:
 * DCT-IV / DST-IV (KIND 0 / 1) through dct4_fast, DCT-II / DST-II (KIND 2 /
 * 3) through dct2_fast */
template <int KIND>
__device__ __forceinline__ void dtt8(const float x[8], float y[8])
{
    if constexpr (KIND == 0 || KIND == 1)
        dct4_fast<KIND == 1>(x, y);
    else
        dct2_fast<KIND == 3>(x, y);
}

/* window sample n -> DTT index (4..7, 7..4, 3..0, 0..3) and back: the two
 * samples that fold onto index u have opposite parity; return the one with
 * parity p. */
__device__ __forceinline__ int fold_sample(int u, int p)
{
    int a = (u >= 4) ? u - 4 : 11 - u;
    int b = (u >= 4) ? 11 - u : 12 + u;
    return ((a & 1) == p) ? a : b;
}

/* window value w(n + s) = sin(pi (2 (n + s) + 1) / 32) from (cos, sin)(pi s / 16) */
__device__ __forceinline__ float shifted_window_lane(int n, float cs, float sn)
{
    return __fmaf_rn(__ldg(&d_hwin[n]), cs, __ldg(&d_hwinc[n]) * sn);
}

/* Workspace of a frame in stages (process_frame): the CLT of the tasks at hand by their
 * place in the task list, [task][camera][colour][256], and their texture lists
 * by tile parity (task, texture list code), written by the forward transform. */
struct FrameSlots {
    float *clt;
    int2 *list;  /* [4][tasks] */
    int *counts; /* [4]        */
};
constexpr int kSlot = 4 * 3 * 256;

} /* namespace tp */

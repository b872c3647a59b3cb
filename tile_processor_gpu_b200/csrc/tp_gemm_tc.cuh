/*
 * tp_gemm_tc.cuh - the learned residual's training GEMM on the tensor cores:
 * C = op(A) op(B) (+ bias, + beta C, optional pre-activation z and GELU), the
 * operation of k_gemm, with FP32 operands split into two TF32 parts,
 *   x = hi + lo,  hi = tf32(x),  lo = x - hi (the MMA reads its TF32 bits),
 * and each product formed as three tcgen05 TF32 MMAs, A_hi B_hi + A_hi B_lo +
 * A_lo B_hi (about 21 significant bits per operand; the dropped A_lo B_lo
 * term is below 2^-21 of a product).  Each K chunk of 32 is accumulated in
 * its own tensor-memory buffer and added into FP32 registers: one
 * accumulator over all of K (169 MMA steps for K = 1350, sums up to ~170
 * times a product) loses about 1e-5 of the result, the per-chunk sums stay
 * within 2e-6.
 *
 * One CTA per 128 x 64 tile of C (and K range), K in chunks of 32, 17 warps in
 * three roles around four stages of shared memory and of tensor memory:
 *   producers (eight warps): unit = one row's four consecutive K values, loaded
 *     in the order that is contiguous for the operand's transpose (16- or
 *     8-byte loads where the rows allow them, two chunks ahead), split, and
 *     stored as one 16-byte piece each of the hi and the lo K-major
 *     128-byte-swizzled image (rows of 32 values, the piece index XOR the row's
 *     low three bits: conflict-free in either order); they arrive on full[s];
 *   the MMA warp: one thread waits for full[s] and for the stage's accumulator,
 *     issues the chunk's 12 MMAs (four K steps of 8) and commits them to
 *     done[s], which frees the images and hands over the accumulator;
 *   gather (eight warps, half a row of C per thread): add the chunk's 32 columns
 *     into 32 registers, one tensor-memory load and wait a chunk, and release
 *     the accumulator (accfree[s]).
 * At the end the tile goes through shared memory and all warps apply bias,
 * beta C, GELU, or (dgelu) the factor gelu'(z), row by row; the tile's column
 * sums, where they are wanted, go out as one part a tile (k_head_sums adds them).
 * What bounds it is shared memory: a chunk's split images are 48 KB written and
 * 72 KB read by the MMAs (N = 64 reads A once per MMA), beside about 10 us of
 * launch, first loads and epilogue.  The earlier form did every step of a chunk
 * in turn with four warps, and GELU on one row per thread: layer 1's forward
 * product at 4096 rows (4096 x 256 x 1350) took 230 us (ncu, cold cache) and now
 * 55 (44 warm), its weight gradient 160 and now 51.  Tried without gain:
 * sixteen producer warps, four chunks in flight (spills), two producer groups
 * on alternate chunks.
 *
 * Every wait is bounded; one that runs out raises the CTA's abort flag, every
 * role leaves its loop, the issued MMAs are drained (one more bounded wait),
 * the tensor memory is freed, *err is set and C is left unwritten.
 */
#pragma once
#include "tp_tc_engine.cuh"
#include "tp_tcgen05.cuh"

namespace tp {

constexpr int kGtM = 128, kGtN = 64, kGtK = 32;
constexpr int kGtABytes = kGtM * kGtK * 4; /* one TF32 part of the A chunk: 16 KB */
constexpr int kGtBBytes = kGtN * kGtK * 4; /* one TF32 part of the B chunk: 8 KB  */
constexpr int kGtStageBytes = 2 * kGtABytes + 2 * kGtBBytes;
constexpr int kGtStages = 4;
constexpr int kGtProdWarps = 8, kGtProd = 32 * kGtProdWarps;
constexpr int kGtGatherWarps = 8;
constexpr int kGtThreads = 32 * (kGtGatherWarps + 1 + kGtProdWarps);
constexpr size_t kGtSmemBytes = (size_t)kGtStages * kGtStageBytes + 1024; /* + alignment of the swizzle atoms */
static_assert(kGtABytes % 1024 == 0 && kGtBBytes % 1024 == 0, "images start on 1024-byte swizzle atoms");
static_assert(kGtStages * kGtN <= 512, "an accumulator per stage");

/* An operand of the GEMM as a rows x K matrix: element (r, k) at p[r * ld + k],
 * or p[k * ld + r] when `across`.  vec: floats of a row that one load may take
 * (4, 2 or 1; 1 when across). */
struct GtOperand {
    const float *p;
    int ld, rows, across, vec;
};

/* What happens to the finished tile.  dgelu: C = acc * gelu'(z), and
 * colsum[N m + n] (unless NULL) = the sum of column n of the m-th 128 rows of C;
 * else C = beta C + acc + bias, with z (if given) that value and C = gelu of it. */
struct GtEpilogue {
    float beta;
    float *C;
    int ldc;
    const float *bias;
    float *z;
    int ldz;
    int dgelu;
    float *colsum;
};

/* A producer thread's N units of an operand: row r, K values 4q .. 4q + 3 of
 * each chunk, r and q from the thread's and the unit's number in the order that
 * is contiguous in memory.  Rows past the operand's last read that row again
 * (they end in rows or columns of the tile that nobody stores); K past the end
 * gives zeros.  Chunks are loaded one after another (load moves on). */
template <bool ACROSS, int ROWS, int N>
struct GtUnits {
    const float *p[N]; /* the unit's first value of the next chunk */
    uint32_t off[N];   /* its piece in an image */
    int ld;
    __device__ __forceinline__ static int row(int t, int u) { return ACROSS ? (t + kGtProd * u) % ROWS : (t + kGtProd * u) >> 3; }
    __device__ __forceinline__ static int piece(int t, int u) { return ACROSS ? (t + kGtProd * u) / ROWS : t & 7; }
    __device__ __forceinline__ GtUnits(const GtOperand &o, int r0, int k0, int t) : ld(o.ld)
    {
#pragma unroll
        for (int u = 0; u < N; u++) {
            const int r = row(t, u), q = piece(t, u);
            const size_t m = (size_t)min(r0 + r, o.rows - 1), k = (size_t)(k0 + 4 * q);
            p[u] = o.p + (ACROSS ? k * o.ld + m : m * o.ld + k);
            off[u] = (uint32_t)(r * 128 + ((q ^ (r & 7)) << 4));
        }
    }
    /* the next chunk, which starts at k0 and (left >= 32) lies inside K or has
     * `left` values left */
    __device__ __forceinline__ void load(int vec, int left, int t, float v[N][4])
    {
        if (left < kGtK) {
#pragma unroll
            for (int u = 0; u < N; u++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    v[u][j] = 4 * piece(t, u) + j < left ? __ldg(p[u] + (ACROSS ? (size_t)j * ld : (size_t)j)) : 0.0f;
        } else if (ACROSS) {
#pragma unroll
            for (int u = 0; u < N; u++)
#pragma unroll
                for (int j = 0; j < 4; j++) v[u][j] = __ldg(p[u] + (size_t)j * ld);
        } else if (vec == 4) {
#pragma unroll
            for (int u = 0; u < N; u++) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(p[u]));
                v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w;
            }
        } else if (vec == 2) {
#pragma unroll
            for (int u = 0; u < N; u++) {
                const float2 x = __ldg(reinterpret_cast<const float2 *>(p[u]));
                const float2 y = __ldg(reinterpret_cast<const float2 *>(p[u]) + 1);
                v[u][0] = x.x; v[u][1] = x.y; v[u][2] = y.x; v[u][3] = y.y;
            }
        } else {
#pragma unroll
            for (int u = 0; u < N; u++)
#pragma unroll
                for (int j = 0; j < 4; j++) v[u][j] = __ldg(p[u] + j);
        }
#pragma unroll
        for (int u = 0; u < N; u++) p[u] += ACROSS ? (size_t)kGtK * ld : (size_t)kGtK;
    }
};

/* Four K values as a hi and a lo piece.  hi is x rounded to TF32 (to nearest,
 * ties away, as cvt.rna.tf32, which takes four integer operations a value): the
 * bits plus half a TF32 ulp, truncated.  A NaN whose payload that carry would
 * turn into a zero still reaches the result through lo = x - hi.  lo, a
 * multiple of x's ulp below 2^12 of them, is stored as it is: the tensor core
 * reads its upper 11 bits, which drops at most the one ulp that rounding it
 * would move it by. */
__device__ __forceinline__ void gt_put4(unsigned char *hi, unsigned char *lo, const float v[4])
{
    float h[4];
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __uint_as_float((__float_as_uint(v[i]) + 0x1000u) & 0xffffe000u);
    *reinterpret_cast<float4 *>(hi) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4 *>(lo) = make_float4(v[0] - h[0], v[1] - h[1], v[2] - h[2], v[3] - h[3]);
}

/* TA, TB: the operands' `across` */
template <bool TA, bool TB>
__global__ void __launch_bounds__(kGtThreads, 1) k_gemm_tc(int K, GtOperand A, GtOperand B, GtEpilogue e,
                                                           int *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char gt_smem[];
    enum { kFull = 0, kDone = kGtStages, kAccFree = 2 * kGtStages, kDrain = 3 * kGtStages, kBars };
    __shared__ __align__(8) uint64_t bars[kBars];
    __shared__ uint32_t tmem_slot;
    __shared__ int flag_store; /* abort */
    volatile int *abort_flag = &flag_store;
    const uint32_t base_s = (uint32_t)__cvta_generic_to_shared(gt_smem);
    const uint32_t pad = (1024 - (base_s & 1023)) & 1023;
    unsigned char *sm = gt_smem + pad;
    const uint32_t a_sm = base_s + pad;
    const uint32_t a_bar = (uint32_t)__cvta_generic_to_shared(bars);
    auto bar = [&](int b) { return a_bar + 8u * (uint32_t)b; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * kGtM, n0 = blockIdx.x * kGtN;
    const bool gather = warp < kGtGatherWarps, issuer = tid == 32 * kGtGatherWarps;
    constexpr int kHalf = kGtN / 2; /* columns of a gather warp: half warp / 4 of lanes 32 (warp % 4) .. */

    if (issuer) {
        for (int b = 0; b < kBars; b++) {
            const uint32_t count = b < kDone ? (uint32_t)kGtProdWarps : (b >= kAccFree && b < kDrain) ? (uint32_t)kGtGatherWarps : 1u;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(b)), "r"(count) : "memory");
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kGtGatherWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&tmem_slot)),
                     "n"(kGtStages * kGtN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    /* this CTA's chunks: the K range blockIdx.z of gridDim.z (several only
     * for a plain product into a zeroed C, see gemm_tc_launch) */
    const int nch = (K + kGtK - 1) / kGtK;
    const int per = (nch + (int)gridDim.z - 1) / (int)gridDim.z;
    const int c_begin = min(nch, (int)blockIdx.z * per);
    const int nloc = min(nch, c_begin + per) - c_begin;
    bool issued = false; /* issuer: MMAs in flight or done */
    float acc[kHalf];    /* gather: this thread's half row of the tile */

    if (gather) {
#pragma unroll
        for (int i = 0; i < kHalf; i++) acc[i] = 0.0f;
        const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * kHalf);
        for (int i = 0; i < nloc; i++) {
            const int s = i % kGtStages;
            const bool ok = tc_wait_or_abort(bar(kDone + s), (uint32_t)((i / kGtStages) & 1), abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float v[kHalf];
            tc_ld32(t_lane + (uint32_t)(s * kGtN), v);
#pragma unroll
            for (int j = 0; j < kHalf; j++) acc[j] += v[j];
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(bar(kAccFree + s));
        }
    } else if (warp == kGtGatherWarps) {
        if (issuer) {
            const uint32_t idesc = tc_idesc(kGtM, kGtN, 2u);
            for (int i = 0; i < nloc; i++) {
                const int s = i % kGtStages;
                const uint32_t ph = (uint32_t)((i / kGtStages) & 1);
                bool ok = tc_wait_or_abort(bar(kFull + s), ph, abort_flag);
                if (ok && i >= kGtStages) ok = tc_wait_or_abort(bar(kAccFree + s), ph ^ 1u, abort_flag);
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ahi = a_sm + (uint32_t)(s * kGtStageBytes), alo = ahi + kGtABytes;
                const uint32_t bhi = alo + kGtABytes, blo = bhi + kGtBBytes;
                const uint32_t d = tmem + (uint32_t)(s * kGtN);
#pragma unroll
                for (int j = 0; j < kGtK / 8; j++) {
                    const uint32_t o = 32u * j;
                    tc_mma_tf32(d, tc_desc_sw128(ahi + o), tc_desc_sw128(bhi + o), idesc, j > 0 ? 1u : 0u);
                    tc_mma_tf32(d, tc_desc_sw128(ahi + o), tc_desc_sw128(blo + o), idesc, 1u);
                    tc_mma_tf32(d, tc_desc_sw128(alo + o), tc_desc_sw128(bhi + o), idesc, 1u);
                }
                tc_commit(bar(kDone + s));
                issued = true;
            }
        }
        __syncwarp();
    } else {
        const int t = tid - 32 * (kGtGatherWarps + 1);
        constexpr int kAU = kGtM * 8 / kGtProd, kBU = kGtN * 8 / kGtProd; /* units per thread: 4 and 2 */
        const int kc = c_begin * kGtK;
        GtUnits<TA, kGtM, kAU> au(A, m0, kc, t);
        GtUnits<TB, kGtN, kBU> bu(B, n0, kc, t);
        auto load = [&](int i, float ra[kAU][4], float rb[kBU][4]) {
            if (i >= nloc) return;
            const int left = K - kc - i * kGtK;
            au.load(A.vec, left, t, ra);
            bu.load(B.vec, left, t, rb);
        };
        /* chunk i into its stage; false: a wait ran out */
        auto store = [&](int i, const float ra[kAU][4], const float rb[kBU][4]) -> bool {
            const int s = i % kGtStages;
            if (i >= kGtStages) {
                /* the MMAs of the stage's last chunk have read its images */
                const bool ok = tc_wait_or_abort(bar(kDone + s), (uint32_t)((i / kGtStages - 1) & 1), abort_flag);
                if (!__all_sync(0xffffffffu, ok)) {
                    *abort_flag = 1;
                    return false;
                }
            }
            unsigned char *ahi = sm + (size_t)s * kGtStageBytes, *alo = ahi + kGtABytes;
            unsigned char *bhi = alo + kGtABytes, *blo = bhi + kGtBBytes;
#pragma unroll
            for (int u = 0; u < kAU; u++) gt_put4(ahi + au.off[u], alo + au.off[u], ra[u]);
#pragma unroll
            for (int u = 0; u < kBU; u++) gt_put4(bhi + bu.off[u], blo + bu.off[u], rb[u]);
            /* the generic-proxy stores visible to the tensor cores' reads */
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(bar(kFull + s));
            return true;
        };
        float ra0[kAU][4], rb0[kBU][4], ra1[kAU][4], rb1[kBU][4];
        load(0, ra0, rb0);
        load(1, ra1, rb1);
        for (int i = 0; i < nloc; i += 2) {
            if (!store(i, ra0, rb0)) break;
            load(i + 2, ra0, rb0);
            if (i + 1 >= nloc || !store(i + 1, ra1, rb1)) break;
            load(i + 3, ra1, rb1);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool failed = *abort_flag != 0;
    if (issuer && failed) {
        /* MMAs issued so far complete before the tensor memory is freed */
        if (issued) {
            tc_commit(bar(kDrain));
            (void)tc_wait(bar(kDrain), 0u);
        }
        if (err) atomicExch(err, 1);
    }
    /* the tile through shared memory (every MMA has read its stage), so that all
     * warps share the epilogue and its accesses of C and z are whole rows */
    float(*tile)[kGtN + 1] = reinterpret_cast<float(*)[kGtN + 1]>(sm);
    static_assert(kGtM * (kGtN + 1) * 4 <= kGtStages * kGtStageBytes, "the tile fits the stages");
    if (gather && !failed) {
#pragma unroll
        for (int i = 0; i < kHalf; i++) tile[(warp & 3) * 32 + lane][(warp >> 2) * kHalf + i] = acc[i];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == kGtGatherWarps)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kGtStages * kGtN)
                     : "memory");
    if (failed) return;
    const int mrows = min(kGtM, A.rows - m0), ncols = min(kGtN, B.rows - n0);
#pragma unroll 2
    for (int x = tid; x < kGtM * kGtN; x += kGtThreads) {
        const int r = x / kGtN, n = x % kGtN;
        if (r >= mrows || n >= ncols) continue;
        const size_t gm = (size_t)(m0 + r), gn = (size_t)(n0 + n);
        float *c = e.C + gm * e.ldc + gn;
        float v = tile[r][n];
        if (gridDim.z > 1) { /* one of several K ranges: its partial sum into the zeroed C */
            atomicAdd(c, v);
            continue;
        }
        if (e.dgelu) {
            v *= gelu_grad_f(e.z[gm * e.ldz + gn]);
            tile[r][n] = v;
        } else {
            if (e.bias) v += e.bias[gn];
            if (e.beta != 0.0f) v = __fmaf_rn(e.beta, *c, v);
            if (e.z) {
                e.z[gm * e.ldz + gn] = v;
                v = gelu_f(v);
            }
        }
        *c = v;
    }
    if (e.dgelu && e.colsum) {
        /* eight partial sums a column, added in their order */
        constexpr int kParts = kGtThreads / kGtN;
        float(*part)[kGtN] = reinterpret_cast<float(*)[kGtN]>(sm + kGtM * (kGtN + 1) * 4);
        static_assert((kGtM * (kGtN + 1) + kParts * kGtN) * 4 <= kGtStages * kGtStageBytes, "and their sums");
        __syncthreads();
        const int n = tid % kGtN, first = tid / kGtN;
        if (first < kParts) {
            float sum = 0.0f;
            for (int r = first; r < mrows; r += kParts) sum += tile[r][n];
            part[first][n] = sum;
        }
        __syncthreads();
        if (tid < ncols) {
            float sum = part[0][tid];
#pragma unroll
            for (int i = 1; i < kParts; i++) sum += part[i][tid];
            e.colsum[(size_t)blockIdx.y * B.rows + n0 + tid] = sum;
        }
    }
}

/* ---- the network's head and bookkeeping ------------------------------------- */

/* out[r] = h2[r] W3 + b3: a warp per row of 128, lane l the values 4l .. 4l + 3 */
__global__ void __launch_bounds__(256) k_head_forward(int rows, const float *__restrict__ h2,
                                                      const float *__restrict__ W3, const float *__restrict__ b3,
                                                      float *__restrict__ out)
{
    const int lane = threadIdx.x & 31;
    float w0[4], w1[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        w0[i] = __ldg(W3 + 2 * (4 * lane + i));
        w1[i] = __ldg(W3 + 2 * (4 * lane + i) + 1);
    }
    const float bias0 = __ldg(b3), bias1 = __ldg(b3 + 1);
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
        const float4 h = __ldg(reinterpret_cast<const float4 *>(h2 + (size_t)r * 128) + lane);
        float o0 = h.x * w0[0], o1 = h.x * w1[0];
        o0 = __fmaf_rn(h.y, w0[1], o0); o1 = __fmaf_rn(h.y, w1[1], o1);
        o0 = __fmaf_rn(h.z, w0[2], o0); o1 = __fmaf_rn(h.z, w1[2], o1);
        o0 = __fmaf_rn(h.w, w0[3], o0); o1 = __fmaf_rn(h.w, w1[3], o1);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            o0 += __shfl_xor_sync(0xffffffffu, o0, d);
            o1 += __shfl_xor_sync(0xffffffffu, o1, d);
        }
        if (lane == 0) *reinterpret_cast<float2 *>(out + 2 * (size_t)r) = make_float2(o0 + bias0, o1 + bias1);
    }
}

/* The loss and everything of the backward pass that is per row of the head, on
 * `chunks` times kHeadRows rows a block, thread c = column c of layer 2: the loss
 * and its gradient dout (k_nll), dz2 = (dout W3^T) gelu'(z2), and this block's
 * part of the gradients of b2 (128), W3 (256) and b3 (2) at part[block], which
 * k_head_sums adds in a fixed order.  The grid's blocks, those past the last row
 * too, zero what the products of the weight gradients add into: zero0 .. zero0 +
 * n0 and zero1 .. zero1 + n1. */
constexpr int kHeadRows = 16, kHeadPart = 128 + 256 + 2;
__global__ void __launch_bounds__(128) k_head_backward(int rows, int chunks, const float *__restrict__ out,
                                                       const float *__restrict__ target, const float *__restrict__ w,
                                                       float inv_count, const float *__restrict__ h2,
                                                       const float *__restrict__ z2, const float *__restrict__ W3,
                                                       float *__restrict__ dout, float *__restrict__ loss_rows,
                                                       float *__restrict__ dz2, float *__restrict__ part, float *zero0,
                                                       int n0, float *zero1, int n1)
{
    __shared__ float s_d[kHeadRows][2];
    const int c = threadIdx.x;
    for (int i = blockIdx.x * 128 + c; i < n0; i += gridDim.x * 128) zero0[i] = 0.0f;
    for (int i = blockIdx.x * 128 + c; i < n1; i += gridDim.x * 128) zero1[i] = 0.0f;
    if (blockIdx.x * chunks * kHeadRows >= rows) return;
    const float w0 = __ldg(W3 + 2 * c), w1 = __ldg(W3 + 2 * c + 1);
    float sb = 0.0f, s0 = 0.0f, s1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
    for (int k = 0; k < chunks; k++) {
        const int r0 = (blockIdx.x * chunks + k) * kHeadRows, nr = min(kHeadRows, rows - r0);
        if (nr <= 0) break;
        float z[kHeadRows], h[kHeadRows];
#pragma unroll
        for (int i = 0; i < kHeadRows; i++) {
            const size_t o = (size_t)(r0 + min(i, nr - 1)) * 128 + c;
            z[i] = __ldg(z2 + o);
            h[i] = __ldg(h2 + o);
        }
        if (k) __syncthreads(); /* the chunk before has been read */
        if (c < 32) {
            float loss = 0.0f, d0 = 0.0f, d1 = 0.0f;
            if (c < nr) {
                nll_row(r0 + c, out, target, w, inv_count, &loss, &d0, &d1);
                loss_rows[r0 + c] = loss;
                *reinterpret_cast<float2 *>(dout + 2 * (size_t)(r0 + c)) = make_float2(d0, d1);
                s_d[c][0] = d0;
                s_d[c][1] = d1;
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                d0 += __shfl_xor_sync(0xffffffffu, d0, d);
                d1 += __shfl_xor_sync(0xffffffffu, d1, d);
            }
            b0 += d0;
            b1 += d1;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kHeadRows; i++) {
            if (i >= nr) break;
            const float d0 = s_d[i][0], d1 = s_d[i][1];
            const float g = __fmaf_rn(d1, w1, d0 * w0) * gelu_grad_f(z[i]);
            dz2[(size_t)(r0 + i) * 128 + c] = g;
            sb += g;
            s0 = __fmaf_rn(h[i], d0, s0);
            s1 = __fmaf_rn(h[i], d1, s1);
        }
    }
    float *p = part + (size_t)blockIdx.x * kHeadPart;
    p[c] = sb;
    p[128 + 2 * c] = s0;
    p[128 + 2 * c + 1] = s1;
    if (c == 0) {
        p[384] = b0;
        p[385] = b1;
    }
}

/* The sums over blocks, each in a fixed order (kSumLanes threads a column, then
 * a tree), so that a step's gradients repeat bit for bit: column n < kHeadPart of
 * the nparts rows of k_head_backward to gb2, gW3, gb3; column n - kHeadPart of
 * ncols1 rows of 256 (the GEMM's column sums) to gb1; the last block adds the
 * rows' losses in double.  What it has read of `part` (the memory of a gradient
 * that a product adds into next) it zeroes. */
constexpr int kSumLanes = 16, kSumCols = 32;
__global__ void __launch_bounds__(kSumCols *kSumLanes) k_head_sums(float *part, int nparts, float *cols1, int ncols1,
                                                                   int rows, const float *__restrict__ loss_rows,
                                                                   float *gb2, float *gW3, float *gb3, float *gb1,
                                                                   double *loss_sum)
{
    const int lane = threadIdx.x / kSumCols;
    if (blockIdx.x == gridDim.x - 1) {
        __shared__ double s_loss[kSumCols * kSumLanes];
        double s = 0.0;
        for (int r = threadIdx.x; r < rows; r += kSumCols * kSumLanes) s += (double)__ldg(loss_rows + r);
        s_loss[threadIdx.x] = s;
        for (int h = kSumCols * kSumLanes / 2; h > 0; h >>= 1) {
            __syncthreads();
            if (threadIdx.x < h) s_loss[threadIdx.x] += s_loss[threadIdx.x + h];
        }
        if (threadIdx.x == 0) *loss_sum = s_loss[0];
        return;
    }
    __shared__ float s_sum[kSumLanes][kSumCols];
    const int col = threadIdx.x % kSumCols, n = blockIdx.x * kSumCols + col, n1 = n - kHeadPart;
    float *src = n1 < 0 ? part + n : cols1 + n1;
    const int ld = n1 < 0 ? kHeadPart : 256, count = n1 < 0 ? nparts : n1 < 256 ? ncols1 : 0;
    float s = 0.0f;
    constexpr int kBatch = 8; /* values in flight */
    for (int i0 = lane; i0 < count; i0 += kBatch * kSumLanes) {
        float v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
            const int i = i0 + k * kSumLanes;
            v[k] = i < count ? src[(size_t)i * ld] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
            const int i = i0 + k * kSumLanes;
            s += v[k];
            if (i < count) src[(size_t)i * ld] = 0.0f;
        }
    }
    s_sum[lane][col] = s;
    for (int h = kSumLanes / 2; h > 0; h >>= 1) {
        __syncthreads();
        if (lane < h) s_sum[lane][col] += s_sum[lane + h][col];
    }
    if (lane == 0) {
        const float v = s_sum[0][col];
        if (n < 128)
            gb2[n] = v;
        else if (n < 384)
            gW3[n - 128] = v;
        else if (n < kHeadPart)
            gb3[n - 384] = v;
        else if (n1 < 256 && ncols1)
            gb1[n1] = v;
    }
}

/* up to kTensors arrays of a network in one launch */
constexpr int kTensors = 8;
struct TensorSet {
    float *p[kTensors];
    long long n[kTensors];
    int count;
};

/* k_adam on every array of a set: p, with its gradient, and its two moments */
__global__ void __launch_bounds__(256) k_adam_set(TensorSet p, TensorSet g, TensorSet m, TensorSet v, float lr,
                                                  float b1, float b2, float eps, float c1, float c2)
{
    const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (int i = 0; i < p.count; i++)
        for (long long k = first; k < p.n[i]; k += step) adam_element(p.p[i], g.p[i], m.p[i], v.p[i], k, lr, b1, b2, eps, c1, c2);
}

} /* namespace tp */

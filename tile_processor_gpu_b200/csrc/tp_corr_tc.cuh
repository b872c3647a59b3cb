/*
 * tp_corr_tc.cuh - pairwise phase correlation with the pixel-domain transform
 * on the tensor cores (the precision form of correlate2D,
 * src/TileProcessor.cuh:1176-1443).
 *
 * Same arithmetic as k_correlate2D up to the normalised, low-pass-filtered
 * CLT-domain product of a pair (correlateAccumulateTiles :2829-2890,
 * normalizeTileAmplitude :2915-2942); its four 8x8 quadrants then go through
 * the DCT-II / DST-II pairs of dttii_shared_mem_nonortho as four 64 x 64
 * GEMMs on the tensor cores (tp_tc_engine.cuh: split FP16 or BF16 operands,
 * FP32 accumulation), and corrUnfoldTile (:2950-3008) folds the pixel-domain
 * quadrants into the (2r+1)^2 output.
 *
 * Runs in the shared pipeline k_tc_stage (tp_tc_engine.cuh) over blocks of
 * 128 index entries: twelve producer warps, one 8-lane group per entry,
 * compute row l of the four accumulated quadrants and write them split into
 * the A image; four epilogue warps, one thread per entry, read the
 * pixel-domain quadrants row by row from tensor memory, unfold and store
 * them.
 *
 * The stage is bound by latency and by its stores: a 1024x768 frame took 0.136
 * ms (ncu) with every lane storing its own entry (a sector per lane and store)
 * and takes 0.085 with the rows of a warp's 32 entries staged and stored run by
 * run.
 *
 * FP16 rows are scaled by `up` (a power of two chosen by the host from the
 * final LPF's largest entry, which bounds the normalised product) so the hi
 * halves stay below 2^15; BF16 needs no scale.
 */
#pragma once
#include "tp_correlate.cuh"
#include "tp_tc_engine.cuh"

namespace tp {

/* The correlation as a tensor-core stage (k_tc_stage): rows are index
 * entries; twelve producer warps (the CLT products are the heavy part), four
 * epilogue warps (512 threads, at most 128 registers each). */
struct CorrTcStage {
    static constexpr int kQuads = 4, kProdWarps = 12, kEpiWarps = 4;
    static constexpr int kThreads = 32 * (kProdWarps + kEpiWarps);
    static constexpr int kMeta = 1;
    static constexpr int kGroupBuf = 0;
    static constexpr int kRowPair = 31; /* two output rows of an entry, padded to an odd pitch */
    static constexpr int kWarpBuf = 32 * kRowPair;
    static constexpr int kAStages = 1;
    Geom g;
    float *const *clt;
    int colors;
    float scale0, scale1, scale2, fat_zero;
    long long num;
    const int *idx;
    size_t stride;
    int radius;
    float *corrs;
    float up; /* FP16 row scale (a power of two); 1 for BF16 */

    __host__ __device__ __forceinline__ long long rows() const { return num; }

    __device__ __forceinline__ int entry(long long n, int *tile, int *pair) const
    {
        const int code = n < num ? __ldg(&idx[n]) : -1;
        *tile = code >> 8;
        *pair = code & 0xff;
        return code >= 0 && *pair < 6 && *tile < g.TX * g.TY;
    }

    template <int FMT>
    __device__ __forceinline__ void produce(long long n, int row, int l, unsigned gm, const TcA<4> &A,
                                            uint32_t *meta, float *) const
    {
        (void)gm;
        (void)meta;
        int tile, pair;
        float2 acc[4][4], scale[4];
        if (entry(n, &tile, &pair)) {
            corr_product<true>(clt[c_pairs[pair][0]] + (size_t)tile * 768, clt[c_pairs[pair][1]] + (size_t)tile * 768,
                               256, colors, scale0, scale1, scale2, fat_zero, l, acc, scale);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                scale[k] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q][k] = make_float2(0.0f, 0.0f);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float2 x = mul2(acc[q][k], scale[k]);
                v[2 * k] = x.x;
                v[2 * k + 1] = x.y;
            }
            A.template put8<FMT>(row, q, l * 8, v, up);
        }
    }

    /* corrUnfoldTile: R[+-i][+-j] from q0[i][j], q1[i][j-1], q2[i-1][j],
     * q3[i-1][j-1], x 1/4 (all lanes of the warp run it: the tensor-memory
     * loads are warp-wide).  A lane holds one entry, so its stores would touch a
     * sector each: the warp stages rows r - i and r + i of its 32 entries in buf
     * and stores them entry by entry, 15 consecutive floats at a time. */
    __device__ __forceinline__ void epilogue(long long n, uint32_t tb, const uint32_t *meta, int part, float *buf) const
    {
        (void)meta;
        (void)part;
        int tile, pair;
        const int lane = threadIdx.x & 31;
        const unsigned valid = __ballot_sync(0xffffffffu, entry(n, &tile, &pair));
        const int r = radius, sz = 2 * r + 1;
        const float down = 1.0f / up; /* a power of two: exact */
        float *const dst = corrs + (size_t)(n - lane) * stride; /* the warp's first entry */
        float *mine = buf + lane * kRowPair;
        float prev2[8], prev3[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            prev2[j] = 0.0f;
            prev3[j] = 0.0f;
        }
        /* lane -> (entry parity, column) of the stores */
        const int col = lane & 15, odd = lane >> 4;
        const int entries = 32 - __clz(valid); /* none after the last valid one */
#pragma unroll 1
        for (int i = 0; i <= r; i++) {
            float v[4][8];
            tc_ld8x4(tb + 8u * i, tb + 64u + 8u * i, tb + 128u + 8u * i, tb + 192u + 8u * i, v);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (j > r) break;
                const float q0 = v[0][j] * down;
                const float q1 = j > 0 ? v[1][j - 1] * down : 0.0f;
                const float q2 = prev2[j];
                const float q3 = j > 0 ? prev3[j - 1] : 0.0f;
                /* row r + i, then row r - i (the one that stays for i = 0, as the
                 * left column stays for j = 0) */
                mine[r + j] = 0.25f * ((q0 + q1) + (q2 + q3));
                mine[r - j] = 0.25f * ((q0 - q1) + (q2 - q3));
                mine[sz + r + j] = 0.25f * ((q0 + q1) - (q2 + q3));
                mine[sz + r - j] = 0.25f * ((q0 - q1) - (q2 - q3));
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                prev2[j] = v[2][j] * down;
                prev3[j] = v[3][j] * down;
            }
            __syncwarp();
            if (col < sz) {
#pragma unroll 4
                for (int e = odd; e < entries; e += 2) {
                    if (!((valid >> e) & 1)) continue;
                    float *d = dst + (size_t)e * stride + col;
                    if (i) d[(r + i) * sz] = buf[e * kRowPair + col];
                    d[(r - i) * sz] = buf[e * kRowPair + sz + col];
                }
            }
            __syncwarp();
        }
    }
};

} /* namespace tp */

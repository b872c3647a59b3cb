/*
 * tp_list.cuh - texture tile list, window of interest and RGBA clear (the
 * drop-ins for the reference's clear_texture_list, mark_texture_tiles,
 * mark_texture_neighbor_tiles, gen_texture_list and clear_texture_rbga,
 * src/TileProcessor.cuh:1618-1853).
 *
 * The reference launches these from a one-thread dynamic-parallelism driver
 * and synchronises on the device; here the list is a short task list's one
 * kernel, on one cluster of eight CTAs whose phases are separated by cluster
 * barriers, or a chain of kernels; every value the reference computed on the
 * driver thread (initial window, cleared counters, final width/height, clear
 * extent) is produced by them or read from device memory by the next kernel, so
 * a whole generate_RBGA sequence needs no host round trip and can be captured
 * in a CUDA graph.
 *
 * Launches bound a short list and the passes over the tasks a long one.  A
 * 256x256 frame (1024 tasks) through its three calls: 59.0 us with the chain,
 * 50.1 with one kernel; a sparse frame of 10,621 tasks 203.7 and 206.8, a
 * 2592x1936 one (78,408) 610.6 and 633 (its RGBA call).  So lists up to one
 * task per thread of the cluster take one kernel.
 */
#pragma once
#include <limits.h>
#include "tp_common.cuh"

namespace tp {

/* First statements of every kernel of the list / RGBA-clear sequence, which
 * the host launches as a chain of programmatic dependents: wait for the
 * launch before (everything it wrote is then visible), and only then let the
 * next one be scheduled.  A kernel that starts early therefore only ever runs
 * ahead of its own predecessor, never of the kernels before that. */
__device__ __forceinline__ void chain_entry()
{
    grid_dependency_wait();
    grid_dependents_launch();
}

/* all threads of the cluster; orders their global and shared accesses.  Not the
 * .aligned forms: those want a warp's threads to execute them together, and
 * nothing makes the threads of a warp meet again after the loops before the
 * barriers, which they leave one by one. */
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ int marker_at(const int *idx, long long i, long long cap)
{
    return (i >= 0 && i < cap) ? __ldcg(idx + i) : 0;
}

/* ---- the list in one kernel ----
 * prepare_texture_list: clear_texture_list, mark_texture_tiles,
 * mark_texture_neighbor_tiles, gen_texture_list and the window of interest.
 * Eight sub-lists: 2x2 tile parity x {inner, border}; inner lists grow up from
 * the start of their quarter of the buffer, border lists down from its end;
 * slots are claimed with one atomic per (warp, sub-list).  Values that CTAs
 * hand one another (markers, the window, a task's bits) go through L2. */
constexpr int kListCtas = 8, kListThreads = 1024;
__global__ void __cluster_dims__(kListCtas, 1, 1) __launch_bounds__(kListThreads) k_texture_list(
    tp_task *tasks, int num_tiles, int *idx, int *counts, int *woi, int width, int height, int TX, int TY,
    int quarter, long long cap, int row_first, int row_last)
{
    chain_entry();
    __shared__ int s_box[4];
    const int first = blockIdx.x * kListThreads + threadIdx.x, lane = threadIdx.x & 31;
    constexpr int kStep = kListCtas * kListThreads;
    /* marker grid: cols 0..width (inclusive, as the reference), rows 0..height-1;
     * consecutive rows overlap in their last column, so the cleared entries are
     * the runs row * TX .. row * TX + width */
    for (int row = first >> 8; row < height; row += kStep >> 8)
        for (int col = first & 255; col <= width; col += 256) {
            const long long i = (long long)col + (long long)row * TX;
            if (i < cap) __stcg(idx + i, 0);
        }
    if (first == 0) {
        __stcg(woi + 0, TX);
        __stcg(woi + 1, TY);
        __stcg(woi + 2, 0);
        __stcg(woi + 3, 0);
    }
    if (first < 8) __stcg(counts + first, 0);
    if (threadIdx.x < 4) s_box[threadIdx.x] = threadIdx.x < 2 ? INT_MAX : INT_MIN;
    cluster_sync();
#pragma unroll 4
    for (int n = first; n < num_tiles; n += kStep) {
        if (!(tasks[n].task & TP_TASK_TEXTURE_BITS)) continue;
        const int cxy = tasks[n].txy;
        const long long i = (long long)(cxy & 0xffff) + (long long)(cxy >> 16) * TX;
        if (i >= 0 && i < cap) __stcg(idx + i, 1);
    }
    cluster_sync();
    int x0 = INT_MAX, y0 = INT_MAX, x1 = INT_MIN, y1 = INT_MIN;
#pragma unroll 4
    for (int n = first; n < num_tiles; n += kStep) {
        const int task = tasks[n].task;
        if (!(task & TP_TASK_TEXTURE_BITS)) continue;
        const int cxy = tasks[n].txy;
        const int x = cxy & 0xffff, y = cxy >> 16;
        x0 = min(x0, x);
        y0 = min(y0, y);
        x1 = max(x1, x);
        y1 = max(y1, y);
        int d = 0;
        if (y > 0 && marker_at(idx, x + (long long)(y - 1) * TX, cap)) d |= 1;
        if (x < TX - 1 && marker_at(idx, (x + 1) + (long long)y * TX, cap)) d |= 2;
        if (y < TY - 1 && marker_at(idx, x + (long long)(y + 1) * TX, cap)) d |= 4;
        if (x > 0 && marker_at(idx, (x - 1) + (long long)y * TX, cap)) d |= 8;
        tasks[n].task = ((task ^ d) & TP_TASK_TEXTURE_BITS) ^ task; /* read again by this thread only */
    }
    /* the window: one update per warp, then one per CTA */
    x0 = __reduce_min_sync(0xffffffffu, x0);
    y0 = __reduce_min_sync(0xffffffffu, y0);
    x1 = __reduce_max_sync(0xffffffffu, x1);
    y1 = __reduce_max_sync(0xffffffffu, y1);
    if (lane == 0) {
        atomicMin(&s_box[0], x0);
        atomicMin(&s_box[1], y0);
        atomicMax(&s_box[2], x1);
        atomicMax(&s_box[3], y1);
    }
    __syncthreads();
    if (threadIdx.x < 2)
        atomicMin(woi + threadIdx.x, s_box[threadIdx.x]);
    else if (threadIdx.x < 4)
        atomicMax(woi + threadIdx.x, s_box[threadIdx.x]);
    cluster_sync();
    const int wx = __ldcg(woi + 0), wy = __ldcg(woi + 1), we = __ldcg(woi + 3);
    /* whole warps, so that every lane joins the vote on sub-lists */
    for (int base_n = first - lane; base_n < num_tiles; base_n += kStep) {
        const int n = base_n + lane;
        int slot = -1, entry = 0, head = 0;
        if (n < num_tiles) {
            const int task = tasks[n].task & TP_TASK_TEXTURE_BITS;
            const int cxy = tasks[n].txy;
            const int x = cxy & 0xffff, y = cxy >> 16;
            /* tiles outside [row_first, row_last) stay marked (they set their
             * neighbours' bits and the window) but are not listed */
            if (task && y >= row_first && y < row_last) {
                const int border = (x == wx) || (y == wy) || (x == TX - 1) || (y == we);
                slot = 0;
                if (x & 1) { head += quarter; slot += 2; }
                if (y & 1) { head += 2 * quarter; slot += 4; }
                if (border) { head += quarter - 1; slot += 1; }
                entry = task | ((x + y * TX) << 8) | (1 << 7);
            }
        }
        const unsigned same = __match_any_sync(0xffffffffu, slot);
        if (slot >= 0) {
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(counts + slot, __popc(same));
            base = __shfl_sync(same, base, leader);
            const int k = base + __popc(same & ((1u << lane) - 1u));
            const long long pos = (slot & 1) ? (long long)head - k : (long long)head + k;
            if (pos >= 0 && pos < cap) idx[pos] = entry;
        }
        __syncwarp();
    }
    /* every CTA has read the raw window */
    cluster_sync();
    if (first == 0) {
        woi[2] = __ldcg(woi + 2) + 1 - wx;
        woi[3] = we + 1 - wy;
    }
}

/* ---- the list as a chain of kernels, one task per thread ---- */

/* marker grid: cols 0..width (inclusive, as the reference), rows 0..height-1;
 * the window and the counts start over */
__global__ void k_clear_texture_list(int *idx, int *woi, int *counts, int width, int height, int TX, int TY,
                                     long long cap)
{
    chain_entry();
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = blockIdx.y;
    if (row == 0 && col < 8) {
        counts[col] = 0;
        if (col < 4) woi[col] = col == 0 ? TX : col == 1 ? TY : 0;
    }
    if (col > width || row >= height) return;
    const long long i = (long long)col + (long long)row * TX;
    if (i >= 0 && i < cap) idx[i] = 0;
}

__global__ void k_mark_texture_tiles(const tp_task *__restrict__ tasks, int num_tiles, int *idx, int TX,
                                     long long cap)
{
    chain_entry();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= num_tiles) return;
    if (!(tasks[n].task & TP_TASK_TEXTURE_BITS)) return;
    const int cxy = tasks[n].txy;
    const long long i = (long long)(cxy & 0xffff) + (long long)(cxy >> 16) * TX;
    if (i >= 0 && i < cap) idx[i] = 1;
}

__global__ void k_mark_neighbor_tiles(tp_task *tasks, int num_tiles, const int *idx, int *woi, int TX,
                                      int TY, long long cap)
{
    chain_entry();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int task = n < num_tiles ? tasks[n].task : 0;
    const bool listed = (task & TP_TASK_TEXTURE_BITS) != 0;
    const int cxy = listed ? tasks[n].txy : 0;
    const int x = cxy & 0xffff, y = cxy >> 16;
    /* the window: one update per warp */
    const int x0 = __reduce_min_sync(0xffffffffu, listed ? x : INT_MAX);
    const int y0 = __reduce_min_sync(0xffffffffu, listed ? y : INT_MAX);
    const int x1 = __reduce_max_sync(0xffffffffu, listed ? x : INT_MIN);
    const int y1 = __reduce_max_sync(0xffffffffu, listed ? y : INT_MIN);
    if (!(threadIdx.x & 31)) {
        atomicMin(woi + 0, x0);
        atomicMin(woi + 1, y0);
        atomicMax(woi + 2, x1);
        atomicMax(woi + 3, y1);
    }
    if (!listed) return;
    int d = 0;
    if (y > 0 && marker_at(idx, x + (long long)(y - 1) * TX, cap)) d |= 1;
    if (x < TX - 1 && marker_at(idx, (x + 1) + (long long)y * TX, cap)) d |= 2;
    if (y < TY - 1 && marker_at(idx, x + (long long)(y + 1) * TX, cap)) d |= 4;
    if (x > 0 && marker_at(idx, (x - 1) + (long long)y * TX, cap)) d |= 8;
    tasks[n].task = ((task ^ d) & TP_TASK_TEXTURE_BITS) ^ task;
}

__global__ void k_gen_texture_list(const tp_task *__restrict__ tasks, int num_tiles, int *idx,
                                   int *counts, const int *woi, int TX, int quarter, long long cap,
                                   int row_first, int row_last)
{
    chain_entry();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int slot = -1, entry = 0, head = 0;
    if (n < num_tiles) {
        const int task = tasks[n].task & TP_TASK_TEXTURE_BITS;
        const int cxy = tasks[n].txy;
        const int x = cxy & 0xffff, y = cxy >> 16;
        /* tiles outside [row_first, row_last) stay marked (they set their
         * neighbours' bits and the window) but are not listed */
        if (task && y >= row_first && y < row_last) {
            const int border = (x == woi[0]) || (y == woi[1]) || (x == TX - 1) || (y == woi[3]);
            slot = 0;
            if (x & 1) { head += quarter; slot += 2; }
            if (y & 1) { head += 2 * quarter; slot += 4; }
            if (border) { head += quarter - 1; slot += 1; }
            entry = task | ((x + y * TX) << 8) | (1 << 7);
        }
    }
    const unsigned same = __match_any_sync(0xffffffffu, slot);
    if (slot < 0) return;
    const int leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counts + slot, __popc(same));
    base = __shfl_sync(same, base, leader);
    const int k = base + __popc(same & ((1u << lane) - 1u));
    const long long pos = (slot & 1) ? (long long)head - k : (long long)head + k;
    if (pos >= 0 && pos < cap) idx[pos] = entry;
}

__global__ void k_woi_finalize(int *woi)
{
    chain_entry();
    if (threadIdx.x == 0) {
        woi[2] += 1 - woi[0];
        woi[3] += 1 - woi[1];
    }
}

/* Zero the RGBA slices: the reference clears (woi_w + 1) * 8 columns plus the
 * 8 floats a thread writes past them when the grid reaches that far, over
 * (woi_h + 1) * 8 * (colors + 1) rows.  woi == NULL: explicit extent. */
__global__ void k_clear_rbga(const int *woi, int colors, int texture_width, int slice_height,
                             size_t stride, float *buf, int *zero, int nzero)
{
    chain_entry();
    /* process_frame's list counts */
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < nzero; i += blockDim.x) zero[i] = 0;
    int tw = texture_width, rows = slice_height;
    if (woi) {
        tw = (woi[2] + 1) * 8;
        rows = (woi[3] + 1) * 8 * (colors + 1);
    }
    if (tw <= 0 || rows <= 0) return;
    const long long reach = ((long long)(tw + 255) / 256) * 256;
    long long cols = (long long)tw + 8;
    if (cols > reach) cols = reach;
    if (cols > (long long)stride) cols = (long long)stride;
    /* one block per row (grid-stride); 16-byte stores when every row starts
     * on a 16-byte boundary, the last cols % 4 floats one by one */
    const bool vec = !(reinterpret_cast<uintptr_t>(buf) & 15) && !(stride & 3);
    const long long quads = vec ? cols >> 2 : 0;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        float *p = buf + (size_t)row * stride;
        float4 *p4 = reinterpret_cast<float4 *>(p);
        for (long long q = threadIdx.x; q < quads; q += blockDim.x) p4[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (long long c = quads * 4 + threadIdx.x; c < cols; c += blockDim.x) p[c] = 0.0f;
    }
}

} /* namespace tp */

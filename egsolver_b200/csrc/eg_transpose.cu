/*
 * eg_transpose.cu -- transpose of a CSR matrix, stable within columns, by one
 * persistent cooperative kernel of five phases with four grid barriers:
 *
 *   check    offsets and columns are in range; the columns' counts to zero
 *   count    an edge's rank of arrival in its column (one atomic per warp and column)
 *   scan     offsets of the columns, each CTA its own power-of-two chunk
 *   place    a record (edge, column, row, value) to the column's next place
 *   order    a record's place among its column's by its edge number
 *
 * A radix sort of (column, edge) pairs took 18 launches and moved each edge
 * once per 8 bits of the column's number; here an edge costs three random
 * accesses (atomic, offset, record).  The order within a column is that of the atomics
 * until the last phase counts, for each record, the smaller edge numbers of
 * its column: the sum of the columns' squared lengths, which the scan adds
 * up, says what that costs, and beyond 64 looks per edge the kernel ends and
 * the caller sorts by radix (a column of 300,000 of 1 M entries: 2.0 ms a call
 * either way).
 *
 * A call with 8,191 entries: 135-150 -> 59-73 us, with 50,000: 370-420 ->
 * 128-137 us (launches and the wait for them were two thirds of it); with
 * 6.3 M the kernels' part is 0.47 -> 0.33 ms of 7-10 ms, which the copies of
 * the host's pageable arrays take.
 */
#include "eg_device.cuh"
#include "eg_transpose.cuh"

#include <algorithm>

namespace eg {
namespace {

constexpr int kThreads = 512, kPerSm = 3, kWarps = kThreads / 32;

/* All CTAs of the grid; false when the wait ran out. */
__device__ __forceinline__ bool all_arrive(const TransposeParams &p, unsigned round)
{
    __shared__ int ok;
    __syncthreads();
    if (gridDim.x == 1) return true;
    if (threadIdx.x == 0) {
        TransposeCtrl *c = p.ctrl;
        const unsigned want = round * gridDim.x;
        ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->arrivals) : "memory");
        const unsigned long long t0 = globaltimer_ns();
        unsigned spins = 0;
        while (ld_acquire_gpu(&c->arrivals) < want) {
            if ((++spins & 255) == 0 && (ld_volatile(&c->abort) || globaltimer_ns() - t0 > p.wait_limit_ns)) {
                atomicExch(&c->abort, 1);
                ok = 0;
                break;
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

/* Exclusive prefix of v over the CTA's threads; *total: their sum. */
__device__ __forceinline__ int block_prefix(int v, int *total)
{
    __shared__ int part[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(~0u, s, d);
        if (lane >= d) s += o;
    }
    if (lane == 31) part[warp] = s;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        before += w < warp ? part[w] : 0;
        all += part[w];
    }
    __syncthreads();
    *total = all;
    return before + s - v;
}

/* The last row in [lo, hi] that starts at or before edge e: e's row. */
__device__ __forceinline__ int row_of(const long long *row_ptr, int e, int lo, int hi)
{
    while (lo < hi) {
        const int mid = lo + ((hi - lo + 1) >> 1);
        if (row_ptr[mid] <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kThreads, kPerSm) k_transpose(const TransposeParams p)
{
    __shared__ int base[kTransposeGrid];
    const unsigned t = blockIdx.x * kThreads + threadIdx.x, step = gridDim.x * kThreads;
    const int lane = threadIdx.x & 31;
    const unsigned nnz = (unsigned)p.nnz;

    /* check */
    bool wrong = false;
    for (unsigned r = t; r < (unsigned)p.nrows; r += step) wrong |= p.row_ptr[r + 1] < p.row_ptr[r];
    for (unsigned e = t; e < nnz; e += step) wrong |= (unsigned)p.col[e] >= (unsigned)p.ncols;
    if (wrong) p.ctrl->bad = 1;
    for (unsigned c = t; c <= (unsigned)p.ncols; c += step) p.count[c] = 0;
    if (!all_arrive(p, 1) || ld_volatile(&p.ctrl->bad)) return;

    /* count: the lanes of a warp that meet in a column share an atomic */
    for (unsigned e0 = t - lane; e0 < nnz; e0 += step) {
        const unsigned e = e0 + lane;
        const bool on = e < nnz;
        const int c = on ? p.col[e] : -1;
        const unsigned same = __match_any_sync(~0u, c);
        const int first = __ffs(same) - 1;
        int at = 0;
        if (on && lane == first) at = atomicAdd(&p.count[c], __popc(same));
        at = __shfl_sync(~0u, at, first) + __popc(same & ((1u << lane) - 1u));
        if (on) p.rank[e] = at;
    }
    if (!all_arrive(p, 2)) return;

    /* scan */
    {
        const long long c0 = (long long)blockIdx.x << p.chunk_shift;
        const long long c1 = min(c0 + (1ll << p.chunk_shift), (long long)p.ncols + 1);
        int carry = 0;
        unsigned long long squares = 0;
        for (long long at = c0; at < c1; at += 4 * kThreads) {
            const long long c = at + 4 * threadIdx.x;
            int v[4], sum = 0, total;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                v[i] = c + i < c1 ? __ldcg(p.count + c + i) : 0;
                sum += v[i];
                squares += (unsigned long long)v[i] * (unsigned)v[i];
            }
            int run = carry + block_prefix(sum, &total);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (c + i < c1) p.count[c + i] = run;
                run += v[i];
            }
            carry += total;
        }
        if (threadIdx.x == 0) p.totals[blockIdx.x] = carry;
#pragma unroll
        for (int d = 16; d; d >>= 1) squares += __shfl_down_sync(~0u, squares, d);
        if (lane == 0 && squares) atomicAdd(&p.ctrl->squares, squares);
    }
    if (!all_arrive(p, 3)) return;
    /* 64 looks per edge on average, and columns of up to 2048 in any case */
    if (*(volatile unsigned long long *)&p.ctrl->squares > 64ull * nnz + (1ull << 22)) {
        if (t == 0) p.ctrl->skewed = 1;
        return;
    }

    /* place: a warp's edges are consecutive, its rows between two searches */
    {
        int total;
        const int mine = threadIdx.x < gridDim.x ? __ldcg(p.totals + threadIdx.x) : 0;
        const int before = block_prefix(mine, &total);
        base[threadIdx.x] = before;
        __syncthreads();
    }
    for (unsigned c = t; c <= (unsigned)p.ncols; c += step)
        p.csc_ptr[c] = __ldcg(p.count + c) + base[c >> p.chunk_shift];
    {
        const unsigned warps = step / 32, len = ((nnz + 31) / 32 + warps - 1) / warps * 32;
        const unsigned long long b = (unsigned long long)(t / 32) * len;
        if (b < nnz) {
            const unsigned e1 = (unsigned)min(b + len, (unsigned long long)nnz);
            int lo = 0, hi = 0;
            if (lane < 2) lo = row_of(p.row_ptr, lane ? (int)e1 - 1 : (int)b, 0, p.nrows - 1);
            hi = __shfl_sync(~0u, lo, 1);
            lo = __shfl_sync(~0u, lo, 0);
            for (unsigned e0 = (unsigned)b; e0 < e1; e0 += 32) {
                const unsigned e = min(e0 + lane, e1 - 1);
                const int r = row_of(p.row_ptr, (int)e, lo, hi);
                if (e0 + lane < e1) {
                    const int c = p.col[e];
                    const int at = __ldcg(p.count + c) + base[c >> p.chunk_shift] + p.rank[e];
                    p.rec[at] = make_int4((int)e, c, r, p.val[e]);
                }
                lo = __shfl_sync(~0u, r, 31);
            }
        }
    }
    if (!all_arrive(p, 4)) return;

    /* order */
    for (unsigned i = t; i < nnz; i += step) {
        const int4 x = p.rec[i];
        const int s = (int)p.csc_ptr[x.y], n = (int)p.csc_ptr[x.y + 1] - s;
        int at = s;
#pragma unroll 4
        for (int j = 0; j < n; j++) at += p.rec[s + j].x < x.x;
        p.csc_row[at] = x.z;
        p.csc_val[at] = x.w;
    }
}

}  // namespace

int transpose_grid(int nrows, int ncols, long long nnz, int sms)
{
    const long long items = std::max<long long>({nnz, nrows, (long long)ncols + 1});
    return (int)std::max<long long>(1, std::min<long long>({(items + 4 * kThreads - 1) / (4 * kThreads),
                                                             (long long)kPerSm * sms, (long long)kTransposeGrid}));
}

cudaError_t launch_transpose(TransposeParams p, int grid, cudaStream_t st)
{
    p.chunk_shift = 2;
    while (((long long)grid << p.chunk_shift) < (long long)p.ncols + 1) p.chunk_shift++;
    void *args[] = {&p};
    return cudaLaunchCooperativeKernel((const void *)k_transpose, dim3((unsigned)grid), dim3(kThreads), args, 0, st);
}

}  // namespace eg

// Stable transpose of a compressed structure on the GPU.
//
// Upstream (src/sparse/CSC_matrix.c:62-104, CSR_matrix.c:144-187) transposes by a
// serial counting sort: count entries per column, scan, then scatter the entries in
// row-major order, which leaves the source rows ascending inside every column. Here
// the count and scatter run in parallel with atomics, which loses the order, so
// each entry carries its source position e and every output segment is then
// sorted by e; because source positions grow in row-major order, that restores
// exactly upstream's order (ties inside one source row included).
//
// Segments of up to 64 keys (nearly all) are sorted tile by tile: a key's place is the
// number of smaller keys in its segment, counted in shared memory. Longer segments go by
// size class: <= 1024 in shared memory by one warp, <= 8192 in shared memory by one CTA,
// larger ones by a CTA merge sort through a global scratch buffer.
#include <algorithm>
#include <vector>

#include "sdl_device.cuh"
#include "sdl_internal.h"

namespace sdl {
namespace {

constexpr int SCATTER_TILE = 2048;
constexpr int SCATTER_THREADS = 256;
constexpr int SCATTER_ITEMS = SCATTER_TILE / SCATTER_THREADS;

// Entries per column, and every entry's place among its column's (in the order the adds
// happen to take). What bounds it: the latency of the adds, so eight entries per thread
// are in flight together. 1.5M entries: 26 us here and 41 us in the scatter, against 19 and
// 70 us with one entry at a time and a second add per entry in the scatter.
__global__ void __launch_bounds__(SCATTER_THREADS) k_count_idx(const int *__restrict__ idx, int nnz,
                                                               int *__restrict__ cnt, int *__restrict__ slot)
{
    const long long e0 = blockIdx.x * (long long)SCATTER_TILE + threadIdx.x;
    int c[SCATTER_ITEMS];
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
    {
        const long long e = e0 + j * SCATTER_THREADS;
        c[j] = e < nnz ? idx[e] : -1;
    }
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
        if (c[j] >= 0) c[j] = atomicAdd(&cnt[c[j]], 1);
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
    {
        const long long e = e0 + j * SCATTER_THREADS;
        if (e < nnz) slot[e] = c[j];
    }
}

// Last r in [lo, hi) with p[r] <= e (p non-decreasing, p[lo] <= e < p[hi]).
__device__ __forceinline__ int row_of(const int *p, int lo, int hi, int e)
{
    while (hi - lo > 1)
    {
        int mid = (lo + hi) >> 1;
        if (p[mid] <= e)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// The same by a whole warp, 32 probes at a time.
__device__ __forceinline__ int warp_row_of(const int *p, int lo, int hi, int e)
{
    const int lane = lane_id();
    while (hi - lo > 1)
    {
        const int step = (int)(((long long)hi - lo + 31) / 32);
        const long long at = lo + (long long)step * lane; // p[lo] <= e: lane 0 holds
        const unsigned le = __ballot_sync(FULL_MASK, at < hi && p[at] <= e);
        const int last = 31 - __clz(le);
        lo += step * last;
        hi = (int)min((long long)hi, (long long)lo + step);
    }
    return lo;
}

// keys[Tp[c] + slot] = (e << 32) | row for every source entry e = (row, c).
__global__ void __launch_bounds__(SCATTER_THREADS) k_scatter_keys(const int *__restrict__ p,
                                                                  const int *__restrict__ idx, int rows, int nnz,
                                                                  const int *__restrict__ Tp,
                                                                  const int *__restrict__ slot,
                                                                  unsigned long long *__restrict__ keys)
{
    __shared__ int r_first, r_last, sp[SCATTER_TILE];
    const long long e0 = (long long)blockIdx.x * SCATTER_TILE;
    const int cnt = (int)min((long long)SCATTER_TILE, nnz - e0);
    int at[SCATTER_ITEMS];
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
    {
        const int i = threadIdx.x + j * SCATTER_THREADS;
        at[j] = i < cnt ? idx[e0 + i] : -1;
    }
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
        if (at[j] >= 0) at[j] = Tp[at[j]] + slot[e0 + threadIdx.x + j * SCATTER_THREADS];
    int lo = 0, n_r = 0;
    if (p)
    {
        // the tile's rows; their offsets in shared memory where they fit
        if (threadIdx.x < 64)
        {
            const int r = warp_row_of(p, 0, rows, (int)(threadIdx.x < 32 ? e0 : e0 + cnt - 1));
            if (threadIdx.x == 0) r_first = r;
            if (threadIdx.x == 32) r_last = r;
        }
        __syncthreads();
        lo = r_first;
        n_r = r_last - lo + 1;
        if (n_r <= SCATTER_TILE)
        {
            for (int k = threadIdx.x; k < n_r; k += SCATTER_THREADS) sp[k] = p[lo + k];
            __syncthreads();
        }
    }
#pragma unroll
    for (int j = 0; j < SCATTER_ITEMS; ++j)
    {
        if (at[j] < 0) continue;
        const int e = (int)e0 + threadIdx.x + j * SCATTER_THREADS;
        const int r = !p ? e : n_r <= SCATTER_TILE ? lo + row_of(sp, 0, n_r, e) : row_of(p, lo, lo + n_r, e);
        keys[at[j]] = ((unsigned long long)e << 32) | (unsigned)r;
    }
}

// size classes of segments beyond SEG_SHORT keys
constexpr int SEG_SHORT = 64;
enum
{
    SEG_W1K = 0,
    SEG_C8K,
    SEG_BIG,
    SEG_NCLS
};
// Keys of a CTA of k_seg_rank: few where the segments outnumber the keys, since a key's
// search then goes through global memory, and is a chain of about 20 loads (4000 keys over
// 1M segments: the conversion 204 -> 179 us).
constexpr int RANK_TILE = 2048, RANK_TILE_SPARSE = 256;
constexpr int RANK_THREADS = 256;

// First segment that starts in each tile of `tile` keys (nseg past the last), and the
// segments beyond SEG_SHORT keys, listed per class (one add per warp and class).
__global__ void k_seg_tiles(const int *__restrict__ off, int nseg, int tile, int ntiles, int *__restrict__ first,
                            int *__restrict__ counts, int *__restrict__ lists)
{
    const int lane = lane_id();
    for (long long s0 = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; s0 <= nseg;
         s0 += (long long)gridDim.x * blockDim.x)
    {
        const long long s = s0 + lane;
        int cls = SEG_NCLS;
        if (s <= nseg)
        {
            const int o = off[s];
            const int b0 = s ? off[s - 1] / tile + 1 : 0;
            const int b1 = s < nseg ? o / tile : ntiles;
            for (int b = b0; b <= b1; ++b) first[b] = (int)s;
            const int len = s < nseg ? off[s + 1] - o : 0;
            if (len > SEG_SHORT) cls = len <= 1024 ? SEG_W1K : len <= 8192 ? SEG_C8K : SEG_BIG;
        }
        if (!__any_sync(FULL_MASK, cls < SEG_NCLS)) continue;
#pragma unroll
        for (int c = 0; c < SEG_NCLS; ++c)
        {
            const unsigned of = __ballot_sync(FULL_MASK, cls == c);
            if (!of) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&counts[c], __popc(of));
            at = __shfl_sync(FULL_MASK, at, 0) + __popc(of & lanemask_lt());
            // a class's segments are at most nkeys / 65 together: its list starts there
            if (cls == c) lists[c * (long long)(off[nseg] / (SEG_SHORT + 1)) + at] = (int)s;
        }
    }
}

// The segments that start in a tile and have at most SEG_SHORT keys: every key finds its
// segment (a search over the tile's offsets, in shared memory where they fit) and its
// place in it. Writes the two halves of the key there, in order. What bounds it: about
// 120 instructions per 32 keys; 1.5M keys in segments of 9 take 33 us, where listing the
// segments and sorting each by a warp's bitonic network took 175 us.
template <int TILE>
__global__ void __launch_bounds__(RANK_THREADS) k_seg_rank(const unsigned long long *__restrict__ keys,
                                                           const int *__restrict__ off, int nkeys,
                                                           const int *__restrict__ first, int *__restrict__ lo_out,
                                                           int *__restrict__ hi_out)
{
    __shared__ unsigned long long sk[TILE + SEG_SHORT];
    __shared__ int so[TILE + 1];
    const int k0 = blockIdx.x * TILE;
    const int cnt = (int)min((long long)TILE + SEG_SHORT - 1, (long long)nkeys - k0);
    const int c0 = first[blockIdx.x], nc = first[blockIdx.x + 1] - c0;
    if (nc == 0) return;
    for (int k = threadIdx.x; k < cnt; k += RANK_THREADS) sk[k] = keys[k0 + k];
    const bool fit = nc <= TILE;
    if (fit)
        for (int k = threadIdx.x; k <= nc; k += RANK_THREADS) so[k] = off[c0 + k];
    __syncthreads();
    const int *o = fit ? so : off + c0; // offsets of the tile's segments, nc + 1 of them
    const int from = o[0] - k0, to = min(cnt, o[nc] - k0);
    // the segments of all of a thread's keys are searched for together
    constexpr int U = (TILE + SEG_SHORT + RANK_THREADS - 1) / RANK_THREADS;
    int seg[U];
#pragma unroll
    for (int j = 0; j < U; ++j) seg[j] = 0;
    for (int w = 1 << (31 - __clz(nc)); w; w >>= 1)
    {
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (seg[j] + w < nc && o[seg[j] + w] <= k0 + from + (int)threadIdx.x + j * RANK_THREADS) seg[j] += w;
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
    {
        const int k = from + threadIdx.x + j * RANK_THREADS;
        if (k >= to) break;
        const int b = o[seg[j]] - k0, e = o[seg[j] + 1] - k0;
        if (e - b > SEG_SHORT) continue;
        const unsigned long long key = sk[k];
        int r = b;
        for (int i = b; i < e; ++i) r += sk[i] < key;
        lo_out[k0 + r] = (int)(key & 0xffffffffu);
        hi_out[k0 + r] = (int)(key >> 32);
    }
}

// <= 1024 keys: one warp per segment, shared-memory bitonic. Like the other
// sorts it writes the two halves of the keys in their order (another kernel that took them from
// the sorted keys: columns of 66 entries, 30M in all, 3.02 -> 2.42 ms).
__global__ void k_segsort_w1k(const int *__restrict__ list, int count, const int *__restrict__ off,
                              const unsigned long long *__restrict__ keys, int *__restrict__ lo_out,
                              int *__restrict__ hi_out)
{
    extern __shared__ unsigned long long smk[];
    const int lane = lane_id();
    const int wpb = blockDim.x >> 5;
    unsigned long long *buf = smk + (threadIdx.x >> 5) * 1024;
    for (long long w = blockIdx.x * (long long)wpb + (threadIdx.x >> 5); w < count;
         w += (long long)gridDim.x * wpb)
    {
        int s = list[w];
        int b = off[s], len = off[s + 1] - b;
        int P = next_pow2(len);
        for (int q = lane; q < P; q += 32) buf[q] = q < len ? keys[b + q] : ~0ull;
        __syncwarp();
        warp_bitonic_sort(buf, P);
        for (int q = lane; q < len; q += 32)
        {
            lo_out[b + q] = (int)(buf[q] & 0xffffffffu);
            hi_out[b + q] = (int)(buf[q] >> 32);
        }
        __syncwarp();
    }
}

// <= 8192 keys: one CTA per segment.
__global__ void k_segsort_c8k(const int *__restrict__ list, int count, const int *__restrict__ off,
                              const unsigned long long *__restrict__ keys, int *__restrict__ lo_out,
                              int *__restrict__ hi_out)
{
    extern __shared__ unsigned long long smk[];
    for (int w = blockIdx.x; w < count; w += gridDim.x)
    {
        int s = list[w];
        int b = off[s], len = off[s + 1] - b;
        int P = next_pow2(len);
        for (int q = threadIdx.x; q < P; q += blockDim.x) smk[q] = q < len ? keys[b + q] : ~0ull;
        __syncthreads();
        block_bitonic_sort(smk, P);
        for (int q = threadIdx.x; q < len; q += blockDim.x)
        {
            lo_out[b + q] = (int)(smk[q] & 0xffffffffu);
            hi_out[b + q] = (int)(smk[q] >> 32);
        }
        __syncthreads();
    }
}

constexpr int BIG_CHUNK = 8192;

// Big segments: sort BIG_CHUNK-sized chunks in shared memory, then merge runs
// pairwise (merge path per thread) between keys and scratch until one run is left, and write
// its halves.
__global__ void k_segsort_big(const int *__restrict__ list, int count, const int *__restrict__ off,
                              unsigned long long *__restrict__ keys,
                              unsigned long long *__restrict__ scratch, int *__restrict__ lo_out,
                              int *__restrict__ hi_out)
{
    extern __shared__ unsigned long long smk[];
    for (int w = blockIdx.x; w < count; w += gridDim.x)
    {
        int s = list[w];
        int b = off[s], len = off[s + 1] - b;
        unsigned long long *src = keys + b, *dst = scratch + b;
        for (int c0 = 0; c0 < len; c0 += BIG_CHUNK)
        {
            int cl = min(BIG_CHUNK, len - c0);
            int P = next_pow2(cl);
            for (int q = threadIdx.x; q < P; q += blockDim.x) smk[q] = q < cl ? src[c0 + q] : ~0ull;
            __syncthreads();
            block_bitonic_sort(smk, P);
            for (int q = threadIdx.x; q < cl; q += blockDim.x) src[c0 + q] = smk[q];
            __syncthreads();
        }
        bool in_src = true;
        for (int width = BIG_CHUNK; width < len; width <<= 1)
        {
            const unsigned long long *in = in_src ? src : dst;
            unsigned long long *out = in_src ? dst : src;
            for (int ps = 0; ps < len; ps += 2 * width)
            {
                int na = min(width, len - ps);
                int nb = max(0, min(width, len - ps - width));
                const unsigned long long *A = in + ps, *B = in + ps + na;
                int tot = na + nb;
                int per = (tot + blockDim.x - 1) / blockDim.x;
                int d0 = min(tot, (int)threadIdx.x * per), d1 = min(tot, d0 + per);
                if (d0 < d1)
                {
                    int lo = max(0, d0 - nb), hi = min(d0, na);
                    while (lo < hi)
                    {
                        int mid = (lo + hi) >> 1;
                        if (A[mid] < B[d0 - 1 - mid])
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    int i = lo, j = d0 - lo;
                    for (int d = d0; d < d1; ++d)
                    {
                        bool takeA = j >= nb || (i < na && A[i] < B[j]);
                        out[ps + d] = takeA ? A[i++] : B[j++];
                    }
                }
            }
            __syncthreads();
            in_src = !in_src;
        }
        const unsigned long long *sorted = in_src ? src : dst;
        for (int q = threadIdx.x; q < len; q += blockDim.x)
        {
            lo_out[b + q] = (int)(sorted[q] & 0xffffffffu);
            hi_out[b + q] = (int)(sorted[q] >> 32);
        }
    }
}

// Sorts every segment [off[s], off[s+1]) of keys ascending (keys unique per segment) and
// writes the keys' two halves in that order; keys is scratch.
void segment_sort(unsigned long long *d_keys, const int *d_off, int nseg, int nkeys, int *lo_out, int *hi_out,
                  cudaStream_t s)
{
    Runtime &rt = runtime();
    const bool sparse = nseg > nkeys;
    const int tile = sparse ? RANK_TILE_SPARSE : RANK_TILE, ntiles = (nkeys - 1) / tile + 1;
    const int stride = nkeys / (SEG_SHORT + 1);
    DevBuf<int> first((size_t)ntiles + 1), counts(SEG_NCLS), lists((size_t)SEG_NCLS * stride + 1);
    SDL_CUDA(cudaMemsetAsync(counts.get(), 0, counts.bytes(), s));
    const int grid = (int)std::min<long long>(((long long)nseg + 256) / 256, (long long)rt.num_sms * 8);
    SDL_LAUNCH(k_seg_tiles, grid, 256, 0, s, d_off, nseg, tile, ntiles, first.get(), counts.get(), lists.get());
    int h[SEG_NCLS];
    SDL_CUDA(cudaMemcpyAsync(h, counts.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    const auto rank = sparse ? k_seg_rank<RANK_TILE_SPARSE> : k_seg_rank<RANK_TILE>;
    SDL_LAUNCH(rank, ntiles, RANK_THREADS, 0, s, d_keys, d_off, nkeys, first.get(), lo_out, hi_out);
    SDL_CUDA(cudaStreamSynchronize(s));
    const int cap = rt.num_sms * 16;
    if (h[SEG_W1K])
    {
        int g = std::min((h[SEG_W1K] + 3) / 4, cap);
        size_t sm = 4 * 1024 * sizeof(unsigned long long);
        SDL_CUDA(cudaFuncSetAttribute(k_segsort_w1k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        SDL_LAUNCH(k_segsort_w1k, g, 128, sm, s, lists.get(), h[SEG_W1K], d_off, d_keys, lo_out, hi_out);
    }
    if (h[SEG_C8K] || h[SEG_BIG])
    {
        size_t sm = 8192 * sizeof(unsigned long long);
        SDL_CUDA(cudaFuncSetAttribute(k_segsort_c8k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        SDL_CUDA(cudaFuncSetAttribute(k_segsort_big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        if (h[SEG_C8K])
        {
            int g = std::min(h[SEG_C8K], cap);
            SDL_LAUNCH(k_segsort_c8k, g, 512, sm, s, lists.get() + SEG_C8K * (size_t)stride, h[SEG_C8K], d_off,
                       d_keys, lo_out, hi_out);
        }
        if (h[SEG_BIG])
        {
            DevBuf<unsigned long long> scratch(nkeys);
            int g = std::min(h[SEG_BIG], rt.num_sms);
            SDL_LAUNCH(k_segsort_big, g, 1024, sm, s, lists.get() + SEG_BIG * (size_t)stride, h[SEG_BIG], d_off,
                       d_keys, scratch.get(), lo_out, hi_out);
            SDL_CUDA(cudaStreamSynchronize(s)); // scratch is freed on return
        }
    }
    SDL_CUDA(cudaStreamSynchronize(s)); // the lists are freed on return
}

} // namespace

void transpose_build(const int *d_p, const int *d_idx, int rows, int cols, int nnz,
                     TransposePlan &out, cudaStream_t s)
{
    const FreeScope frees;
    out.rows = rows;
    out.cols = cols;
    out.nnz = nnz;
    out.Tp.reset((size_t)cols + 1);
    out.Ti.reset(nnz);
    out.src.reset(nnz);
    if (nnz == 0)
    {
        SDL_CUDA(cudaMemsetAsync(out.Tp.get(), 0, out.Tp.bytes(), s));
        SDL_CUDA(cudaStreamSynchronize(s));
        return;
    }
    DevBuf<int> cnt((size_t)cols + 1), slot((size_t)nnz);
    SDL_CUDA(cudaMemsetAsync(cnt.get(), 0, cnt.bytes(), s));
    const int tiles = (int)(((long long)nnz + SCATTER_TILE - 1) / SCATTER_TILE);
    SDL_LAUNCH(k_count_idx, tiles, SCATTER_THREADS, 0, s, d_idx, nnz, cnt.get(), slot.get());
    exclusive_scan_i32_checked(cnt.get(), out.Tp.get(), cols, s);
    DevBuf<unsigned long long> keys(nnz);
    SDL_LAUNCH(k_scatter_keys, tiles, SCATTER_THREADS, 0, s, d_p, d_idx, rows, nnz, out.Tp.get(), slot.get(),
               keys.get());
    segment_sort(keys.get(), out.Tp.get(), cols, nnz, out.Ti.get(), out.src.get(), s);
}

} // namespace sdl

// COO coalescing (and the matrix sums built on it): the plan sorts the triplets
// once, stably, by (row, column), so they sit in (row, column, triplet)
// order; the first triplet of each distinct (row, column) opens an output, which
// gives the coalesced CSR structure and, in the same order, the triplet-to-output
// permutation. A value refill is then a gather in output order: one thread per
// output summing its triplets' values (times their factors, when given) from +0.0
// in ascending triplet order -- upstream's memset + accumulator order, bit for bit
// -- with the permutation read in order and the values gathered once each.
#include <algorithm>

#include "sdl_device.cuh"
#include "sdl_internal.h"

namespace sdl {

namespace {

int grid_coal(long long n, int per_block)
{
    long long g = (n + per_block - 1) / per_block;
    return (int)std::max<long long>(1, std::min<long long>(g, 148LL * 32));
}

// A thread per output, four outputs (one grid stride apart) at a time: the first
// triplet of each is fetched before any is summed, so four dependent chains (start
// -> position -> value) are in flight together; further triplets of an output (the
// duplicates) follow in ascending order. Each output is summed from +0.0 in
// ascending triplet order.
constexpr int COAL_ILP = 4;
__global__ void k_coal_fill(const int *__restrict__ ostart, const int *__restrict__ perm, const double *__restrict__ x,
                            const double *__restrict__ f, int nout, double *__restrict__ C)
{
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long base = blockIdx.x * (long long)blockDim.x + threadIdx.x; base < nout; base += step * COAL_ILP)
    {
        int q0[COAL_ILP], q1[COAL_ILP];
#pragma unroll
        for (int j = 0; j < COAL_ILP; ++j)
        {
            const long long o = base + j * step;
            q0[j] = q1[j] = 0;
            if (o < nout)
            {
                q0[j] = __ldcs(ostart + o);
                q1[j] = __ldcs(ostart + o + 1);
            }
        }
        int t[COAL_ILP];
#pragma unroll
        for (int j = 0; j < COAL_ILP; ++j) t[j] = q0[j] < q1[j] ? __ldcs(perm + q0[j]) : -1;
        double v[COAL_ILP];
#pragma unroll
        for (int j = 0; j < COAL_ILP; ++j)
            v[j] = t[j] < 0 ? 0.0 : (f ? __dmul_rn(f[t[j]], x[t[j]]) : x[t[j]]);
#pragma unroll
        for (int j = 0; j < COAL_ILP; ++j)
        {
            const long long o = base + j * step;
            if (o >= nout) continue;
            double acc = __dadd_rn(0.0, v[j]);
            for (int q = q0[j] + 1; q < q1[j]; ++q)
            {
                const int tq = __ldcs(perm + q);
                acc = __dadd_rn(acc, f ? __dmul_rn(f[tq], x[tq]) : x[tq]);
            }
            __stcs(C + o, acc);
        }
    }
}

// Structure and refill plan of a coalescing in one sort: the triplets stably
// radix-sorted by (row, column); the first triplet of every distinct (row, column)
// opens an output, in CSR order. The sorted triplets are the refill's permutation.
constexpr int CS_TILE = 2048; // triplets of a CTA
constexpr int CS_THREADS = 256;
constexpr int CS_ITEMS = CS_TILE / CS_THREADS;

__device__ __forceinline__ bool cs_opens(const unsigned long long *__restrict__ keys, int n, long long q)
{
    return q < n && (q == 0 || keys[q] != keys[q - 1]);
}

// Outputs that each tile's triplets open (and no gaps yet).
__global__ void __launch_bounds__(CS_THREADS) k_cs_count(const unsigned long long *__restrict__ keys, int n,
                                                         int *__restrict__ tile_outs, int *__restrict__ ngaps)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *ngaps = 0;
    __shared__ int part[CS_THREADS / 32];
    const long long q0 = (long long)blockIdx.x * CS_TILE + threadIdx.x;
    int c = 0;
#pragma unroll
    for (int j = 0; j < CS_ITEMS; ++j) c += cs_opens(keys, n, q0 + j * CS_THREADS);
    c = __reduce_add_sync(FULL_MASK, c);
    if (lane_id() == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int k = 1; k < CS_THREADS / 32; ++k) c += part[k];
        tile_outs[blockIdx.x] = c;
    }
}

// A run of row offsets of one value, [first, last] (rows up to INT_MAX, so both ends are
// inclusive), that k_cs_emit leaves to k_cs_gaps.
struct CsGap
{
    int first, last, value;
};
constexpr int CS_GAP = 1 << 16; // longest run that one warp writes, about 9 us
__host__ __device__ constexpr long long cs_gap_cap(int m) { return 2 * (((long long)m + 1) / CS_GAP); }

// Column and first triplet of every output, and the row offsets: the first output of a
// row closes the rows between the previous output's row and its own, one past the last
// triplet the rows after it. Runs of up to 8 rows are written by the lane that finds them,
// of up to CS_GAP by its warp; longer ones are listed in gaps, cut into pieces of CS_GAP
// rows, at most cs_gap_cap(m) in all (a run of CS_GAP + 1 rows or more gives at most two
// pieces per CS_GAP rows). A warp takes CS_ITEMS times 32 consecutive triplets, so that an
// output's neighbours are written beside it.
__global__ void __launch_bounds__(CS_THREADS) k_cs_emit(const unsigned long long *__restrict__ keys, int n, int m,
                                                        int col_bits, const int *__restrict__ tile_first,
                                                        int *__restrict__ ostart, int *__restrict__ Ci,
                                                        int *__restrict__ Cp, CsGap *__restrict__ gaps,
                                                        int *__restrict__ ngaps)
{
    __shared__ int part[CS_THREADS / 32];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const long long q0 = (long long)blockIdx.x * CS_TILE + warp * (32 * CS_ITEMS) + lane;
    unsigned long long key[CS_ITEMS], prev[CS_ITEMS];
#pragma unroll
    for (int j = 0; j < CS_ITEMS; ++j)
    {
        const long long q = q0 + 32 * j;
        key[j] = q < n ? keys[q] : 0;
        prev[j] = q > 0 && q <= n ? keys[q - 1] : 0;
    }
    unsigned heads[CS_ITEMS];
    int c = 0;
#pragma unroll
    for (int j = 0; j < CS_ITEMS; ++j)
    {
        const long long q = q0 + 32 * j;
        heads[j] = __ballot_sync(FULL_MASK, q < n && (q == 0 || key[j] != prev[j]));
        c += __popc(heads[j]);
    }
    if (lane == 0) part[warp] = c;
    __syncthreads();
    int o0 = tile_first[blockIdx.x];
    for (int k = 0; k < warp; ++k) o0 += part[k];
    const unsigned long long cmask = (1ull << col_bits) - 1;
#pragma unroll
    for (int j = 0; j < CS_ITEMS; ++j)
    {
        const long long q = q0 + 32 * j;
        const int o = o0 + __popc(heads[j] & lanemask_lt());
        unsigned lo = 0, hi = 0; // Cp[lo .. hi) = o (hi is up to 2^31)
        if ((heads[j] >> lane) & 1u)
        {
            ostart[o] = (int)q;
            Ci[o] = (int)(key[j] & cmask);
            lo = q == 0 ? 0 : (unsigned)(prev[j] >> col_bits) + 1;
            hi = (unsigned)(key[j] >> col_bits) + 1;
        }
        else if (q == n) // one past the last triplet
        {
            ostart[o] = n;
            lo = (unsigned)(prev[j] >> col_bits) + 1;
            hi = (unsigned)m + 1;
        }
        unsigned longs = __ballot_sync(FULL_MASK, hi - lo > 8);
        if (hi - lo <= 8)
            for (unsigned r = lo; r < hi; ++r) Cp[r] = o;
        for (; longs; longs &= longs - 1)
        {
            const int l = __ffs(longs) - 1;
            const unsigned x = __shfl_sync(FULL_MASK, lo, l), y = __shfl_sync(FULL_MASK, hi, l);
            const int v = __shfl_sync(FULL_MASK, o, l);
            if (y - x <= CS_GAP)
            {
                for (unsigned r = x + lane; r < y; r += 32) Cp[r] = v;
                continue;
            }
            const int pieces = (int)((y - x + CS_GAP - 1) / CS_GAP);
            int at = 0;
            if (lane == 0) at = atomicAdd(ngaps, pieces);
            at = __shfl_sync(FULL_MASK, at, 0);
            for (int p = lane; p < pieces; p += 32)
            {
                const unsigned r = x + (unsigned)p * CS_GAP;
                gaps[at + p] = CsGap{(int)r, (int)(min(r + CS_GAP, y) - 1), v};
            }
        }
        o0 += __popc(heads[j]);
    }
}

// The long runs of row offsets, a CTA per piece. Written by the warp that found them, runs
// took the build of 1M triplets in 10 rows out of 500M from 4.7 to 67 ms.
__global__ void __launch_bounds__(CS_THREADS) k_cs_gaps(const CsGap *__restrict__ gaps, const int *__restrict__ ngaps,
                                                        int *__restrict__ Cp)
{
    for (int g = blockIdx.x; g < *ngaps; g += gridDim.x)
    {
        const CsGap G = gaps[g];
        const int rows = G.last - G.first + 1; // at most CS_GAP
        for (int k = threadIdx.x; k < rows; k += CS_THREADS) Cp[(long long)G.first + k] = G.value;
    }
}

// What a one-pass refill of the plan would meet: the most triplets of an output, and the
// 128-byte lines of values that the CS_TILE neighbours of a tile in sorted order read, summed
// over one tile in CS_SAMPLE. (Per 32 neighbours the lines of interleaved sorted streams, six
// sorted matrices to be added up, count several times.)
constexpr int CS_SAMPLE = 16;
__global__ void __launch_bounds__(CS_THREADS) k_cs_spread(const int *__restrict__ ostart, int nout,
                                                          const int *__restrict__ perm, int n,
                                                          int *__restrict__ longest, int *__restrict__ lines)
{
    static_assert(2 * CS_TILE == 1 << 12, "the places that the top 12 bits of a hash name");
    __shared__ int seen[2 * CS_TILE];
    int most = 0, mlines = 0;
    for (long long o = blockIdx.x * (long long)CS_THREADS + threadIdx.x; o < nout; o += (long long)gridDim.x * CS_THREADS)
        most = max(most, ostart[o + 1] - ostart[o]);
    for (long long t = (long long)blockIdx.x * CS_SAMPLE * CS_TILE; t < n; t += (long long)gridDim.x * CS_SAMPLE * CS_TILE)
    {
        __syncthreads();
        for (int k = threadIdx.x; k < 2 * CS_TILE; k += CS_THREADS) seen[k] = -1;
        __syncthreads();
        for (int i = threadIdx.x; i < CS_TILE && t + i < n; i += CS_THREADS)
        {
            const int line = perm[t + i] >> 4;
            // (the table has twice as many places as there are lines, so a probe ends)
            for (unsigned h = (unsigned)line * 2654435761u;; h += 1u << 20)
            {
                const int old = atomicCAS(&seen[h >> 20], -1, line);
                mlines += old == -1;
                if (old == -1 || old == line) break;
            }
        }
    }
    most = __reduce_max_sync(FULL_MASK, most);
    mlines = __reduce_add_sync(FULL_MASK, mlines);
    if (lane_id() == 0)
    {
        atomicMax(longest, most);
        if (mlines) atomicAdd(lines, mlines);
    }
}

// ------------------------------------------------------------------ bucketed refill
// For large inputs the one-pass refill gathers every triplet value at random from an
// array larger than L2, so DRAM moves whole sectors for 8 useful bytes. The bucketed
// refill takes two passes. The sorted triplets are cut, at outputs, into buckets of
// about CB_SPAN, whose values lie together in buf, ordered by input chunk:
//  1. a CTA per input chunk reads its values (times their factors, when given) into
//     shared memory and writes them out bucket by bucket, so a bucket's values of one
//     chunk leave as one run;
//  2. a CTA per bucket reads its values into shared memory and sums every output from
//     there, in ascending triplet order from +0.0: the one-pass refill's sums.
// A bucket beyond CB_CAP values (an output of over a thousand triplets) keeps its
// values in sorted order and is summed from global memory.
// What bounds it: HBM, 8 + 6 + 8 bytes per triplet in pass 1, 8 + 2 in pass 2 and 4 + 8
// per output (2.0 GB for 50M triplets of 35M outputs), both passes at two thirds of the
// copy bandwidth: 580 -> 445 us there. Before, buckets of 2^20 outputs were gathered from
// L2, at 8 useful bytes a sector: 194 us for pass 1, 377 for pass 2.
// The sizes: long runs matter more than a second CTA per SM to overlap the phases (chunks
// of 8192 / 12288 / 14336 / 26624: 553 / 492 / 482 / 445 us; buckets of 10752, two CTAs:
// 471), since a run's two ends are partial sectors. Values sent to buf straight from
// registers, one sector a lane, took 643 us for pass 1 alone.
constexpr int CB_CAP = 22528;  // values of a bucket in shared memory, with 2 bytes of order each
constexpr int CB_SPAN = 21504; // triplets after which the next output opens a bucket
constexpr int CB_THREADS = 1024;
constexpr size_t CB_SMEM = (size_t)(CB_CAP + 2) * sizeof(double) + (CB_CAP + 16) * sizeof(short);
constexpr int CB_CHUNK = 26624; // triplets of a chunk
constexpr int CB_CHUNK_THREADS = 1024;
constexpr size_t CB_CHUNK_SMEM = (size_t)CB_CHUNK * sizeof(double);
constexpr int CB_RANGES = 8192;   // input ranges (whole chunks) that a bucket keeps in order
constexpr int CB_BINS = 8192;     // ranges of buf that a chunk is written in the order of
constexpr size_t CB_ORDER_SMEM = (size_t)CB_CHUNK * (sizeof(int) + sizeof(short)) + CB_BINS * sizeof(int);

// First output of every bucket: the one that opens at or after b * CB_SPAN.
__global__ void k_cb_begin(const int *__restrict__ ostart, int nout, int nb, int *__restrict__ begin)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nb) return;
    const long long q = (long long)b * CB_SPAN;
    begin[b] = b == nb || q > INT_MAX ? nout : lower_bound_dev(ostart, nout, (int)q);
}

// Exclusive prefix sums of cnt[0 .. N) in place, by the whole block.
template <int N, int THREADS>
__device__ __forceinline__ void cb_prefix(int *cnt, int *scr)
{
    constexpr int PER = N / THREADS;
    int c[PER], sum = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k)
    {
        c[k] = cnt[threadIdx.x * PER + k];
        sum += c[k];
    }
    int run = block_incl_scan_int(sum, scr) - sum;
#pragma unroll
    for (int k = 0; k < PER; ++k)
    {
        cnt[threadIdx.x * PER + k] = run;
        run += c[k];
    }
    __syncthreads();
}

// A CTA per bucket: the place of each of its triplets in buf, counted out by input range
// in shared memory -- pos of the triplet, and of every sorted triplet its place inside
// the bucket.
__global__ void __launch_bounds__(CB_THREADS) k_cb_plan(const int *__restrict__ perm, const int *__restrict__ begin,
                                                        const int *__restrict__ ostart, int range,
                                                        int *__restrict__ pos, unsigned short *__restrict__ local)
{
    __shared__ int at[CB_RANGES];
    __shared__ int scr[32];
    const int q0 = ostart[begin[blockIdx.x]], q1 = ostart[begin[blockIdx.x + 1]];
    if (q1 - q0 > CB_CAP)
    {
        for (int q = q0 + threadIdx.x; q < q1; q += CB_THREADS) pos[perm[q]] = q;
        return;
    }
    for (int k = threadIdx.x; k < CB_RANGES; k += CB_THREADS) at[k] = 0;
    __syncthreads();
    for (int q = q0 + threadIdx.x; q < q1; q += CB_THREADS) atomicAdd(&at[perm[q] / range], 1);
    cb_prefix<CB_RANGES, CB_THREADS>(at, scr);
    for (int q = q0 + threadIdx.x; q < q1; q += CB_THREADS)
    {
        const int t = perm[q];
        const int l = atomicAdd(&at[t / range], 1);
        local[q] = (unsigned short)l;
        pos[t] = q0 + l;
    }
}

// A CTA per chunk: its triplets in the order of their places in buf (to ranges of
// 2^shift places): which triplet of the chunk, and its place (over pos).
__global__ void __launch_bounds__(CB_CHUNK_THREADS) k_cb_order(int *__restrict__ pos, int n, int shift,
                                                               unsigned short *__restrict__ from)
{
    extern __shared__ int cb_order_smem[];
    int *sp = cb_order_smem;
    unsigned short *sf = reinterpret_cast<unsigned short *>(sp + CB_CHUNK);
    int *at = reinterpret_cast<int *>(sf + CB_CHUNK);
    __shared__ int scr[32];
    const long long t0 = (long long)blockIdx.x * CB_CHUNK;
    const int cnt = (int)min((long long)CB_CHUNK, n - t0);
    constexpr int PER = CB_CHUNK / CB_CHUNK_THREADS;
    int p[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j)
    {
        const int i = threadIdx.x + j * CB_CHUNK_THREADS;
        p[j] = i < cnt ? pos[t0 + i] : -1;
    }
    for (int k = threadIdx.x; k < CB_BINS; k += CB_CHUNK_THREADS) at[k] = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j)
        if (p[j] >= 0) atomicAdd(&at[p[j] >> shift], 1);
    cb_prefix<CB_BINS, CB_CHUNK_THREADS>(at, scr);
#pragma unroll
    for (int j = 0; j < PER; ++j)
        if (p[j] >= 0)
        {
            const int k = atomicAdd(&at[p[j] >> shift], 1);
            sp[k] = p[j];
            sf[k] = (unsigned short)(threadIdx.x + j * CB_CHUNK_THREADS);
        }
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += CB_CHUNK_THREADS)
    {
        pos[t0 + i] = sp[i];
        from[t0 + i] = sf[i];
    }
}

// Pass 1: a CTA per chunk.
__global__ void __launch_bounds__(CB_CHUNK_THREADS) k_cb_scatter(const double *__restrict__ x,
                                                                 const double *__restrict__ f, int n,
                                                                 const unsigned short *__restrict__ from,
                                                                 const int *__restrict__ to, double *__restrict__ buf)
{
    extern __shared__ __align__(16) double cb_smem[];
    const long long t0 = (long long)blockIdx.x * CB_CHUNK;
    const int cnt = (int)min((long long)CB_CHUNK, n - t0);
    if (f)
        for (int i = threadIdx.x; i < cnt; i += CB_CHUNK_THREADS)
            cb_smem[i] = __dmul_rn(__ldcs(f + t0 + i), __ldcs(x + t0 + i));
    else
    {
        // 16 bytes at a time where the values are aligned to them
        const int w = ((uintptr_t)x & 15) == 0 ? cnt & ~1 : 0;
        for (int i = 2 * threadIdx.x; i < w; i += 2 * CB_CHUNK_THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(cb_smem + i)),
                         "l"(x + t0 + i)
                         : "memory");
        for (int i = w + threadIdx.x; i < cnt; i += CB_CHUNK_THREADS)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(cb_smem + i)),
                         "l"(x + t0 + i)
                         : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    constexpr int U = 4;
    for (int i0 = threadIdx.x; i0 < cnt; i0 += U * CB_CHUNK_THREADS)
    {
        int fr[U], p[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
        {
            const int i = i0 + j * CB_CHUNK_THREADS;
            if (i < cnt)
            {
                fr[j] = __ldcs(from + t0 + i);
                p[j] = __ldcs(to + t0 + i);
            }
        }
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (i0 + j * CB_CHUNK_THREADS < cnt) buf[p[j]] = cb_smem[fr[j]];
    }
}

// Pass 2: a CTA per bucket, a thread per output, four outputs at a time so that their
// loads are in flight together (the first ones beside the bucket's copy).
__global__ void __launch_bounds__(CB_THREADS) k_cb_sum(const int *__restrict__ begin, const int *__restrict__ ostart,
                                                       const unsigned short *__restrict__ local,
                                                       const double *__restrict__ buf, double *__restrict__ C)
{
    extern __shared__ __align__(16) double cb_smem[];
    const int o_begin = begin[blockIdx.x], o_end = begin[blockIdx.x + 1];
    if (o_begin == o_end) return;
    const int b0 = ostart[o_begin], b1 = ostart[o_end];
    const bool fits = b1 - b0 <= CB_CAP;
    const double *sv = cb_smem + (b0 & 1);
    unsigned short *sl0 = reinterpret_cast<unsigned short *>(cb_smem + CB_CAP + 2);
    const unsigned short *sl = sl0 + (b0 & 7) - b0; // by sorted triplet
    if (threadIdx.x == 0) prefetch_l2(ostart + o_begin, ostart + o_end + 1);
    if (fits)
    {
        // 16 bytes at a time from the even place at or before the first (buf has a spare
        // value at its end)
        const double *src = buf + (b0 & ~1);
        const int pairs = (b1 - (b0 & ~1) + 1) / 2;
        for (int k = threadIdx.x; k < pairs; k += CB_THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(cb_smem + 2 * k)),
                         "l"(src + 2 * k)
                         : "memory");
        const unsigned short *lsrc = local + (b0 & ~7);
        const int octs = (b1 - (b0 & ~7) + 7) / 8;
        for (int k = threadIdx.x; k < octs; k += CB_THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(sl0 + 8 * k)),
                         "l"(lsrc + 8 * k)
                         : "memory");
    }
    constexpr int U = 4;
    bool waited = false;
    for (int o0 = o_begin + threadIdx.x; o0 < o_end || !waited; o0 += U * CB_THREADS)
    {
        int q0[U], q1[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
        {
            const int o = o0 + j * CB_THREADS;
            q0[j] = o < o_end ? __ldcs(ostart + o) : 0;
            q1[j] = o < o_end ? __ldcs(ostart + o + 1) : 0;
        }
        if (!waited)
        {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            waited = true;
        }
#pragma unroll
        for (int j = 0; j < U; ++j)
        {
            if (q0[j] >= q1[j]) continue;
            double acc = __dadd_rn(0.0, fits ? sv[sl[q0[j]]] : buf[q0[j]]);
            for (int q = q0[j] + 1; q < q1[j]; ++q) acc = __dadd_rn(acc, fits ? sv[sl[q]] : buf[q]);
            __stcs(C + o0 + j * CB_THREADS, acc);
        }
    }
}

void bucket_build(const int *ostart, const int *perm, int n, int nout, CoalesceBuckets &B, cudaStream_t s)
{
    SDL_CUDA(cudaFuncSetAttribute(k_cb_sum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CB_SMEM));
    SDL_CUDA(cudaFuncSetAttribute(k_cb_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CB_CHUNK_SMEM));
    SDL_CUDA(cudaFuncSetAttribute(k_cb_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CB_ORDER_SMEM));
    B.n = n;
    B.nb = (int)(((long long)n + CB_SPAN - 1) / CB_SPAN);
    B.nchunks = (int)(((long long)n + CB_CHUNK - 1) / CB_CHUNK);
    B.begin.reset((size_t)B.nb + 1);
    B.to.reset((size_t)n);
    B.from.reset((size_t)n);
    B.local.reset((size_t)n + 8);
    B.buf.reset((size_t)n + 1);
    const int range = CB_CHUNK * ((B.nchunks + CB_RANGES - 1) / CB_RANGES);
    int shift = 0;
    while ((n - 1) >> shift >= CB_BINS) ++shift;
    SDL_LAUNCH(k_cb_begin, B.nb / 256 + 1, 256, 0, s, ostart, nout, B.nb, B.begin.get());
    SDL_LAUNCH(k_cb_plan, B.nb, CB_THREADS, 0, s, perm, B.begin.get(), ostart, range, B.to.get(),
               B.local.get());
    SDL_LAUNCH(k_cb_order, B.nchunks, CB_CHUNK_THREADS, CB_ORDER_SMEM, s, B.to.get(), n, shift, B.from.get());
}

// Whether the plan's refill goes through buckets (the rule beside COALESCE_BUCKET_MIN).
bool takes_buckets(const int *ostart, const int *perm, int n, int nout, cudaStream_t s)
{
    if (n < COALESCE_BUCKET_MIN_HEAVY) return false;
    if (n >= (long long)COALESCE_HEAVY * nout) return true;
    if (n < COALESCE_BUCKET_MIN) return false;
    DevBuf<int> stats(2);
    SDL_CUDA(cudaMemsetAsync(stats.get(), 0, stats.bytes(), s));
    const int grid = 148 * 8;
    SDL_LAUNCH(k_cs_spread, grid, CS_THREADS, 0, s, ostart, nout, perm, n, stats.get(), stats.get() + 1);
    int h[2] = {0, 0}; // longest, lines
    SDL_CUDA(cudaMemcpyAsync(h, stats.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    SDL_CUDA(cudaStreamSynchronize(s));
    return h[0] >= COALESCE_HEAVY || h[1] > coalesce_lines(n) * (n / CS_SAMPLE);
}

} // namespace

int coalesce_build(const int *rows, const int *cols, int n, int m, int ncols, DevBuf<int> &Cp, DevBuf<int> &Ci,
                   DevBuf<int> &perm, DevBuf<int> &ostart, CoalesceBuckets &buckets, cudaStream_t s)
{
    const FreeScope frees;
    buckets = CoalesceBuckets{};
    Cp.reset((size_t)m + 1);
    perm.reset((size_t)std::max(1, n));
    if (n == 0)
    {
        SDL_CUDA(cudaMemsetAsync(Cp.get(), 0, Cp.bytes(), s));
        Ci.reset(1);
        ostart.reset(1);
        SDL_CUDA(cudaMemsetAsync(ostart.get(), 0, sizeof(int), s));
        SDL_CUDA(cudaStreamSynchronize(s));
        return 0;
    }
    auto bits_of = [](int v) {
        int b = 1;
        while (b < 31 && ((long long)1 << b) < (long long)v) ++b;
        return b;
    };
    const int col_bits = bits_of(ncols);
    DevBuf<unsigned long long> ka((size_t)n), kb((size_t)n);
    DevBuf<int> pb((size_t)n);
    if (radix_sort_coo(rows, cols, n, bits_of(m), col_bits, ka.get(), (unsigned *)perm.get(), kb.get(),
                       (unsigned *)pb.get(), s))
    {
        std::swap(ka, kb);
        std::swap(perm, pb);
    }
    // tiles of the n triplets and the one position after them
    const int ntiles = (int)((long long)n / CS_TILE + 1);
    DevBuf<int> outs((size_t)ntiles + 1), first((size_t)ntiles + 1);
    int *ngaps = outs.get() + ntiles;
    SDL_LAUNCH(k_cs_count, ntiles, CS_THREADS, 0, s, ka.get(), n, outs.get(), ngaps);
    const int nout = exclusive_scan_i32_checked(outs.get(), first.get(), ntiles, s);
    if (take_device_error(s)) fail(SDL_ERR_INTERNAL, "coalesce plan: the sort of the triplets did not finish");
    Ci.reset((size_t)std::max(1, nout));
    ostart.reset((size_t)nout + 1);
    const long long gap_cap = cs_gap_cap(m);
    DevBuf<CsGap> gaps((size_t)gap_cap);
    SDL_LAUNCH(k_cs_emit, ntiles, CS_THREADS, 0, s, ka.get(), n, m, col_bits, first.get(), ostart.get(), Ci.get(),
               Cp.get(), gaps.get(), ngaps);
    if (gap_cap)
        SDL_LAUNCH(k_cs_gaps, (unsigned)std::min(gap_cap, 148LL * 8), CS_THREADS, 0, s, gaps.get(), ngaps,
                   Cp.get());
    if (takes_buckets(ostart.get(), perm.get(), n, nout, s)) bucket_build(ostart.get(), perm.get(), n, nout, buckets, s);
    SDL_CUDA(cudaStreamSynchronize(s));
    return nout;
}

void coalesce_order_fill(const int *ostart, const int *perm, const double *x, const double *f, int nout, double *C,
                         cudaStream_t s)
{
    if (nout <= 0) return;
    SDL_LAUNCH(k_coal_fill, grid_coal(nout, 256), 256, 0, s, ostart, perm, x, f, nout, C);
}

void coalesce_bucket_fill(const CoalesceBuckets &B, const int *ostart, const double *x, const double *f, double *C,
                          cudaStream_t s)
{
    SDL_LAUNCH(k_cb_scatter, B.nchunks, CB_CHUNK_THREADS, CB_CHUNK_SMEM, s, x, f, B.n, B.from.get(), B.to.get(),
               B.buf.get());
    SDL_LAUNCH(k_cb_sum, B.nb, CB_THREADS, CB_SMEM, s, B.begin.get(), ostart, B.local.get(), B.buf.get(), C);
}

} // namespace sdl

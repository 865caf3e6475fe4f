// Stable LSD radix sort of pairs, 8 bits per pass, used once per pattern: (32-bit key, 8-byte
// payload) pairs order the terms of the rows beyond the tile budget by window, or by output;
// (row << bits | column, triplet) pairs order COO triplets. Stability keeps, inside every key,
// the input order -- upstream's visiting order. The method is that of A. Adinets and
// D. Merrill, "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs" (2022), with
// the look-back of D. Merrill and M. Garland, "Single-pass Parallel Prefix Scan with Decoupled
// Look-back" (2016); the code is this library's own.
//
// One kernel reads the keys once for the digit counts of all passes; then each pass is
// one kernel that reads and writes every pair once. A CTA takes the next tile (a ticket,
// so earlier tiles are always running or done), ranks its pairs by digit -- warps rank
// their own consecutive pairs with ballots, so equal digits keep their order -- and
// publishes its 256 digit counts; thread d then adds up digit d's counts of the tiles
// before it (decoupled look-back: each tile's word holds its own count, or the sum of
// all counts up to it once known). The tile is reordered by digit in shared memory, so
// the pairs of one digit leave for consecutive positions.
//
// What bounds it: latency at 32 warps per SM (64 registers) more than any unit: per pass of
// 10M (64-bit, 32-bit) pairs, 92 us, 55 % of the issue slots (170 instructions per 32 pairs),
// 55 % of the shared-memory pipe and 26 % of HBM are used, and a warp waits 13.8 cycles per
// instruction, for loads (2.8), fixed latencies (2.3), shared memory (2.1) and barriers (1.5).
// With a histogram kernel, a scan of all tiles' digit counts and a scatter that read the keys
// twice more, a pass took 210 us; match_any in place of the ballots: 130 us.
#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "sdl_device.cuh"
#include "sdl_internal.h"

namespace sdl {
namespace {

constexpr int RS_THREADS = 256; // one per digit value
constexpr int RS_WARPS = RS_THREADS / 32;
// Pairs of a thread, and CTAs per SM: 12 x 4 against 16 x 3, 20 x 2, 14 x 3 and 8 x 5,
// which took 1-8 % longer.
constexpr int RS_ITEMS = 12;
constexpr int RS_CTAS = 4;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_MAX_PASSES = 8;
constexpr int RS_LOOK = 4;        // tile words read at once (1: 110 us a pass, 16: 113, 4: 101)
constexpr int RS_POLLS = 1 << 22; // look-back reads of one tile word at most
constexpr int RS_ERR = 4;         // device error bit: a look-back wait ran out

// Where a pass reads its pairs.
template <class K, class V>
struct PairSource
{
    const K *keys;
    const V *vals;
    __device__ K key(int i) const { return keys[i]; }
    __device__ V val(int i) const { return vals[i]; }
};
// COO triplets: the key is row << bits | column, the payload the triplet.
struct CooSource
{
    const int *rows, *cols;
    int bits;
    __device__ unsigned long long key(int i) const
    {
        return ((unsigned long long)(unsigned)rows[i] << bits) | (unsigned)cols[i];
    }
    __device__ unsigned val(int i) const { return (unsigned)i; }
};

// The 8 bits of a key from bit `bit` on.
__device__ __forceinline__ unsigned digit(unsigned key, int bit) { return (key >> bit) & 255u; }
__device__ __forceinline__ unsigned digit(unsigned long long key, int bit)
{
    return __byte_perm((unsigned)key, (unsigned)(key >> 32), bit >> 3) & 255u; // (whole bytes)
}

template <class Src>
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(Src src, int n, int low_bit, int passes,
                                                       unsigned *__restrict__ hist)
{
    __shared__ unsigned cnt[RS_MAX_PASSES * 256];
    for (int k = threadIdx.x; k < passes * 256; k += RS_THREADS) cnt[k] = 0;
    __syncthreads();
    const int lane = lane_id();
    constexpr int U = 8; // pairs per thread whose loads are in flight together
    for (long long base = (long long)blockIdx.x * RS_THREADS * U; base < n; base += (long long)gridDim.x * RS_THREADS * U)
    {
        decltype(src.key(0)) key[U];
#pragma unroll
        for (int j = 0; j < U; ++j)
        {
            const long long i = base + j * RS_THREADS + threadIdx.x;
            key[j] = i < n ? src.key((int)i) : 0;
        }
#pragma unroll
        for (int j = 0; j < U; ++j)
        {
            const unsigned act = __ballot_sync(FULL_MASK, base + j * RS_THREADS + threadIdx.x < n);
            for (int p = 0; p < passes; ++p)
            {
                // neighbours often share their high digits: one add for the warp then
                const unsigned d = digit(key[j], low_bit + 8 * p);
                const unsigned same = __ballot_sync(FULL_MASK, d == __shfl_sync(FULL_MASK, d, 0));
                if ((same & act) == act)
                {
                    if (lane == 0 && act) atomicAdd(&cnt[p * 256 + d], __popc(act));
                }
                else if ((act >> lane) & 1u)
                    atomicAdd(&cnt[p * 256 + d], 1u);
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < passes * 256; k += RS_THREADS)
        if (cnt[k]) atomicAdd(&hist[k], cnt[k]);
}

// A tile's word per digit: the two highest bits say what the others count -- 0 nothing
// yet, 1 the tile's own pairs, 2 the pairs of all tiles up to it.
template <class W>
struct TileWord
{
    static constexpr int SHIFT = 8 * sizeof(W) - 2;
    static constexpr W MASK = (W(1) << SHIFT) - 1;
};

// The lanes whose digit is this lane's: all but those that differ from it in some bit, which
// are those whose place in the ballot of that bit does not hold this lane's bit.
__device__ __forceinline__ unsigned warp_match8(unsigned dg)
{
    unsigned differ = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b)
    {
        const unsigned mine = (unsigned)((int)(dg << (31 - b)) >> 31); // bit b, in every place
        differ |= __ballot_sync(FULL_MASK, mine) ^ mine;
    }
    return ~differ;
}

template <class K, class V>
constexpr size_t rs_smem_bytes()
{
    return (size_t)RS_TILE * (sizeof(K) + sizeof(V)) + (RS_WARPS + 1) * 256 * sizeof(int);
}

template <class K, class V, class W, class Src>
__global__ void __launch_bounds__(RS_THREADS, RS_CTAS) k_rs_pass(Src src, int n, int bit,
                                                                  const unsigned *__restrict__ hist, W *words,
                                                                  int *__restrict__ ticket, K *__restrict__ okeys,
                                                                  V *__restrict__ ovals, int *__restrict__ err)
{
    extern __shared__ __align__(16) unsigned char rs_smem[];
    K *sk = reinterpret_cast<K *>(rs_smem);
    V *sv = reinterpret_cast<V *>(sk + RS_TILE);
    int(*wc)[256] = reinterpret_cast<int(*)[256]>(sv + RS_TILE);
    int *gbase = &wc[RS_WARPS][0];
    __shared__ int tile_sh, scr[32];
    const int lane = lane_id(), w = threadIdx.x >> 5, d = threadIdx.x;
    if (threadIdx.x == 0) tile_sh = atomicAdd(ticket, 1);
    for (int k = threadIdx.x; k < RS_WARPS * 256; k += RS_THREADS) (&wc[0][0])[k] = 0;
    const int count = (int)hist[d];
    const int dstart = block_incl_scan_int(count, scr) - count; // pairs of smaller digits
    const int tile = tile_sh;
    const long long tbase = (long long)tile * RS_TILE;
    const int tn = (int)min((long long)RS_TILE, (long long)n - tbase);
    // the warp's pairs, 32 consecutive ones at a time; places past the last pair count as
    // the largest key, so they rank behind every pair of the tile
    const int first = w * 32 * RS_ITEMS + lane; // in the tile
    K key[RS_ITEMS];
    V val[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) key[j] = first + 32 * j < tn ? src.key((int)tbase + first + 32 * j) : ~K(0);
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) val[j] = first + 32 * j < tn ? src.val((int)tbase + first + 32 * j) : V{};
    // rank inside the warp: the pairs of the digit counted so far, and those of earlier lanes
    int rank[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j)
    {
        const unsigned dg = digit(key[j], bit);
        int *c = &wc[w][dg];
        const unsigned grp = warp_match8(dg);
        rank[j] = *c + __popc(grp & lanemask_lt());
        __syncwarp();
        if (lane == 31 - __clz(grp)) *c = rank[j] + 1;
        __syncwarp();
    }
    __syncthreads();
    // digit d: the warps' counts become offsets inside the tile's run of d
    int total = 0;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww)
    {
        const int c = wc[ww][d];
        wc[ww][d] = total;
        total += c;
    }
    if (d == (int)digit(~K(0), bit)) total -= RS_TILE - tn;
    volatile W *word = words + (size_t)tile * 256 + d;
    *word = (W(tile ? 1 : 2) << TileWord<W>::SHIFT) | W(total);
    const int lstart = block_incl_scan_int(total, scr) - total; // (ends with a barrier)
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) wc[ww][d] += lstart;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j)
    {
        const int pos = wc[w][digit(key[j], bit)] + rank[j];
        sk[pos] = key[j];
        sv[pos] = val[j];
    }
    // digit d's pairs in the tiles before this one, the words of RS_LOOK tiles at a time
    W before = 0;
    for (int t = tile - 1; t >= 0;)
    {
        volatile const W *tw = words + (size_t)t * 256 + d;
        W x[RS_LOOK];
#pragma unroll
        for (int j = 0; j < RS_LOOK; ++j) x[j] = tw[-256 * min(j, t)];
        bool done = false;
#pragma unroll
        for (int j = 0; j < RS_LOOK; ++j)
        {
            if (done || j > t) continue;
            for (int it = 0; !(x[j] >> TileWord<W>::SHIFT) && it < RS_POLLS; ++it)
            {
                if (it > 64) __nanosleep(32);
                x[j] = tw[-256 * j];
            }
            if (!(x[j] >> TileWord<W>::SHIFT)) atomicOr(err, RS_ERR);
            before += x[j] & TileWord<W>::MASK;
            done = x[j] >> TileWord<W>::SHIFT != 1; // all tiles counted (or the wait ran out)
        }
        if (done) break;
        t -= RS_LOOK;
    }
    if (tile) *word = (W(2) << TileWord<W>::SHIFT) | (before + W(total));
    gbase[d] = dstart + (int)before - lstart;
    __syncthreads();
    for (int j = threadIdx.x; j < tn; j += RS_THREADS)
    {
        const K k = sk[j];
        const unsigned pos = (unsigned)(gbase[digit(k, bit)] + j);
        if (pos < (unsigned)n) // (always, unless a look-back wait ran out)
        {
            okeys[pos] = k;
            ovals[pos] = sv[j];
        }
    }
}

template <class K, class V, class W, class Src>
void rs_pass(const Src &src, int n, int bit, const unsigned *hist, W *words, int *ticket, K *okeys, V *ovals,
             int ntiles, cudaStream_t s)
{
    const auto kern = k_rs_pass<K, V, W, Src>;
    {
        // the kernel attribute is per device: set it once for each device the process
        // sorts on (plans may be built from several host threads)
        static std::mutex mu;
        static std::set<int> done;
        int dev = 0;
        SDL_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (done.insert(dev).second)
            SDL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)rs_smem_bytes<K, V>()));
    }
    SDL_CUDA(cudaMemsetAsync(words, 0, (size_t)ntiles * 256 * sizeof(W), s));
    SDL_LAUNCH(kern, ntiles, RS_THREADS, (rs_smem_bytes<K, V>()), s, src, n, bit, hist, words, ticket, okeys, ovals,
               runtime().d_error);
}

// Sorts the n pairs of `first` by `bits` bits of the key from low_bit on (a multiple of 8
// for 64-bit keys): pass 0 writes them to
// (kb, vb), the next to (ka, va), and so on. True if they end in (kb, vb).
template <class K, class V, class W, class Src>
bool rs_sort(const Src &first, K *ka, V *va, K *kb, V *vb, int n, int low_bit, int bits,
             cudaStream_t s)
{
    const int ntiles = (int)(((long long)n + RS_TILE - 1) / RS_TILE);
    const int passes = std::max(1, (bits + 7) / 8);
    DevBuf<unsigned> hist(RS_MAX_PASSES * 256 + RS_MAX_PASSES); // the digit counts, then the passes' tickets
    SDL_CUDA(cudaMemsetAsync(hist.get(), 0, hist.bytes(), s));
    DevBuf<W> words((size_t)ntiles * 256);
    const int grid = std::min(ntiles, runtime().num_sms * 8);
    SDL_LAUNCH(k_rs_hist<Src>, grid, RS_THREADS, 0, s, first, n, low_bit, passes, hist.get());
    bool in_b = false;
    for (int p = 0; p < passes; ++p, in_b = !in_b)
    {
        int *ticket = reinterpret_cast<int *>(hist.get() + RS_MAX_PASSES * 256) + p;
        K *ok = in_b ? ka : kb;
        V *ov = in_b ? va : vb;
        if (p == 0)
            rs_pass<K, V, W>(first, n, low_bit, hist.get(), words.get(), ticket, ok, ov, ntiles, s);
        else
            rs_pass<K, V, W>(PairSource<K, V>{in_b ? kb : ka, in_b ? vb : va}, n,
                             low_bit + 8 * p, hist.get() + 256 * p,
                             words.get(), ticket, ok, ov, ntiles, s);
    }
    return in_b;
}

constexpr int RS_WORD32_MAX = 1 << 30; // pairs that a 32-bit tile word can count

} // namespace

bool radix_sort_pairs(unsigned *keys, uint2 *vals, unsigned *keys_tmp, uint2 *vals_tmp, int n, int low_bit,
                      int bits, cudaStream_t s)
{
    if (n <= 0) return false;
    const PairSource<unsigned, uint2> src{keys, vals};
    return n < RS_WORD32_MAX
               ? rs_sort<unsigned, uint2, unsigned>(src, keys, vals, keys_tmp, vals_tmp, n, low_bit, bits, s)
               : rs_sort<unsigned, uint2, unsigned long long>(src, keys, vals, keys_tmp, vals_tmp, n, low_bit, bits,
                                                              s);
}

bool radix_sort_coo(const int *rows, const int *cols, int n, int row_bits, int col_bits, unsigned long long *ka,
                    unsigned *va, unsigned long long *kb, unsigned *vb, cudaStream_t s)
{
    const CooSource src{rows, cols, col_bits};
    const int bits = row_bits + col_bits;
    return n < RS_WORD32_MAX
               ? rs_sort<unsigned long long, unsigned, unsigned>(src, ka, va, kb, vb, n, 0, bits, s)
               : rs_sort<unsigned long long, unsigned, unsigned long long>(src, ka, va, kb, vb, n, 0, bits, s);
}

} // namespace sdl

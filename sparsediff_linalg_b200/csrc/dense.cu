// Dense blocks times a sparse CSR on the GPU: C_k = B_k S[col_perm_k, :]
// (upstream src/permuted_dense/permuted_dense_linalg.c:313-430 BA_pd_csr_*,
// src/stacked_pd/stacked_pd_linalg.c:657-671 BA_spd_csr_*).
//
// Upstream's structure: C_k's columns are the union of the patterns of S's rows
// col_perm_k (ascending), and the fill sums, for every output (i, c), the terms
// B_k[i, r] * S[col_perm_k[r], c] over the compact CSC of S[col_perm_k, :] in its
// order (r ascending), from +0.0, one rounding per product and per sum. Here a
// warp computes whole output columns with its lanes on the block's rows, reading
// the block's columns contiguously from a transposed copy, and each output is
// summed in exactly that order (__dmul_rn / __dadd_rn: no FMA, as the upstream
// build has none).
#include <algorithm>
#include <climits>
#include <map>

#include "capi_common.h"
#include "dense_plan.h"
#include "sdl_device.cuh"

namespace sdl {
namespace {

int grid_cap(long long work_items, int per_block, int cap)
{
    long long g = (work_items + per_block - 1) / per_block;
    return (int)std::max<long long>(1, std::min<long long>(g, cap));
}

constexpr int BC_THREADS = 256;

// What a fill lays out before its products, in one launch (the two halves do not depend
// on each other): the first `gather_ctas` CTAs gather S.x into compact order, the others
// take a 32 x 32 tile each of the transposed copies BT of the source blocks (n0 x m0
// row-major, so that one column of a block is contiguous). The tiles are listed: a grid of
// the largest block's tiles for every block was mostly CTAs without work where shapes
// differ (one block of 2000 x 400 beside 3000 of 8 x 8: the fill 2.13 ms), and overran the
// launch limits beside a few large blocks. A thread's four loads are in flight together (2400
// blocks of 64 x 128: 86 -> 67 us).
__global__ void __launch_bounds__(BC_THREADS) k_blocks_csr_inputs(
    const int *__restrict__ pos, const double *__restrict__ Sx, long long n, double *__restrict__ vals,
    int gather_ctas, const BlkTrTile *__restrict__ tr, const double *__restrict__ B, double *__restrict__ BT)
{
    __shared__ double t[32][33];
    if ((int)blockIdx.x < gather_ctas)
    {
        for (long long d = blockIdx.x * (long long)blockDim.x + threadIdx.x; d < n;
             d += (long long)gather_ctas * blockDim.x)
            vals[d] = Sx[pos[d]];
        return;
    }
    const BlkTrTile D = tr[blockIdx.x - gather_ctas];
    const int i0 = D.i0, r0 = D.r0;
    const double *src = B + D.b_off;
    double *dst = BT + D.b_off;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    constexpr int ROWS = 32 / (BC_THREADS / 32); // of a thread
#pragma unroll
    for (int j = 0; j < ROWS; ++j)
    {
        const int y = ty + j * (32 / ROWS), i = i0 + y, r = r0 + tx;
        if (i < D.m0 && r < D.n0_B) t[y][tx] = src[(long long)i * D.n0_B + r];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROWS; ++j)
    {
        const int y = ty + j * (32 / ROWS), r = r0 + y, i = i0 + tx;
        if (r < D.n0_B && i < D.m0) dst[(long long)r * D.m0 + i] = t[tx][y];
    }
}

// ------------------------------------------------------------------ resident slabs
// A CTA keeps a slab of its block (up to 64 rows by n0 columns, at most 128 KB,
// transposed) in shared memory, and its warps take units of 16 output columns one after
// the other, with no barrier between them.
//
// What bounds it: every output and term takes 8 bytes of the block from shared memory
// (64 blocks of 64 x 256 times 256 x 100000 with 6 per column: 19.7 GB, 0.53 ms at 128
// bytes a clock and SM; 0.68 ms measured without the stores), and C is written at 4.5
// TB/s (0.73 ms without the sums). So
// * the reads are conflict-free 16-byte ones: four lanes (p = lane & 3) share a column
//   and read 64 bytes of it, two columns at a time use the two halves of a 128-byte
//   line (odd columns take the halves in the other order), and a term's {value, column}
//   record is one read for all 16 Q rows;
// * the sums leave from registers, eight columns of four rows at a time, as whole 32-byte
//   sectors of C: a lane's rows are those with row % 4 == p, so they share an alignment
//   in C whatever n0_C is, and the lane's columns start up to 3 early to meet it. With
//   the segments where they fell, rows of odd length took 1.5 times as long (5 blocks of
//   50 x 256 times 256 x 99991 with 5 per column: 115 -> 80 us).
// The fill above: 1.93 -> 1.07 ms against k_blocks_csr (32 x 64 tiles through shared
// memory, the block read from L1). Through a warp-private 32 x 16 tile instead of
// registers it took 1.15 ms, with 32 rows a pass 1.11-1.16 ms.
// Blocks of more than RS_N0_MAX columns stay with k_blocks_csr: slabs of only 16 rows
// spread a record's read too thin (8 blocks of 64 x 1000 with 40 per column: 711 against
// 601 us; with slabs of 32 rows, n0 = 512 and 6 per column, 96 against 143 us). Up to there
// the slabs hold their lead at every density (16 blocks of 64 x 256 times 256 x 8000, us in
// slabs and in tiles: 36 and 36 at 1 per column, 58 and 85 at 12, 130 and 202 at 40, 636 and
// 1011 at 250), also where a unit's records are staged in parts or read from global memory.
constexpr int RS_WARPS = 16; // warps of a CTA
constexpr int RS_COLS = 16;  // output columns of a unit
constexpr int RS_SHIFT = 3;  // columns a unit may start early, to meet C's 32-byte sectors
constexpr int RS_REC = 128;  // records a warp stages at once
// The CTAs share the units out by their cost: a unit's stores and fixed work take about as
// long as 128 terms (16 blocks of 64 x 256 times 256 x 8000: 38 us at one entry per column,
// 58 at 12, 130 at 40, 261 at 100). With an even share of the units each, a tenth of the
// columns at 100 entries and the others at 2 took 238 us, 64 us so (147 by k_blocks_csr).
constexpr int RS_UNIT_COST = 128;
// Where a CTA would have several slabs in turn (more than RS_FEW_SLABS per SM in all), a slab's
// load has to pay: a block stays with k_blocks_csr if its columns and entries are too few for
// that (rs_pays). The line is fitted to both kernels' times over 600 and 2400 blocks of 16 x
// 100 to 64 x 256 by 14 to 400 columns of 1 to 20 entries: within 0.6 % of the better one on
// average. 600 blocks of 64 x 64: in slabs 27 us at 14 columns of 6 (19 us in tiles), 29 at
// 60 (29), 64 at 400 (95); of 64 x 256: 78 (54), 82 (66), 127 (137).
constexpr int RS_FEW_SLABS = 1;
constexpr bool rs_pays(int n0, int q, long long cols, long long entries)
{
    const long long load = 4LL * n0 + 300 + 30 * entries / cols;
    return 4 * cols + entries >= (q == 1 ? load / 2 : load); // (slabs of 16 rows: two CTAs per SM)
}
constexpr int RS_SLAB_BYTES = 128 * 1024;
constexpr int RS_N0_MAX = RS_SLAB_BYTES / (32 * 8);
constexpr int RS_WARP_BYTES = 2 * RS_REC * 16; // two units' records

// One term of NQ 16-row groups: acc[4 k + 2 h + b] is row 16 k + 8 (h ^ sw) + 4 b + p.
template <int NQ>
__device__ __forceinline__ void rs_term(const char *col, int sw64, double v, double (&acc)[4 * NQ])
{
#pragma unroll
    for (int k = 0; k < NQ; ++k)
    {
        const double2 b0 = *reinterpret_cast<const double2 *>(col + 128 * k + sw64);
        const double2 b1 = *reinterpret_cast<const double2 *>(col + 128 * k + (sw64 ^ 64));
        acc[4 * k] = __dadd_rn(acc[4 * k], __dmul_rn(b0.x, v));
        acc[4 * k + 1] = __dadd_rn(acc[4 * k + 1], __dmul_rn(b0.y, v));
        acc[4 * k + 2] = __dadd_rn(acc[4 * k + 2], __dmul_rn(b1.x, v));
        acc[4 * k + 3] = __dadd_rn(acc[4 * k + 3], __dmul_rn(b1.y, v));
    }
}

// Starts copying the records of entries [d0, d1) (at most RS_REC) into `recs`: the
// value in the first 8 bytes, the block column in the next 4.
__device__ __forceinline__ void rs_stage(int4 *recs, int d0, int d1, const int *__restrict__ rows,
                                         const double *__restrict__ vals)
{
    for (int d = d0 + lane_id(); d < d1; d += 32)
    {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(recs + (d - d0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(vals + d) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 8), "l"(rows + d) : "memory");
    }
}

// One unit: the columns from c0 + shift on, 16 of them, of a slab of NQ 16-row groups.
// `off`: lane j holds the first entry of column c0 - RS_SHIFT + j. `recs` holds the
// unit's records when `whole`; else they are staged eight columns at a time, and read
// from rows / vals where even those exceed RS_REC.
template <int NQ>
__device__ __forceinline__ void rs_unit(const char *Bq, int4 *recs, bool whole, int off, int shift, int c0, int n0_C,
                                        const int *__restrict__ rows, const double *__restrict__ vals,
                                        double *__restrict__ C, int nr)
{
    constexpr int row_bytes = 16 * NQ * 8;
    const int lane = lane_id(), p = lane & 3, cl = lane >> 2, sw64 = (cl & 1) * 64;
    const int d0 = __shfl_sync(FULL_MASK, off, 0);
#pragma unroll
    for (int g = 0; g < RS_COLS / 8; ++g)
    {
        const int j = 8 * g + cl + RS_SHIFT + shift, c = c0 - RS_SHIFT + j;
        const int s = __shfl_sync(FULL_MASK, off, j);
        const int e = __shfl_sync(FULL_MASK, off, j + 1);
        int base = d0;
        bool staged = whole;
        if (!whole)
        {
            base = __shfl_sync(FULL_MASK, off, 8 * g);
            const int ge = __shfl_sync(FULL_MASK, off, 8 * g + 8 + RS_SHIFT);
            staged = ge - base <= RS_REC;
            __syncwarp();
            if (staged)
            {
                rs_stage(recs, base, ge, rows, vals);
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            __syncwarp();
        }
        double acc[4 * NQ];
#pragma unroll
        for (int k = 0; k < 4 * NQ; ++k) acc[k] = 0.0;
        if (staged)
        {
#pragma unroll 2
            for (int d = s; d < e; ++d)
            {
                const int4 r = recs[d - base];
                rs_term<NQ>(Bq + r.z * row_bytes, sw64, __hiloint2double(r.y, r.x), acc);
            }
        }
        else
            for (int d = s; d < e; ++d) rs_term<NQ>(Bq + rows[d] * row_bytes, sw64, vals[d], acc);
        if (c >= 0 && c < n0_C)
        {
            double *o = C + c + (long long)p * n0_C;
#pragma unroll
            for (int q = 0; q < 4 * NQ; ++q, o += 4 * (long long)n0_C)
            {
                // even columns hold rows 0-7 of a group first, odd columns rows 8-15
                const double x = sw64 ? acc[q ^ 2] : acc[q];
                if (4 * q + p < nr) __stcs(o, x);
            }
        }
    }
}

// Slabs of 16 * (Q - 1) + 1 .. 16 * Q rows.
template <int Q>
__global__ void __launch_bounds__(RS_WARPS * 32, Q <= 2 ? 2 : 1) k_blocks_csr_slabs(
    const BlkSlab *__restrict__ slabs, const BlkShare *__restrict__ shares, int slab_smem,
    const int *__restrict__ cp_all, const int *__restrict__ rows_all,
    const double *__restrict__ vals_all, const double *__restrict__ BT_vals, double *__restrict__ C_vals)
{
    extern __shared__ __align__(16) unsigned char rs_smem[];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    double *Bs = reinterpret_cast<double *>(rs_smem);
    int4 *recs = reinterpret_cast<int4 *>(rs_smem + slab_smem + warp * RS_WARP_BYTES);
    // this CTA's share of the units, contiguous: it loads few slabs
    long long u = shares[blockIdx.x].unit;
    const long long u_end = shares[blockIdx.x + 1].unit;
    for (int si = shares[blockIdx.x].slab; u < u_end; ++si)
    {
        const BlkSlab sl = slabs[si];
        const BlkDesc &D = sl.D;
        constexpr int ld = 16 * Q;
        const int n_units = (int)(min(sl.unit_end, u_end) - u);
        const int u_first = (int)(u - sl.unit_begin);
        const int *cp = cp_all + D.cp_off;
        const int *rows = rows_all + D.d_off;
        const double *vals = vals_all + D.d_off;
        // column offsets of the warp's unit k: lane j holds the first entry of column j - RS_SHIFT
        const auto offs = [&](int k) {
            const int c = (u_first + k) * RS_COLS - RS_SHIFT + lane;
            return k < n_units ? cp[max(0, min(c, D.n0_C))] : 0;
        };
        int off = offs(warp), off_next = offs(warp + RS_WARPS), buf = 0;
        // the slab, transposed and padded with zero rows to whole 16-row groups
        __syncthreads();
        const double *src = BT_vals + D.b_off + sl.i0;
        for (int x0 = threadIdx.x; x0 < D.n0_B * ld; x0 += 8 * RS_WARPS * 32)
        {
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                const int x = x0 + j * RS_WARPS * 32, r = x / ld, y = x - r * ld;
                const int i = (y & ~7) | ((y & 1) << 2) | ((y >> 1) & 3); // rows i and i + 4 side by side
                v[j] = r < D.n0_B && i < sl.nrow ? src[(long long)r * D.m0 + i] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                const int x = x0 + j * RS_WARPS * 32;
                if (x < D.n0_B * ld) Bs[x] = v[j];
            }
        }
        __syncthreads();
        const char *Bl = reinterpret_cast<const char *>(Bs) + (lane & 3) * 16;
        double *Cs = C_vals + D.c_off + (long long)sl.i0 * D.n0_C;
        // the rows of a lane (i mod 4 alike) have the same alignment in C: its columns start
        // 0 .. RS_SHIFT early, so that every 8 columns of a row are two whole 32-byte sectors
        const int shift = -(int)((((uintptr_t)Cs >> 3) + (unsigned long long)(lane & 3) * D.n0_C) & 3);
        // a unit's records are copied in while the unit before it is computed, and its
        // column offsets are read one unit earlier still
        const auto stage = [&](int off, int4 *to) {
            const int d0 = __shfl_sync(FULL_MASK, off, 0), d1 = __shfl_sync(FULL_MASK, off, RS_COLS + RS_SHIFT);
            const bool whole = d1 - d0 <= RS_REC;
            if (whole) rs_stage(to, d0, d1, rows, vals);
            asm volatile("cp.async.commit_group;" ::: "memory");
            return whole;
        };
        bool whole = stage(off, recs);
        for (int k = warp; k < n_units; k += RS_WARPS)
        {
            __syncwarp(); // the other buffer's unit is done with it
            const bool whole_next = stage(off_next, recs + (buf ^ RS_REC));
            const int off_after = offs(k + 2 * RS_WARPS);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            rs_unit<Q>(Bl, recs + buf, whole, off, shift, (u_first + k) * RS_COLS, D.n0_C, rows, vals, Cs, sl.nrow);
            off = off_next;
            off_next = off_after;
            whole = whole_next;
            buf ^= RS_REC;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        u += n_units;
    }
}

using SlabKernel = void (*)(const BlkSlab *, const BlkShare *, int, const int *, const int *, const double *,
                            const double *, double *);
// The first unit of each CTA, of at most `grid`, and one past the last (cp: the compact CSCs'
// column offsets). A CTA begins where the cost of the units before reaches its part of the
// whole. Where that is less than a unit per warp, a second slab would cost it more than its
// units do: each slab is then shared out among CTAs of its own (16 blocks of 64 x 256 times
// 256 x 500: 16.6 -> 12.7 us).
std::vector<BlkShare> share_units(const std::vector<BlkSlab> &slabs, const int *cp, int grid)
{
    // cost of the slab's first k units, and of all of them
    const auto cost = [&](const BlkSlab &S, long long k) {
        return k * RS_UNIT_COST + cp[S.D.cp_off + std::min<long long>(k * RS_COLS, S.D.n0_C)];
    };
    const auto all = [&](const BlkSlab &S) { return cost(S, S.unit_end - S.unit_begin); };
    // the slab's first unit that `from` or more cost comes before
    const auto unit_at = [&](const BlkSlab &S, long long from) {
        long long lo = 0, hi = S.unit_end - S.unit_begin;
        while (lo < hi)
        {
            const long long mid = (lo + hi) / 2;
            if (cost(S, mid) < from)
                lo = mid + 1;
            else
                hi = mid;
        }
        return S.unit_begin + lo;
    };
    long long total = 0;
    for (const BlkSlab &S : slabs) total += all(S);
    const auto part = [](long long whole, long long k, long long n) { return (long long)((__int128)whole * k / n); };
    std::vector<BlkShare> out;
    if ((long long)slabs.size() <= grid && slabs.back().unit_end < (long long)grid * RS_WARPS)
    {
        for (size_t si = 0; si < slabs.size(); ++si)
        {
            const BlkSlab &S = slabs[si];
            const long long n = std::max(1LL, std::min(part(grid, all(S), total), S.unit_end - S.unit_begin));
            for (long long k = 0; k < n; ++k) out.push_back(BlkShare{unit_at(S, part(all(S), k, n)), (int)si, 0});
        }
    }
    else
    {
        size_t si = 0;
        long long before = 0; // cost of the slabs before slab si
        for (int b = 0; b < grid; ++b)
        {
            const long long from = part(total, b, grid);
            for (; before + all(slabs[si]) <= from; ++si) before += all(slabs[si]);
            const long long unit = unit_at(slabs[si], from - before);
            out.push_back(BlkShare{unit, (int)si + (unit == slabs[si].unit_end), 0});
        }
    }
    out.push_back(BlkShare{slabs.back().unit_end, (int)slabs.size(), 0});
    return out;
}
SlabKernel slab_kernel(int q)
{
    return q == 1 ? k_blocks_csr_slabs<1> : q == 2 ? k_blocks_csr_slabs<2> : q == 3 ? k_blocks_csr_slabs<3> : k_blocks_csr_slabs<4>;
}

// ------------------------------------------------------------------ wider blocks
#ifndef SDL_BC_COLS
#define SDL_BC_COLS 32
#endif
constexpr int BC_COLS = SDL_BC_COLS; // output columns of a CTA tile
constexpr int BC_ROWS = 64; // block rows per pass (two per lane)

// One CTA: output columns [c0, c0 + 32) of one block; each warp takes four columns
// one after the other, its lanes the block's rows (two per lane): every term of a
// column is a broadcast (row r of the block, value of S) times a contiguous read of
// column r of the block (BT). The 64 x 32 results go through shared memory and are
// written row by row, 256 bytes per row.
__global__ void __launch_bounds__(BC_THREADS) k_blocks_csr(const BlkTile *__restrict__ tiles,
                                                           const BlkDesc *__restrict__ descs,
                                                           const int *__restrict__ cp_all,
                                                           const int *__restrict__ rows_all,
                                                           const double *__restrict__ vals_all,
                                                           const double *__restrict__ BT_vals,
                                                           double *__restrict__ C_vals)
{
    __shared__ double tile[BC_ROWS][BC_COLS + 1];
    const BlkTile t = tiles[blockIdx.x];
    const BlkDesc D = descs[t.blk];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int *cp = cp_all + D.cp_off;
    const int *rows = rows_all + D.d_off;
    const double *vals = vals_all + D.d_off;
    const double *BT = BT_vals + D.b_off;
    const int ncol = min(BC_COLS, D.n0_C - t.c0);
    for (int i0 = 0; i0 < D.m0; i0 += BC_ROWS)
    {
        const int ia = i0 + lane, ib = i0 + 32 + lane;
        for (int cl = warp; cl < BC_COLS; cl += BC_THREADS / 32)
        {
            double a0 = 0.0, a1 = 0.0;
            if (cl < ncol)
            {
                const int c = t.c0 + cl;
                const int d1 = cp[c + 1];
                for (int d = cp[c]; d < d1; ++d)
                {
                    const double *col = BT + (long long)rows[d] * D.m0;
                    const double v = vals[d];
                    if (ia < D.m0) a0 = __dadd_rn(a0, __dmul_rn(col[ia], v));
                    if (ib < D.m0) a1 = __dadd_rn(a1, __dmul_rn(col[ib], v));
                }
            }
            tile[lane][cl] = a0;
            tile[32 + lane][cl] = a1;
        }
        __syncthreads();
        const int nrow = min(BC_ROWS, D.m0 - i0);
        double *C = C_vals + D.c_off + (long long)i0 * D.n0_C + t.c0;
        for (int e = threadIdx.x; e < nrow * BC_COLS; e += BC_THREADS)
        {
            const int ri = e / BC_COLS, cl = e % BC_COLS;
            if (cl < ncol) C[(long long)ri * D.n0_C + cl] = tile[ri][cl];
        }
        __syncthreads();
    }
}

} // namespace

std::unique_ptr<BlocksCsrPlan> blocks_csr_build(int n_src, const int *m0, const int *n0,
                                                const int *const *col_perm, const int *Sp, const int *Si,
                                                int S_m, int S_n, bool keep_empty, cudaStream_t s)
{
    if (n_src < 0 || S_m < 0 || S_n < 0) fail(SDL_ERR_INVALID, "blocks x CSR: negative size");
    auto P = std::make_unique<BlocksCsrPlan>();
    P->S_m = S_m;
    P->S_n = S_n;
    P->S_nnz = S_m ? Sp[S_m] : 0;
    P->n_src = n_src;
    // compact CSCs, one per distinct col_perm (upstream builds one per block)
    struct Csc
    {
        std::vector<int> col_perm_C, cp, rows, pos;
        long long cp_off = 0, d_off = 0;
    };
    std::map<std::vector<int>, int> seen;
    std::vector<Csc> cscs;
    std::vector<int> csc_of(n_src);
    std::vector<int> mark(std::max(1, S_n));
    for (int k = 0; k < n_src; ++k)
    {
        if (m0[k] < 0 || n0[k] < 0) fail(SDL_ERR_INVALID, "blocks x CSR: negative block shape");
        std::vector<int> key(col_perm[k], col_perm[k] + n0[k]);
        for (int r = 0; r < n0[k]; ++r)
            if (key[r] < 0 || key[r] >= S_m || (r && key[r] <= key[r - 1]))
                fail(SDL_ERR_INVALID, "blocks x CSR: a col_perm is not strictly increasing rows of S");
        auto it = seen.find(key);
        if (it != seen.end())
        {
            csc_of[k] = it->second;
            continue;
        }
        Csc cc;
        std::fill(mark.begin(), mark.end(), -1);
        long long nnz_K = 0;
        for (int row : key)
        {
            for (int q = Sp[row]; q < Sp[row + 1]; ++q)
            {
                if (Si[q] < 0 || Si[q] >= S_n) fail(SDL_ERR_INVALID, "blocks x CSR: column index of S out of range");
                mark[Si[q]] = 0;
            }
            nnz_K += Sp[row + 1] - Sp[row];
        }
        if (nnz_K > INT_MAX) fail(SDL_ERR_OVERFLOW, "blocks x CSR: compact CSC exceeds INT_MAX entries");
        for (int j = 0; j < S_n; ++j)
            if (mark[j] >= 0)
            {
                mark[j] = (int)cc.col_perm_C.size();
                cc.col_perm_C.push_back(j);
            }
        const int n0C = (int)cc.col_perm_C.size();
        cc.cp.assign((size_t)n0C + 1, 0);
        for (int row : key)
            for (int q = Sp[row]; q < Sp[row + 1]; ++q) cc.cp[mark[Si[q]] + 1]++;
        for (int c = 0; c < n0C; ++c) cc.cp[c + 1] += cc.cp[c];
        cc.rows.resize((size_t)nnz_K);
        cc.pos.resize((size_t)nnz_K);
        std::vector<int> next(cc.cp.begin(), cc.cp.end() - 1);
        for (int r = 0; r < (int)key.size(); ++r)
            for (int q = Sp[key[r]]; q < Sp[key[r] + 1]; ++q)
            {
                const int dd = next[mark[Si[q]]]++;
                cc.rows[dd] = r;
                cc.pos[dd] = q;
            }
        csc_of[k] = (int)cscs.size();
        seen.emplace(std::move(key), csc_of[k]);
        cscs.push_back(std::move(cc));
    }
    long long cp_total = 0;
    for (Csc &cc : cscs)
    {
        cc.cp_off = cp_total;
        cc.d_off = P->d_total;
        cp_total += (long long)cc.cp.size();
        P->d_total += (long long)cc.rows.size();
    }
    std::vector<int> h_cp((size_t)std::max<long long>(1, cp_total)), h_rows((size_t)std::max<long long>(1, P->d_total)),
        h_pos((size_t)std::max<long long>(1, P->d_total));
    for (const Csc &cc : cscs)
    {
        std::copy(cc.cp.begin(), cc.cp.end(), h_cp.begin() + cc.cp_off);
        std::copy(cc.rows.begin(), cc.rows.end(), h_rows.begin() + cc.d_off);
        std::copy(cc.pos.begin(), cc.pos.end(), h_pos.begin() + cc.d_off);
    }
    // A slab takes up to 64 rows and RS_SLAB_BYTES, a block's rows shared out evenly.
    struct SlabCut
    {
        long long n; // its slabs
        int per;     // rows of each
        bool pays;
    };
    const auto slab_cut = [&](int k) {
        const Csc &cc = cscs[csc_of[k]];
        if (n0[k] > RS_N0_MAX || cc.col_perm_C.empty() || m0[k] == 0) return SlabCut{0, 0, false};
        const int qmax = std::max(1, std::min(SLAB_Q, RS_SLAB_BYTES / (16 * 8 * std::max(1, n0[k]))));
        const long long n = ((long long)m0[k] + 16 * qmax - 1) / (16 * qmax);
        const int per = (int)((m0[k] + n - 1) / n);
        return SlabCut{n, per, rs_pays(n0[k], (per + 15) / 16, (long long)cc.col_perm_C.size(), (long long)cc.rows.size())};
    };
    long long in_turn = 0; // slabs whose load does not pay
    for (int k = 0; k < n_src; ++k)
        if (const SlabCut c = slab_cut(k); !c.pays) in_turn += c.n;
    const bool small_in_tiles = in_turn > RS_FEW_SLABS * (long long)runtime().num_sms;
    // output blocks and their work tiles
    std::vector<BlkDesc> descs;
    std::vector<BlkTile> tiles;
    std::vector<BlkSlab> slabs[SLAB_Q];
    long long b_off = 0;
    for (int k = 0; k < n_src; ++k)
    {
        const Csc &cc = cscs[csc_of[k]];
        const int n0C = (int)cc.col_perm_C.size();
        const long long bk = (long long)m0[k] * n0[k];
        if ((n0C > 0 && m0[k] > 0) || keep_empty)
        {
            if ((long long)m0[k] * n0C > INT_MAX) fail(SDL_ERR_OVERFLOW, "blocks x CSR: output block exceeds INT_MAX values");
            BlkDesc D{};
            D.b_off = b_off;
            D.c_off = P->c_total;
            D.cp_off = cc.cp_off;
            D.d_off = cc.d_off;
            D.m0 = m0[k];
            D.n0_B = n0[k];
            D.n0_C = n0C;
            const int blk = (int)descs.size();
            const SlabCut cut = slab_cut(k);
            if (n0[k] > RS_N0_MAX || (small_in_tiles && !cut.pays))
                for (int c0 = 0; c0 < n0C && m0[k] > 0; c0 += BC_COLS) tiles.push_back(BlkTile{blk, c0});
            else
                for (long long i0 = 0; cut.n > 0 && i0 < m0[k]; i0 += cut.per)
                {
                    const int nrow = (int)std::min<long long>(cut.per, m0[k] - i0), q = (nrow + 15) / 16;
                    auto &cls = P->slab_cls[q - 1];
                    const long long u0 = cls.units;
                    cls.units += (n0C + RS_SHIFT + RS_COLS - 1) / RS_COLS;
                    slabs[q - 1].push_back(BlkSlab{D, (int)i0, nrow, u0, cls.units});
                    cls.smem = std::max(cls.smem, n0[k] * q * 16 * 8);
                }
            descs.push_back(D);
            P->src.push_back(k);
            P->col_perm.push_back(cc.col_perm_C);
            P->m0.push_back(m0[k]);
            P->n0_C.push_back(n0C);
            P->c_total += (long long)m0[k] * n0C;
        }
        b_off += bk;
    }
    P->b_total = b_off;
    P->ntiles = (int)tiles.size();
    P->cp = upload(h_cp.data(), h_cp.size(), s);
    P->rows = upload(h_rows.data(), h_rows.size(), s);
    P->pos = upload(h_pos.data(), h_pos.size(), s);
    P->vals.reset((size_t)std::max<long long>(1, P->d_total));
    P->BT.reset((size_t)std::max<long long>(1, P->b_total));
    // transpose work: the blocks' 32 x 32 tiles
    std::vector<BlkTrTile> tr;
    for (size_t q = 0; q < descs.size(); ++q)
        for (long long i0 = 0; i0 < descs[q].m0 && descs[q].n0_C > 0; i0 += 32)
            for (long long r0 = 0; r0 < descs[q].n0_B; r0 += 32) 
                tr.push_back(BlkTrTile{descs[q].b_off, descs[q].m0, descs[q].n0_B, (int)i0, (int)r0});
    if (tr.size() > INT_MAX / 2) fail(SDL_ERR_OVERFLOW, "blocks x CSR: too many blocks");
    P->ntr = (int)tr.size();
    P->tr = upload(tr.data(), tr.size(), s);
    P->desc = upload(descs.data(), std::max<size_t>(1, descs.size()), s);
    P->tiles = upload(tiles.data(), tiles.size(), s);
    std::vector<BlkShare> shares[SLAB_Q];
    for (int q = 0; q < SLAB_Q; ++q)
        if (!slabs[q].empty())
        {
            auto &cls = P->slab_cls[q];
            cls.n = (int)slabs[q].size();
            cls.slabs = upload(slabs[q].data(), slabs[q].size(), s);
            // a persistent grid: the CTAs that fit, but no more than give every warp a unit,
            // or one per SM where the units are few
            const int smem = cls.smem + RS_WARPS * RS_WARP_BYTES;
            const auto kern = slab_kernel(q + 1);
            SDL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          RS_SLAB_BYTES + RS_WARPS * RS_WARP_BYTES));
            int per_sm = 1;
            SDL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RS_WARPS * 32, smem));
            cls.grid = (int)std::max<long long>(
                1, std::min<long long>((long long)runtime().num_sms * std::max(1, per_sm),
                                       std::max((cls.units + RS_WARPS - 1) / RS_WARPS,
                                                std::min<long long>(cls.units, runtime().num_sms))));
            shares[q] = share_units(slabs[q], h_cp.data(), cls.grid);
            cls.grid = (int)shares[q].size() - 1;
            cls.shares = upload(shares[q].data(), shares[q].size(), s);
        }
    SDL_CUDA(cudaStreamSynchronize(s));
    return P;
}

void blocks_csr_fill(const BlocksCsrPlan &P, const double *B_vals, const double *S_x, double *C_vals,
                     cudaStream_t s)
{
    if (P.c_total == 0) return;
    // (a source feeding two outputs would be transposed twice: they are one to one here)
    const int gather = P.d_total > 0 ? grid_cap(P.d_total, BC_THREADS, runtime().num_sms * 8) : 0;
    SDL_LAUNCH(k_blocks_csr_inputs, gather + P.ntr, BC_THREADS, 0, s, P.pos.get(), S_x, P.d_total, P.vals.get(),
               gather, P.tr.get(), B_vals, P.BT.get());
    for (int q = 0; q < SLAB_Q; ++q)
    {
        const auto &c = P.slab_cls[q];
        if (c.n)
            SDL_LAUNCH(slab_kernel(q + 1), c.grid, RS_WARPS * 32, c.smem + RS_WARPS * RS_WARP_BYTES, s, c.slabs.get(),
                       c.shares.get(), c.smem, P.cp.get(), P.rows.get(), P.vals.get(), P.BT.get(),
                       C_vals);
    }
    if (P.ntiles)
        SDL_LAUNCH(k_blocks_csr, P.ntiles, BC_THREADS, 0, s, P.tiles.get(), P.desc.get(), P.cp.get(),
                   P.rows.get(), P.vals.get(), P.BT.get(), C_vals);
}

} // namespace sdl

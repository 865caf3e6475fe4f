"""Kernels at the sizes where their tiling can go wrong (edges of tiles, remainders,
smallest and largest of each dispatch class), against the CPU oracle. Every comparison
here is bit for bit: the kernels keep upstream's order of roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.int64)


def T(a, dtype=None):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


# ---------------------------------------------------------------- dense blocks x CSR
# rows: one 16-row group and its edges, a full 64-row slab, several slabs; columns: the
# limits of 64 / 48 / 32-row slabs (256, 341, 512) and one beyond them;
# S columns: one unit of 16 and its edges; entries per column up to every row of S, so
# that a unit's entries (and eight columns' entries) exceed the staged records
@pytest.mark.parametrize("m0,n0,S_n,dens", [
    (1, 1, 1, 1.0), (15, 5, 16, 0.5), (16, 7, 17, 0.9), (17, 64, 15, 0.1), (33, 256, 33, 0.03),
    (64, 256, 100, 0.02), (64, 257, 50, 0.3), (65, 341, 40, 1.0), (48, 342, 31, 0.05), (130, 512, 20, 0.2),
    (31, 513, 18, 0.02), (20, 1024, 19, 0.6), (70, 1025, 34, 0.1)])
def test_blocks_csr_slab_edges_bit_exact(sdl, orc, m0, n0, S_n, dens):
    import torch
    from sparsediff_linalg_b200.device import BlocksCsr
    rng = np.random.default_rng(m0 * 7919 + n0)
    D = rng.random((n0, S_n)) < dens
    D[n0 // 2, S_n // 2] = True
    Sp = np.concatenate([[0], np.cumsum(D.sum(1))]).astype(np.int32)
    Si = np.nonzero(D)[1].astype(np.int32)
    Sx = rng.standard_normal(len(Si))
    Sx[::5] = -0.0
    # the block of these sizes, a smaller one (another slab class) on a subset of the
    # rows, and the first once more
    half = np.sort(rng.permutation(n0)[:max(1, n0 // 2)]).astype(np.int32)
    full = np.arange(n0, dtype=np.int32)
    blocks = [(rng.standard_normal((m0, n0)), full), (rng.standard_normal(((m0 + 1) // 2, len(half))), half),
              (rng.standard_normal((m0, n0)), full)]
    P = BlocksCsr([X.shape[0] for X, _ in blocks], [X.shape[1] for X, _ in blocks], [c for _, c in blocks], Sp, Si,
                  n0, S_n)
    Cv = torch.full((max(1, P.c_values),), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(np.concatenate([X.ravel() for X, _ in blocks])), T(Sx), Cv)
    got = Cv.cpu().numpy()
    want = orc.blocks_csr(blocks, Sp, Si, Sx, S_n)
    at = 0
    for src, mk, nk, perm in P.blocks:
        cols, Cw = want[src]
        assert np.array_equal(perm, cols) and Cw.shape == (mk, nk)
        assert np.array_equal(bits(got[at:at + mk * nk]), bits(Cw.ravel()))
        at += mk * nk
    assert at == P.c_values


# blocks whose largest row count and largest column count are not the same block's (64000 x
# 4000 tiles of 32 x 32 between them, nine blocks: more than a launch can have), beside
# small ones and one without output columns
def test_blocks_csr_uneven_shapes_bit_exact(sdl, orc):
    import torch
    from sparsediff_linalg_b200.device import BlocksCsr
    rng = np.random.default_rng(8)
    S_m, S_n = 2048000, 40
    at = np.sort(rng.permutation(S_m)[:300])
    at[:2] = [0, 7]
    Si = rng.integers(0, S_n, len(at)).astype(np.int32)
    Sp = np.zeros(S_m + 1, np.int32)
    Sp[at + 1] = 1
    Sp = np.cumsum(Sp).astype(np.int32)
    Sx = rng.standard_normal(len(at))
    blocks = [(rng.standard_normal((1, S_m)), np.arange(S_m, dtype=np.int32)),
              (rng.standard_normal((128000, 1)), np.array([7], np.int32)),
              (rng.standard_normal((5, 3)), np.array([1, 2, 3], np.int32))]
    blocks += [(rng.standard_normal((9, 40)), np.sort(rng.permutation(at)[:40]).astype(np.int32)) for _ in range(7)]
    P = BlocksCsr([X.shape[0] for X, _ in blocks], [X.shape[1] for X, _ in blocks], [c for _, c in blocks], Sp, Si,
                  S_m, S_n)
    Cv = torch.full((P.c_values,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(np.concatenate([X.ravel() for X, _ in blocks])), T(Sx), Cv)
    got = Cv.cpu().numpy()
    want = orc.blocks_csr(blocks, Sp, Si, Sx, S_n)
    at = 0
    for src, mk, nk, perm in P.blocks:
        cols, Cw = want[src]
        assert np.array_equal(perm, cols) and Cw.shape == (mk, nk)
        assert np.array_equal(bits(got[at:at + mk * nk]), bits(Cw.ravel()))
        at += mk * nk
    assert at == P.c_values


# so many small blocks of few columns that they are not kept in slabs (more than one per SM),
# one slab fewer, enough columns, and such blocks beside one of more columns and one of more
# rows
@pytest.mark.parametrize("nb,n0C,extra", [(148, 20, False), (149, 20, False), (400, 120, False), (350, 1, True)])
def test_blocks_csr_many_small_blocks_bit_exact(sdl, orc, nb, n0C, extra):
    import torch
    from sparsediff_linalg_b200.device import BlocksCsr
    rng = np.random.default_rng(nb + n0C)
    S_m, S_n = 60, 200
    D = np.zeros((S_m, S_n), bool)
    D[:7, :n0C] = rng.random((7, n0C)) < 0.4
    D[3, :n0C] = True
    D[7:, :] = rng.random((S_m - 7, S_n)) < 0.05
    Sp = np.concatenate([[0], np.cumsum(D.sum(1))]).astype(np.int32)
    Si = np.nonzero(D)[1].astype(np.int32)
    Sx = rng.standard_normal(len(Si))
    small, full = np.arange(7, dtype=np.int32), np.arange(S_m, dtype=np.int32)
    blocks = [(rng.standard_normal((1 + k % 9, 7)), small) for k in range(nb)]
    if extra:
        blocks[200] = (rng.standard_normal((20, S_m)), full)
        blocks.append((rng.standard_normal((150, 7)), small))
    P = BlocksCsr([X.shape[0] for X, _ in blocks], [X.shape[1] for X, _ in blocks], [c for _, c in blocks], Sp, Si,
                  S_m, S_n)
    Cv = torch.full((P.c_values,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(np.concatenate([X.ravel() for X, _ in blocks])), T(Sx), Cv)
    got = Cv.cpu().numpy()
    want = orc.blocks_csr(blocks, Sp, Si, Sx, S_n)
    at = 0
    for src, mk, nk, perm in P.blocks:
        cols, Cw = want[src]
        assert np.array_equal(perm, cols) and Cw.shape == (mk, nk)
        assert np.array_equal(bits(got[at:at + mk * nk]), bits(Cw.ravel()))
        at += mk * nk
    assert at == P.c_values


# columns of very different entry counts, so that CTAs take shares of very different numbers
# of units: nearly all entries at the start, in the middle or at the end, several slabs and
# blocks, and more CTAs than units
@pytest.mark.parametrize("m0,n0,S_n,heavy", [(64, 300, 9000, slice(0, 700)), (70, 200, 9001, slice(4000, 4020)),
                                             (130, 500, 5003, slice(4990, 5003)), (16, 100, 40, slice(0, 1))])
def test_blocks_csr_uneven_columns_bit_exact(sdl, orc, m0, n0, S_n, heavy):
    import torch
    from sparsediff_linalg_b200.device import BlocksCsr
    rng = np.random.default_rng(n0)
    dens = np.full(S_n, 1.5 / n0)
    dens[heavy] = 0.9
    D = rng.random((n0, S_n)) < dens
    Sp = np.concatenate([[0], np.cumsum(D.sum(1))]).astype(np.int32)
    Si = np.nonzero(D)[1].astype(np.int32)
    Sx = rng.standard_normal(len(Si))
    full, half = np.arange(n0, dtype=np.int32), np.arange(0, n0, 2, dtype=np.int32)
    blocks = [(rng.standard_normal((m0, len(c))), c) for c in (full, half, full, half)]
    P = BlocksCsr([X.shape[0] for X, _ in blocks], [X.shape[1] for X, _ in blocks], [c for _, c in blocks], Sp, Si,
                  n0, S_n)
    Cv = torch.full((P.c_values,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(np.concatenate([X.ravel() for X, _ in blocks])), T(Sx), Cv)
    got = Cv.cpu().numpy()
    want = orc.blocks_csr(blocks, Sp, Si, Sx, S_n)
    at = 0
    for src, mk, nk, perm in P.blocks:
        cols, Cw = want[src]
        assert np.array_equal(perm, cols) and Cw.shape == (mk, nk)
        assert np.array_equal(bits(got[at:at + mk * nk]), bits(Cw.ravel()))
        at += mk * nk
    assert at == P.c_values


# ---------------------------------------------------------------- sorting triplets
# sizes around a sort tile (3072 pairs) and a structure tile (2048); matrices whose keys
# take one digit pass up to seven, one cell only (every key equal), rows in order, and a
# few rows far apart (long runs of empty rows)
@pytest.mark.parametrize("n", [1, 2, 33, 2047, 2048, 2049, 3071, 3072, 3073, 6144, 40000])
@pytest.mark.parametrize("m,ncols,kind", [(1, 1, "random"), (9, 7, "random"), (70000, 3, "sorted"),
                                          (5000000, 2000000000, "random"), (3000000, 50, "far")])
def test_coalesce_sort_edges_bit_exact(sdl, orc, n, m, ncols, kind):
    import torch
    from sparsediff_linalg_b200.device import Coalesce
    rng = np.random.default_rng(n + m % 1000)
    rows = rng.integers(0, m, n)
    if kind == "sorted":
        rows = np.sort(rows)
    elif kind == "far":
        rows = rng.choice([5, 6, m // 2, m - 1], n)
    cols = rng.integers(0, ncols, n)
    x = rng.standard_normal(n)
    x[::3] = -0.0
    C = Coalesce(T(rows, torch.int32), T(cols, torch.int32), m, ncols)
    Cx = torch.full((C.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    C.fill(T(x), Cx)
    wp, wi, wx = orc.coalesce(rows.astype(np.int32), cols.astype(np.int32), x, m, ncols)
    assert np.array_equal(C.Cp.cpu().numpy(), wp) and np.array_equal(C.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(Cx.cpu().numpy()), bits(wx))


# runs of empty rows at, below and above the lengths that a lane (8 rows), a warp (65536)
# and a CTA per piece of 65536 write, before the first output, between two and after the last
@pytest.mark.parametrize("gap", [7, 8, 9, 65535, 65536, 65537, 131072, 131073, 200001])
def test_coalesce_row_gaps(sdl, gap):
    import torch
    from sparsediff_linalg_b200.device import Coalesce
    rows = np.repeat([gap, 2 * gap, 2 * gap + 1, 3 * gap + 2], [1, 40, 3, 5])
    m = 4 * gap + 3
    cols = np.arange(len(rows)) % 17
    C = Coalesce(T(rows, torch.int32), T(cols, torch.int32), m, 17)
    want = np.unique(rows.astype(np.int64) * 17 + cols)
    wp = np.concatenate([[0], np.cumsum(np.bincount(want // 17, minlength=m))])
    assert np.array_equal(C.Cp.cpu().numpy(), wp) and np.array_equal(C.Ci.cpu().numpy(), want % 17)


# the largest row count there is: row offsets up to index 2^31 - 1, none of them left out
def test_coalesce_largest_row_count(sdl):
    import torch
    from sparsediff_linalg_b200.device import Coalesce
    m = 2**31 - 1
    rows = [3, 3, 2**30, 2**30 + 9, m - 40, m - 2]
    C = Coalesce(T(np.array(rows), torch.int32), T(np.arange(6), torch.int32), m, 6)
    assert C.nnz == 6 and C.Cp.numel() == m + 1
    at = 0
    for r, before in [(3, 0), (2**30, 2), (2**30 + 9, 3), (m - 40, 4), (m - 2, 5), (m, 6)]:
        run = C.Cp[at:r + 1]
        assert run.numel() == r + 1 - at
        assert int(run.min()) == before and int(run.max()) == before
        at = r + 1
    assert at == m + 1


# more than 2^30 triplets, where the sort's tile words are 64 bits wide: every cell of 32768
# columns once, in an order scattered by a multiplication modulo the prime 2^30 + 3, each
# triplet's value its cell
def test_coalesce_over_2_30_triplets(sdl):
    import torch
    from sparsediff_linalg_b200.device import Coalesce
    n, ncols = 2**30 + 3, 32768
    cell = torch.arange(n, dtype=torch.int64, device="cuda")
    cell.mul_(2654435761).remainder_(n)
    rows, cols = torch.div(cell, ncols, rounding_mode="floor").to(torch.int32), (cell % ncols).to(torch.int32)
    x = cell.to(torch.float64)
    del cell
    m = n // ncols + 1
    C = Coalesce(rows, cols, m, ncols)
    del rows, cols
    assert C.nnz == n
    assert torch.equal(C.Cp.cpu(), torch.arange(m + 1, dtype=torch.int64).mul_(ncols).clamp_(max=n).to(torch.int32))
    out = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    C.fill(x, out)
    torch.cuda.synchronize()
    del x
    step = 1 << 26
    for at in range(0, n, step):
        q = torch.arange(at, min(n, at + step), dtype=torch.int64, device="cuda")
        assert torch.equal(out[at:at + step], q.to(torch.float64))
        assert torch.equal(C.Ci[at:at + step], (q % ncols).to(torch.int32))
    del C, out, q
    torch.cuda.empty_cache()
    sdl.sdl_release_cached_memory()


# ---------------------------------------------------------------- bucketed refill
MIN = 10 << 20  # triplets from which a refill goes through buckets


# the smallest input that takes it; outputs of so many triplets that they fill a bucket
# (22528 values) exactly, exceed it by one or take most of the input; few buckets' worth
# of single-triplet outputs; values and factors from buffers at odd offsets
@pytest.mark.parametrize("n,heavy", [(MIN, 0), (MIN + 1, 22528), (MIN + 3, 22529), (MIN + 2, 3000000)])
def test_coalesce_buckets_edges_bit_exact(sdl, n, heavy):
    import torch
    from oracle import parallel
    from sparsediff_linalg_b200.device import Coalesce
    rng = np.random.default_rng(n + heavy)
    m, ncols = 5001, 4003
    rows, cols = rng.integers(0, m, n), rng.integers(0, ncols, n)
    at = rng.permutation(n)[:heavy]
    rows[at], cols[at] = 1500, 7
    rows, cols = rows.astype(np.int32), cols.astype(np.int32)
    x = rng.standard_normal(n + 1)
    x[::3] = -0.0
    C = Coalesce(T(rows), T(cols), m, ncols)
    xd = T(x)
    for off in (0, 1):
        Cx = torch.full((C.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        C.fill(xd[off:off + n], Cx)
        wp, wi, wx = parallel.coalesce(rows, cols, x[off:off + n].copy(), m, ncols)[:3]
        assert np.array_equal(C.Cp.cpu().numpy(), wp) and np.array_equal(C.Ci.cpu().numpy(), wi)
        assert np.array_equal(bits(Cx.cpu().numpy()), bits(wx))


# inputs of that size whose neighbours in sorted order are neighbours in the input, which are
# gathered in one pass: sorted, 4 x 4 elements along the rows, sorted with an output of
# so many triplets (96) that it keeps buckets or one fewer; and shuffled for half of them
@pytest.mark.parametrize("kind", ["sorted", "elements", "heavy95", "heavy96", "half"])
def test_coalesce_ordered_input_bit_exact(sdl, kind):
    import torch
    from oracle import parallel
    from sparsediff_linalg_b200.device import Coalesce
    rng = np.random.default_rng(len(kind))
    n, m, ncols = MIN + 48, 700000, 700000
    if kind == "elements":
        at = np.sort(rng.integers(0, m - 4, n // 16))[:, None]
        rows, cols = (at + np.repeat(np.arange(4), 4)).ravel(), (at + np.tile(np.arange(4), 4)).ravel()
    else:
        key = np.sort(rng.integers(0, m * ncols, n))
        if kind.startswith("heavy"):
            key[5000000:5000000 + int(kind[5:])] = key[5000000]
        if kind == "half":
            key[:n // 2] = rng.permutation(key[:n // 2])
        rows, cols = key // ncols, key % ncols
    rows, cols = rows.astype(np.int32), cols.astype(np.int32)
    x = rng.standard_normal(len(rows))
    x[::3] = -0.0
    C = Coalesce(T(rows), T(cols), m, ncols)
    Cx = torch.full((C.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    C.fill(T(x), Cx)
    wp, wi, wx = parallel.coalesce(rows, cols, x, m, ncols)[:3]
    assert np.array_equal(C.Cp.cpu().numpy(), wp) and np.array_equal(C.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(Cx.cpu().numpy()), bits(wx))


# the same with a factor per triplet: a scaled sum of two sparse operands with MIN entries
# together, one fewer and one more; each output is (0 + d1 a) + d2 b, one rounding each. Few
# long rows in random order, since rows in order are gathered in one pass (the last case)
@pytest.mark.parametrize("extra,shuffled", [(-1, True), (0, True), (1, True), (1, False)])
def test_scaled_sum_through_buckets_bit_exact(sdl, extra, shuffled):
    from sparsediff_linalg_b200 import matrices as M
    from test_gpu_dense_ops import Lib, csr_of
    from test_gpu_sums import SIGS
    L = M.mlib()
    for name, (res, args) in SIGS.items():
        getattr(L, name).restype, getattr(L, name).argtypes = res, args
    lib = Lib(L)
    rng = np.random.default_rng(900 + extra)
    m, n = 16, 725000
    nnz = [MIN // 2, MIN // 2 + extra]
    cells = [rng.permutation(m * n)[:k] for k in nnz]
    cells = [c[np.argsort(c // n, kind="stable")] if shuffled else np.sort(c) for c in cells]
    vals = [rng.standard_normal(k) for k in nnz]
    vals[0][::5] = -0.0
    d = [rng.uniform(-2, 2, m) for _ in range(2)]
    A, B = (lib.make(("sparse", (np.concatenate([[0], np.cumsum(np.bincount(c // n, minlength=m))]).astype(np.int32),
                                 (c % n).astype(np.int32), v, m, n))) for c, v in zip(cells, vals))
    S = L.new_sparse_matrix_alloc(m, n, sum(nnz))
    L.sum_matrices_alloc(A, B, S)
    L.sum_scaled_matrices_fill_values(A, B, S, d[0].ctypes.data, d[1].ctypes.data)
    p, i, x = csr_of(S)
    lib.free(S, B, A)
    want, has = np.zeros(m * n), np.zeros(m * n, bool)
    for c, v, f in zip(cells, vals, d):
        want[c] = want[c] + f[c // n] * v
        has[c] = True
    at = np.flatnonzero(has)
    assert np.array_equal(p, np.concatenate([[0], np.cumsum(np.bincount(at // n, minlength=m))]))
    assert np.array_equal(i, at % n) and np.array_equal(bits(x), bits(want[at]))


# fewer triplets, but many per output: the smallest input that goes through buckets, one
# triplet or one output to either side of it, and a few outputs that hold them all
@pytest.mark.parametrize("n,nout", [(4 << 20, (4 << 20) // 96), (4 << 20, (4 << 20) // 96 + 1),
                                    ((4 << 20) - 1, 1000), ((4 << 20) + 1, 999), (5000011, 7)])
def test_coalesce_heavy_outputs_bit_exact(sdl, n, nout):
    import torch
    from oracle import parallel
    from sparsediff_linalg_b200.device import Coalesce
    rng = np.random.default_rng(nout)
    m, ncols = 3000, 20
    cell = rng.permutation(m * ncols)[:nout]
    at = cell[rng.permutation(n) % nout]
    rows, cols = (at // ncols).astype(np.int32), (at % ncols).astype(np.int32)
    x = rng.standard_normal(n) * 10.0 ** rng.integers(-6, 7, n)
    x[::3] = -0.0
    C = Coalesce(T(rows), T(cols), m, ncols)
    assert C.nnz == nout
    Cx = torch.full((C.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    C.fill(T(x), Cx)
    wp, wi, wx = parallel.coalesce(rows, cols, x, m, ncols)[:3]
    assert np.array_equal(C.Cp.cpu().numpy(), wp) and np.array_equal(C.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(Cx.cpu().numpy()), bits(wx))


# ---------------------------------------------------------------- transpose
# columns of every sorting class and its edges (64 keys counted in place, 1024 a warp,
# 8192 a CTA), beside empty and short ones; entries around the 2048-entry tiles; far more
# columns than entries, far more rows than entries, and columns repeated inside a row
@pytest.mark.parametrize("rows,cols,lens", [
    (1, 1, [1]), (5, 3, [0, 3, 0]), (700, 40, [64, 65, 63, 0, 1, 2] * 3), (3000, 9, [1024, 1025, 1, 8192, 8193, 64]),
    (2047, 2047, [1] * 2047), (2048, 64, [32] * 64), (100000, 70, [64] * 32 + [1]), (50, 500000, [3] * 1000),
    (4, 3000, [0, 2] * 1500), (20000, 6, [20001, 0, 17000, 64, 5])])
def test_transpose_segment_edges(sdl, orc, rows, cols, lens):
    import torch
    from sparsediff_linalg_b200.device import Transpose
    rng = np.random.default_rng(rows + cols)
    at = np.sort(rng.permutation(cols)[:min(len(lens), cols)])
    col = np.repeat(at, lens[:len(at)])
    nnz = len(col)
    row = rng.integers(0, rows, nnz)
    order = np.lexsort((col, row))
    row, col = row[order], col[order].astype(np.int32)
    p = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=rows))]).astype(np.int32)
    x = rng.standard_normal(nnz)
    t = Transpose(T(p), T(col), rows, cols)
    tx = torch.empty(max(1, nnz), dtype=torch.float64, device="cuda")[:nnz]
    t.fill(T(x), tx)
    wp, wi, wx = orc.transpose(p, col, x, rows, cols)
    assert np.array_equal(t.Tp.cpu().numpy(), wp) and np.array_equal(t.Ti.cpu().numpy(), wi)
    assert np.array_equal(bits(tx.cpu().numpy()), bits(wx))


# ---------------------------------------------------------------- rows beyond the tile budget
# windows of about one term per output, of many (few outputs a window), rows of so many
# that they keep lists, rows whose columns crowd so that windows are halved, and rows with
# one output of more terms than a window holds; one row of exactly one window and its edges
@pytest.mark.parametrize("kind,nL,nA,n,per_row", [
    ("even", 12, 3000, 200000, 5), ("even", 7, 2500, 2500, 20), ("even", 5, 2000, 300, 40),
    ("crowded", 9, 4000, 60000, 6), ("hot", 6, 6000, 90000, 3), ("even", 3, 1025, 2048, 2),
    ("even", 2, 1024, 2047, 3), ("even", 4, 20000, 2049, 1)])
def test_large_row_windows_bit_exact(sdl, orc, kind, nL, nA, n, per_row):
    import torch
    from sparsediff_linalg_b200.device import Batch, Product
    rng = np.random.default_rng(nA + n)
    rows = []
    for _ in range(nA):
        if kind == "crowded":   # most columns in a twentieth of the range
            c = np.where(rng.random(per_row) < 0.8, rng.integers(0, n // 20, per_row), rng.integers(0, n, per_row))
        elif kind == "hot":     # one column in every row
            c = np.concatenate([[7], rng.integers(0, n, per_row)])
        else:
            c = rng.integers(0, n, per_row)
        rows.append(np.unique(c))
    Bp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    Bi = np.concatenate(rows).astype(np.int32)
    lens = rng.integers(nA // 2, nA + 1, nL)
    lens[0], lens[-1] = nA, 3
    Ap = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    Ai = np.concatenate([np.sort(rng.permutation(nA)[:k]) for k in lens]).astype(np.int32)
    P = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    Q = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    batch = Batch([P, Q], stream=s)
    for rnd in range(2):
        Ax, Bx, d = rng.standard_normal(len(Ai)), rng.standard_normal(len(Bi)), rng.uniform(0.1, 10, nA)
        Ax[::3] = -0.0
        wp, wi, wx = orc.spgemm((Ap, Ai, Ax, nL, nA), (Bp, Bi, Bx, nA, n))
        assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
        C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        P.fill(T(Ax), None, T(Bx), C)
        assert np.array_equal(bits(C.cpu().numpy()), bits(wx))
        # the same with a diagonal, single and batched: (a * d) * b, one rounding each
        wd = orc.spgemm((Ap, Ai, Ax * d[Ai], nL, nA), (Bp, Bi, Bx, nA, n))[2]
        dev = [T(Ax), T(d), T(Bx)]
        C.fill_(float("nan"))
        P.fill(dev[0], dev[1], dev[2], C)
        assert np.array_equal(bits(C.cpu().numpy()), bits(wd))
        out = [torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
        for i in range(2):
            batch.bind(i, dev[0], dev[1], dev[2], out[i])
        torch.cuda.synchronize()
        batch.refill(stream=s)
        torch.cuda.synchronize()
        for o in out:
            assert np.array_equal(bits(o.cpu().numpy()), bits(wd))


# outputs around the 64 terms that one thread puts in order, and of many more: windows of more
# terms than one part holds (4096), where one output's terms end a part exactly, miss or
# exceed it by one, or take several parts; in the same product rows of over 32 terms per
# output (lists), tile rows and an empty row
@pytest.mark.parametrize("n,hot", [(60000, (63, 64, 65, 3500)), (700, (66, 2000)), (60000, (4095, 4096, 4097)),
                                   (60000, (8192, 8193, 20000)), (700, (5000, 12289))])
def test_large_row_many_terms_bit_exact(sdl, orc, n, hot):
    import torch
    from sparsediff_linalg_b200.device import Batch, Product
    rng = np.random.default_rng(n + hot[0])
    nA, few = 24000, 3000
    # rows of A: a column of all the rows of one L row each (hot), and two others; the last
    # ones over 50 columns only
    rows = [np.unique(np.concatenate([[7], rng.integers(0, n, 2)])) for _ in range(nA - few)]
    rows += [np.unique(rng.integers(0, 50, 3)) for _ in range(few)]
    cold = [np.unique(rng.integers(8, n, 3)) for _ in range(1500)]  # without the hot column
    rows += cold
    Bp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    Bi = np.concatenate(rows).astype(np.int32)
    ent = [np.concatenate([np.sort(rng.permutation(nA - few)[:k]), np.arange(nA, nA + 1500)]) for k in hot]
    ent += [np.arange(nA - few, nA), np.array([], np.int64), np.array([5, 77, nA + 3])]
    ent.append(np.arange(1, 2400))
    Ap = np.concatenate([[0], np.cumsum([len(e) for e in ent])]).astype(np.int32)
    Ai = np.concatenate(ent).astype(np.int32)
    nL, nR = len(ent), len(rows)
    P, Q = (Product(T(Ap), T(Ai), T(Bp), T(Bi), n) for _ in range(2))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    batch = Batch([P, Q], stream=s)
    for rnd in range(2):
        Ax, Bx = rng.standard_normal(len(Ai)), rng.standard_normal(len(Bi))
        Ax[::3] = -0.0
        wp, wi, wx = orc.spgemm((Ap, Ai, Ax, nL, nR), (Bp, Bi, Bx, nR, n))
        assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
        C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        dev = [T(Ax), T(Bx)]
        P.fill(dev[0], None, dev[1], C)
        assert np.array_equal(bits(C.cpu().numpy()), bits(wx))
        out = [torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
        for i in range(2):
            batch.bind(i, dev[0], None, dev[1], out[i])
        torch.cuda.synchronize()
        batch.refill(stream=s)
        torch.cuda.synchronize()
        for o in out:
            assert np.array_equal(bits(o.cpu().numpy()), bits(wx))


# banded rows, whose middle outputs have most of the terms, so that windows are built again
# narrower (half, a quarter); alone, and beside a row with an output of 6000 terms, whose
# window stays one in parts
@pytest.mark.parametrize("per_l,per_a,step,hot", [(100, 100, 3, False), (200, 100, 9, False), (100, 100, 3, True),
                                                  (60, 60, 1, True)])
def test_large_row_banded_windows_bit_exact(sdl, orc, per_l, per_a, step, hot):
    import torch
    from sparsediff_linalg_b200.device import Product
    rng = np.random.default_rng(per_l + hot)
    nL, nA = 60, 7000
    n = nA * step + per_a * step + 1
    base = np.arange(nA)[:, None] * step + rng.integers(0, 2, (nA, 1))
    rows = base + step * np.arange(per_a)[None]
    if hot:
        rows[:, 0] = 0
    Bp, Bi = (np.arange(nA + 1) * per_a).astype(np.int32), rows.astype(np.int32).ravel()
    ent = [at + np.arange(per_l) for at in np.linspace(10, nA - per_l, nL).astype(int)]
    if hot:
        ent[7] = np.arange(500, 6500)
    Ap = np.concatenate([[0], np.cumsum([len(e) for e in ent])]).astype(np.int32)
    Ai = np.concatenate(ent).astype(np.int32)
    Ax, Bx = rng.standard_normal(len(Ai)), rng.standard_normal(len(Bi))
    Ax[::3] = -0.0
    P = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(Ax), None, T(Bx), C)
    wp, wi, wx = orc.spgemm((Ap, Ai, Ax, nL, nA), (Bp, Bi, Bx, nA, n))
    assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(C.cpu().numpy()), bits(wx))


# ---------------------------------------------------------------- symbolic warp sorts
# rows whose terms fill the sorted sizes (32, 64, 128, 256, 512) exactly, miss or exceed
# them by one, with columns repeated inside a row or not at all; empty rows between
@pytest.mark.parametrize("n", [40, 700, 100000])
def test_row_sort_edges_bit_exact(sdl, orc, n):
    import torch
    from sparsediff_linalg_b200.device import Product
    rng = np.random.default_rng(n)
    want = [1, 2, 31, 32, 33, 0, 63, 64, 65, 127, 128, 129, 0, 0, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025]
    rows = [np.unique(rng.integers(0, n, k)) for k in rng.integers(1, 30, 400)]
    blens = np.array([len(r) for r in rows])
    ent = []
    for w in want:  # distinct rows of B whose lengths add up to w
        left, mine = w, []
        for k in rng.permutation(400):
            if blens[k] <= left:
                mine.append(k)
                left -= blens[k]
        ent.append(np.sort(np.array(mine, np.int64)))
    Ap = np.concatenate([[0], np.cumsum([len(e) for e in ent])]).astype(np.int32)
    Ai = np.concatenate(ent).astype(np.int32)
    Bp = np.concatenate([[0], np.cumsum(blens)]).astype(np.int32)
    Bi = np.concatenate(rows).astype(np.int32)
    Ax, Bx = rng.standard_normal(len(Ai)), rng.standard_normal(len(Bi))
    P = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(Ax), None, T(Bx), C)
    wp, wi, wx = orc.spgemm((Ap, Ai, Ax, len(want), 400), (Bp, Bi, Bx, 400, n))
    assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(C.cpu().numpy()), bits(wx))


# ---------------------------------------------------------------- refill schedule
# tiles at their limit of 256 rows: rows without terms, of one term, of 7 and 8 terms (the
# edge of the cheaper row), alone and mixed, with tile budgets down to the smallest
@pytest.mark.parametrize("lens", [(0,), (1,), (0, 1), (7,), (8,), (7, 8, 0, 1, 300)])
@pytest.mark.parametrize("budget", [0, 128, 500, 1152])
def test_tiles_of_short_rows_bit_exact(sdl, orc, lens, budget):
    import torch
    from sparsediff_linalg_b200.device import Product
    rng = np.random.default_rng(len(lens) * 7 + budget)
    nL, nA, n = 5000, 800, 900
    rows = rng.choice(lens, nL)
    rows[[17, 4000]] = 3
    Ap = np.concatenate([[0], np.cumsum(rows)]).astype(np.int32)
    Ai = np.concatenate([np.sort(rng.permutation(nA)[:k]) for k in rows]).astype(np.int32)
    Bp, Bi = np.arange(nA + 1, dtype=np.int32), rng.integers(0, n, nA).astype(np.int32)
    Ax, Bx = rng.standard_normal(len(Ai)), rng.standard_normal(nA)
    P = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    if budget:
        P.replan(tile_budget=budget)
    C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(Ax), None, T(Bx), C)
    wp, wi, wx = orc.spgemm((Ap, Ai, Ax, nL, nA), (Bp, Bi, Bx, nA, n))
    assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
    assert np.array_equal(bits(C.cpu().numpy()), bits(wx))


# list sections of more words (about 70M) than the schedule's first scratch (64Mi) holds: they
# are built again in a larger one
def test_schedule_of_many_list_words_bit_exact(sdl, orc):
    import torch
    from sparsediff_linalg_b200.device import Product
    rng = np.random.default_rng(11)
    nL, per_l, nA, per_a, n = 66000, 25, 1000, 40, 60
    Bi = np.concatenate([np.sort(rng.permutation(n)[:per_a]) for _ in range(nA)]).astype(np.int32)
    Bp = (np.arange(nA + 1) * per_a).astype(np.int32)
    Ai = np.sort((rng.integers(0, nA, (nL, 1)) + 37 * np.arange(per_l)) % nA, axis=1).astype(np.int32).ravel()
    Ap = (np.arange(nL + 1) * per_l).astype(np.int32)
    Ax, Bx = rng.standard_normal(len(Ai)), rng.standard_normal(len(Bi))
    P = Product(T(Ap), T(Ai), T(Bp), T(Bi), n)
    wp, wi, wx = orc.spgemm((Ap, Ai, Ax, nL, nA), (Bp, Bi, Bx, nA, n))
    assert len(Ai) * per_a + len(wi) > 64 << 20  # terms in lists, and their headers
    assert np.array_equal(P.Cp.cpu().numpy(), wp) and np.array_equal(P.Ci.cpu().numpy(), wi)
    C = torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    P.fill(T(Ax), None, T(Bx), C)
    assert np.array_equal(bits(C.cpu().numpy()), bits(wx))


# operands changed between the structure of C and its refill plan (columns that some rows of
# C lack): the plan is refused, the error does not stick, and restored operands get their plan
def test_schedule_of_changed_operands_is_refused(sdl):
    import torch
    from sparsediff_linalg_b200.device import Product
    from sparsediff_linalg_b200.learned import LearnedFilledProduct, Mlp
    rng = np.random.default_rng(5)
    n, nA, nL = 5000, 900, 700
    rows = [np.unique(rng.integers(0, n, k)) for k in rng.integers(1, 9, nA)]
    Bp = T(np.concatenate([[0], np.cumsum([len(r) for r in rows])]), torch.int32)
    good = T(np.concatenate(rows), torch.int32)
    Bi = good.clone()
    ent = [np.sort(rng.permutation(nA)[:k]) for k in rng.integers(1, 60, nL)]
    Ap = T(np.concatenate([[0], np.cumsum([len(e) for e in ent])]), torch.int32)
    Ai = T(np.concatenate(ent), torch.int32)
    Ax = torch.randn(Ai.numel(), dtype=torch.float64, device="cuda")
    Bx = torch.randn(Bi.numel(), dtype=torch.float64, device="cuda")
    Q = LearnedFilledProduct(Ap, Ai, Bp, Bi, n, Mlp(seed=1), Ax, None, Bx)
    Bi.copy_((good + 1) % n)
    torch.cuda.synchronize()
    with pytest.raises(Exception):
        Q.complete_plan()
    assert not Q.plan_ready()
    Bi.copy_(good)
    torch.cuda.synchronize()
    Q.complete_plan()
    P = Product(Ap, Ai, Bp, Bi, n)
    cp, cq = (torch.full((P.nnz,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    P.fill(Ax, None, Bx, cp)
    Q.fill(Ax, None, Bx, cq)
    torch.cuda.synchronize()
    assert torch.equal(P.Cp, Q.Cp) and torch.equal(cp.view(torch.int64), cq.view(torch.int64))

"""Kernels at the sizes where they can go wrong (GPU, through the public entry
points): row lengths around the widths a lane group works in, misaligned row
starts, unsorted and repeated columns, empty rows, caller buffers off a 16-byte
boundary.

Tolerances: every operand here is non-negative, so an FP32 sum of k products
lies within (k + 2) * 2^-24 of its FP64 value, relative, in any order (values
stored in 16 bits are rounded to their type before the FP64 sum).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENS = [0, 1, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 127, 128, 129, 255, 256, 257, 511, 513, 1025, 4099]


def edge_csr(seed, cols, sorted_rows):
    """Rows of every length in LENS at every start offset modulo 8, in random
    order; unsorted rows may repeat a column."""
    rng = np.random.default_rng(seed)
    lens = np.array(LENS * 8)
    rng.shuffle(lens)
    lens = np.concatenate([[1], lens, [0, 0, 5]])
    rows = [np.sort(rng.choice(cols, n, replace=False)) if sorted_rows else rng.integers(0, cols, n) for n in lens]
    rp = np.zeros(len(lens) + 1, np.uint64)
    rp[1:] = np.cumsum(lens)
    col = np.concatenate(rows).astype(np.uint32)
    val = rng.uniform(0.05, 1.0, len(col)).astype(np.float32)
    return rng, rp, col, val


def stored(torch, val, vt):
    """The values as the handle stores them, in FP64."""
    return torch.from_numpy(val).to([torch.float32, torch.float16, torch.bfloat16][vt]).double().numpy()


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("sorted_rows", [True, False])
@pytest.mark.parametrize("off", [0, 1])
def test_scatter_back_projection(pkg, cuda, vt, sorted_rows, off):
    cols = 4999
    rng, rp, col, val = edge_csr(21, cols, sorted_rows)
    ratio = rng.uniform(0.0, 2.0, len(rp) - 1).astype(np.float32)
    ratio[rng.random(len(ratio)) < 0.1] = 0.0
    rid = np.repeat(np.arange(len(rp) - 1), np.diff(rp.astype(np.int64)))
    v = stored(cuda, val, vt)
    want = np.bincount(col, weights=v * ratio[rid].astype(np.float64), minlength=cols)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt, build_transpose=False)
    r = cuda.from_numpy(ratio).cuda()
    out = cuda.full((cols + off,), -1.0, device="cuda")[off:]
    m.back_project(r.data_ptr(), out.data_ptr(), bp_mode=pkg.BP_SCATTER)
    cuda.cuda.synchronize()
    got = out.cpu().numpy().astype(np.float64)
    k = np.bincount(col, minlength=cols)
    assert np.all(np.abs(got - want) <= (k + 2) * 2.0**-24 * want)
    m.close()


@pytest.mark.parametrize("lanes", [8, 16, 32])
@pytest.mark.parametrize("unroll", [1, 2])
def test_fused_pass_repeated_columns(pkg, O, lanes, unroll):
    """The rescan form on rows that repeat columns, against the FP64 oracle (the
    image tolerance of the fused pass, 1e-5 relative L2)."""
    cols = 4999
    rng, rp, col, val = edge_csr(22, cols, False)
    A = (rp, col, val)
    g = rng.poisson(O.project_f64(*A, rng.uniform(0.0, 1.0, cols)) * 20.0).astype(np.int32)
    norm = O.colsum(*A, cols, f64=True)
    f0 = np.full(cols, O.initial_value(g, norm), np.float32)
    m = pkg.Matrix.from_csr(*A, cols, norm=norm, build_transpose=False)
    got = m.run(g, 8, f0=f0, bp_mode=pkg.BP_FUSED, kernel=pkg.KERNEL_DIRECT, lanes=lanes, unroll=unroll)
    assert O.rel_l2(got, O.mlem_f64(A, g, norm, f0, 8)) < 1e-5
    m.close()


def d16_rows(seed, cols, long_rows):
    """Ascending rows whose columns jump by more than 65,535 (once, twice, in a
    row's first entries, back to back), repeat, and end at and around the steps of
    8 entries per lane; mean length on the wanted side of 128."""
    rng = np.random.default_rng(seed)
    lens = [n for n in LENS if n <= (4099 if long_rows else 129)] * (6 if long_rows else 40)
    rows = []
    for i, n in enumerate(lens):
        c = np.sort(rng.integers(0, cols if i % 3 else 3000, n))
        if n > 12 and i % 4 == 0:
            c[n // 2:] = np.minimum(c[n // 2:] + 200_000, cols - 1)
            c = np.sort(c)
        rows.append(c)
    rp = np.zeros(len(rows) + 1, np.uint64)
    rp[1:] = np.cumsum([len(c) for c in rows])
    col = np.concatenate(rows).astype(np.uint32)
    val = rng.uniform(0.05, 1.0, len(col)).astype(np.float32)
    val[::97] = -0.0
    return rng, rp, col, val


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("long_rows", [True, False])
@pytest.mark.parametrize("unroll", [1, 2])
def test_delta_coded_projection(pkg, cuda, vt, long_rows, unroll):
    """Delta-coded rows of A and of its transpose against FP64, and against the
    csr-vector kernel where x holds infinities and NaN: an element outside a row
    must not reach its sum through the dummies or the padding."""
    cols = 600_000
    rng, rp, col, val = d16_rows(31, cols, long_rows)
    rows = len(rp) - 1
    rid = np.repeat(np.arange(rows), np.diff(rp.astype(np.int64)))
    v = stored(cuda, val, vt)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt, compress=True)
    assert m.d16["lanes"] == (8 if long_rows else 4)
    x = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    r = rng.uniform(0.5, 1.5, rows).astype(np.float32)
    g = cuda.zeros(rows, dtype=cuda.int32, device="cuda")

    def project(x, r, **kw):
        dx, dr = cuda.from_numpy(x).cuda(), cuda.from_numpy(r).cuda()
        ratio, fp, bp = cuda.empty(rows, device="cuda"), cuda.empty(rows, device="cuda"), cuda.empty(cols, device="cuda")
        m.forward_project(dx.data_ptr(), g.data_ptr(), ratio.data_ptr(), fp.data_ptr(), **kw)
        m.back_project(dr.data_ptr(), bp.data_ptr(), **kw)
        cuda.cuda.synchronize()
        return fp.cpu().numpy(), bp.cpu().numpy()

    fp, bp = project(x, r, kernel=pkg.KERNEL_D16, unroll=unroll)
    want = np.bincount(rid, weights=v * x[col].astype(np.float64), minlength=rows)
    assert np.all(np.abs(fp - want) <= (np.bincount(rid, minlength=rows) + 2) * 2.0**-24 * want)
    want = np.bincount(col, weights=v * r[rid].astype(np.float64), minlength=cols)
    assert np.all(np.abs(bp - want) <= (np.bincount(col, minlength=cols) + 2) * 2.0**-24 * want)
    x[rng.choice(cols, 4000, replace=False)] = np.inf
    x[rng.choice(cols, 4000, replace=False)] = np.nan
    r[rng.choice(rows, 8, replace=False)] = -np.inf
    for a, b in zip(project(x, r, kernel=pkg.KERNEL_D16, unroll=unroll), project(x, r, kernel=pkg.KERNEL_DIRECT)):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        np.testing.assert_array_equal(a[np.isinf(b)], b[np.isinf(b)])
        np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b))
    m.close()


def test_tuned_copy_stays_private(pkg, cuda):
    """A handle that the tuner gave a delta-coded copy of its own still reports
    none and still refuses the kernel that needs compress_indices; its image
    stays within the FP32 tolerance of the csr-vector kernel's."""
    rng = np.random.default_rng(5)
    rows, cols, n = 40_000, 50_000, 450  # 18 M nonzeros: 144 MB, more than L2
    start = rng.integers(0, cols - 2 * n, rows)
    col = (start[:, None] + np.arange(0, 2 * n, 2)[None, :]).astype(np.uint32).ravel()
    rp = (np.arange(rows + 1) * n).astype(np.uint64)
    val = rng.uniform(0.05, 1.0, col.size).astype(np.float32)
    g = rng.poisson(50.0, rows).astype(np.int32)
    m = pkg.Matrix.from_csr(rp, col, val, cols)
    direct = m.run(g, 5, kernel=pkg.KERNEL_DIRECT)
    auto = m.run(g, 5)
    assert np.linalg.norm(auto - direct) <= 1e-5 * np.linalg.norm(direct)
    np.testing.assert_array_equal(m.run(g, 5), auto)
    with pytest.raises(pkg.MlemError, match="compress_indices"):
        m.run(g, 1, kernel=pkg.KERNEL_D16)
    info = pkg.MatrixInfo()
    pkg.load_library().mlem_matrix_get_info(m.handle, C.byref(info))
    assert (info.d16_slots, info.d16_slots_t, info.d16_lanes, info.d16_lanes_t) == (0, 0, 0, 0)
    m.close()


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("secsize", [1, 5, 64, 512])
@pytest.mark.parametrize("long_rows", [True, False])
def test_merge_tiles_with_empty_runs(pkg, cuda, vt, secsize, long_rows):
    """Merge-path projections of rows on both sides of the 8 / 16 lane choice, with
    runs of empty rows longer than a tile at the start, inside and at the end, and
    rows longer than several tiles next to them."""
    cols = 4999
    rng, rp, col, val = edge_csr(41, cols, False)
    lens = np.diff(rp.astype(np.int64))
    if not long_rows:  # many short rows bring the mean below 96
        short = rng.integers(0, 40, 4000)
        lens, col = np.concatenate([lens, short]), np.concatenate([col, rng.integers(0, cols, short.sum())])
    big = np.array([30_000, 1, 200_000 if secsize < 512 else 70_000])
    lens = np.concatenate([np.zeros(700, int), lens, np.zeros(9000, int), big, np.zeros(300, int)])
    col = np.concatenate([col, rng.integers(0, cols, big.sum())]).astype(np.uint32)
    if long_rows:
        lens = lens[lens > 0]  # no empty rows at all: a mean above 96
        lens = np.concatenate([[0], lens, [0, 0]])
    rows = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    val = rng.uniform(0.05, 1.0, len(col)).astype(np.float32)
    assert (len(col) // rows >= 96) == long_rows
    rid = np.repeat(np.arange(rows), lens)
    v = stored(cuda, val, vt)
    x = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    r = rng.uniform(0.5, 1.5, rows).astype(np.float32)
    g = rng.integers(0, 50, rows).astype(np.int32)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt)
    dx, dr, dg = (cuda.from_numpy(a).cuda() for a in (x, r, g))
    ratio, fp, bp = (cuda.full((n,), -1.0, device="cuda") for n in (rows, rows, cols))
    kw = dict(spmv=pkg.SPMV_MERGE, secsize_fp=secsize, secsize_bp=secsize)
    m.forward_project(dx.data_ptr(), dg.data_ptr(), ratio.data_ptr(), fp.data_ptr(), **kw)
    m.back_project(dr.data_ptr(), bp.data_ptr(), **kw)
    cuda.cuda.synchronize()
    fp, bp, ratio = fp.cpu().numpy(), bp.cpu().numpy(), ratio.cpu().numpy()
    want = np.bincount(rid, weights=v * x[col].astype(np.float64), minlength=rows)
    assert np.all(np.abs(fp - want) <= (lens + 2) * 2.0**-24 * want)
    np.testing.assert_array_equal(ratio, np.where(fp != 0, g.astype(np.float32) / np.where(fp != 0, fp, 1), 0))
    want = np.bincount(col, weights=v * r[rid].astype(np.float64), minlength=cols)
    assert np.all(np.abs(bp - want) <= (np.bincount(col, minlength=cols) + 2) * 2.0**-24 * want)
    m.close()


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("mean", [20, 150])
@pytest.mark.parametrize("longest", [1, 640, 641, 1300])
def test_merge_tiles_of_whole_rows(pkg, cuda, vt, mean, longest):
    """Longest rows around the items of a tile (128 threads x 5 items, or 8 mean rows),
    where the merge-path tiles change from whole rows to shared ones, beside tiles
    that hold no row end: single products and an image of 40 iterations."""
    rng, cols = np.random.default_rng(longest + mean), 3001
    lens = rng.integers(0, 2 * mean, 3000)
    lens[rng.random(3000) < 0.2] = 0
    lens = np.minimum(lens, longest)
    lens[[0, 77, 78, 79, 2999]] = longest
    col = rng.integers(0, cols, lens.sum()).astype(np.uint32)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    val = rng.uniform(0.05, 1.0, len(col)).astype(np.float32)
    rid, v = np.repeat(np.arange(3000), lens), stored(cuda, val, vt)
    x = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    g = rng.integers(0, 50, 3000).astype(np.int32)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt)
    dx, dg = cuda.from_numpy(x).cuda(), cuda.from_numpy(g).cuda()
    ratio, fp, bp = (cuda.full((n,), -1.0, device="cuda") for n in (3000, 3000, cols))
    m.forward_project(dx.data_ptr(), dg.data_ptr(), ratio.data_ptr(), fp.data_ptr(), spmv=pkg.SPMV_MERGE)
    m.back_project(ratio.data_ptr(), bp.data_ptr(), spmv=pkg.SPMV_MERGE)
    fp, bp, ratio = fp.cpu().numpy(), bp.cpu().numpy(), ratio.cpu().numpy()
    want = np.bincount(rid, weights=v * x[col].astype(np.float64), minlength=3000)
    assert np.all(np.abs(fp - want) <= (lens + 2) * 2.0**-24 * want)
    want = np.bincount(col, weights=v * ratio[rid].astype(np.float64), minlength=cols)
    assert np.all(np.abs(bp - want) <= (np.bincount(col, minlength=cols) + 2) * 2.0**-24 * want)
    # an iteration's relative rounding error is at most the two sums' (lens + column
    # entries) plus 5 operations; iterations with positive weights do not amplify it
    # beyond their sum, here with a factor of 4 to spare for the ratio's share
    f = {k: m.run(g, 40, x, spmv=k) for k in (pkg.SPMV_MERGE, pkg.SPMV_CSR_VECTOR)}
    a, b = (np.asarray(q, np.float64) for q in f.values())
    per = int(lens.max()) + int(np.bincount(col, minlength=cols).max()) + 5
    assert np.linalg.norm(a - b) <= 4 * 40 * per * 2.0**-24 * np.linalg.norm(b)
    m.close()


@pytest.mark.parametrize("vt", [0, 1, 2])
@pytest.mark.parametrize("long_rows", [True, False])
@pytest.mark.parametrize("unroll", [1, 2])
def test_merge_tiles_delta_coded(pkg, cuda, vt, long_rows, unroll):
    """Merge-path tiles over delta-coded rows, among runs of empty rows longer than a
    block, against FP64, and against the CSR tiles where x holds infinities and NaN."""
    cols = 600_000
    rng, rp, col, val = d16_rows(37, cols, long_rows)
    gap = 150 if long_rows else 1000
    at = (len(rp) - 1) // 2
    rp = np.concatenate([np.zeros(gap // 2, np.uint64), rp[:at + 1], np.repeat(rp[at], gap), rp[at + 1:],
                         np.repeat(rp[-1], gap // 5)])
    rows = len(rp) - 1
    lens = np.diff(rp.astype(np.int64))
    rid, v = np.repeat(np.arange(rows), lens), stored(cuda, val, vt)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt, compress=True)
    x = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    r = rng.uniform(0.5, 1.5, rows).astype(np.float32)
    g = cuda.from_numpy(rng.integers(0, 50, rows).astype(np.int32)).cuda()

    def project(x, r, **kw):
        dx, dr = cuda.from_numpy(x).cuda(), cuda.from_numpy(r).cuda()
        ratio, fp, bp = (cuda.full((n,), -1.0, device="cuda") for n in (rows, rows, cols))
        kw = dict(kw, spmv=pkg.SPMV_MERGE, secsize_fp=64, secsize_bp=64)
        m.forward_project(dx.data_ptr(), g.data_ptr(), ratio.data_ptr(), fp.data_ptr(), **kw)
        m.back_project(dr.data_ptr(), bp.data_ptr(), **kw)
        return fp.cpu().numpy(), bp.cpu().numpy(), ratio.cpu().numpy()

    fp, bp, ratio = project(x, r, kernel=pkg.KERNEL_D16, unroll=unroll)
    want = np.bincount(rid, weights=v * x[col].astype(np.float64), minlength=rows)
    assert np.all(np.abs(fp - want) <= (lens + 2) * 2.0**-24 * want)
    gs = g.cpu().numpy().astype(np.float32)
    np.testing.assert_array_equal(ratio, np.where(fp != 0, gs / np.where(fp != 0, fp, 1), 0))
    want = np.bincount(col, weights=v * r[rid].astype(np.float64), minlength=cols)
    assert np.all(np.abs(bp - want) <= (np.bincount(col, minlength=cols) + 2) * 2.0**-24 * want)
    x[rng.choice(cols, 4000, replace=False)] = np.inf
    x[rng.choice(cols, 4000, replace=False)] = np.nan
    r[rng.choice(rows, 8, replace=False)] = -np.inf
    for a, b in zip(project(x, r, kernel=pkg.KERNEL_D16, unroll=unroll), project(x, r, kernel=pkg.KERNEL_DIRECT)):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        np.testing.assert_array_equal(a[np.isinf(b)], b[np.isinf(b)])
        np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b))
    m.close()


@pytest.mark.parametrize("vt", [0, 1])
def test_batch_slots_and_row_lengths(pkg, O, cuda, vt):
    """Batches that leave slots of every width unused, on rows around the 32 entries
    of a chunk: the same bits in every tile and count, alone and together, and the
    FP64 oracle's image (the batched tolerance, 1e-5 relative L2)."""
    cols = 4999
    rng, rp, col, val = edge_csr(51, cols, False)
    v = stored(cuda, val, vt).astype(np.float32)
    x = rng.uniform(0.0, 1.0, (5, cols))
    G = np.stack([rng.poisson(O.project_f64(rp, col, v, xi) * 20.0) for xi in x]).astype(np.int32)
    m = pkg.Matrix.from_csr(rp, col, val, cols, value_type=vt)
    norm = O.colsum(rp, col, v, cols, f64=True)
    its = [3, 5, 2, 4, 5]
    alone = [m.batch_run(G[k:k + 1], its[k:k + 1])[0] for k in range(5)]
    for k in range(5):
        f0 = np.full(cols, m.initial_value(G[k]), np.float32)
        assert O.rel_l2(alone[k], O.mlem_f64((rp, col, v), G[k], norm, f0, its[k])) < 1e-5
    for count in (1, 4, 5, 9, 13, 20, 24, 29, 33):
        which = np.arange(count) % 5
        for tile in (0, 8, 16, 32):
            out = m.batch_run(G[which], [its[k] for k in which], tile=tile)
            for b, k in enumerate(which):
                np.testing.assert_array_equal(out[b], alone[k], err_msg=f"count {count} tile {tile} instance {b}")
    m.close()


@pytest.mark.parametrize("cols", [1, 31, 33, 256, 257, 8192, 8193, 65_537, 2_000_000])
@pytest.mark.parametrize("nnz", [1, 4095, 4097, 70_001])
def test_transpose_pass_shapes(pkg, cols, nnz):
    """The stable counting sort on both sides of the number of its passes, of a full
    digit and of a tile of 4,096 elements: bit-exact."""
    rng = np.random.default_rng(61)
    rows = 37
    lens = rng.multinomial(nnz, np.ones(rows) / rows)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    col = rng.integers(0, cols, nnz).astype(np.uint32)
    val = rng.standard_normal(nnz).astype(np.float32)
    cp, ri, v = pkg.transpose(rp, col, val, cols)
    order = np.argsort(col, kind="stable")
    np.testing.assert_array_equal(cp, np.concatenate([[0], np.cumsum(np.bincount(col, minlength=cols))]).astype(np.uint64))
    np.testing.assert_array_equal(ri, np.repeat(np.arange(rows, dtype=np.uint32), lens)[order])
    np.testing.assert_array_equal(v.view(np.uint32), val[order].view(np.uint32))


@pytest.mark.parametrize("cols", [1, 2, 200, 300, 65_536, 16_777_217])
def test_transpose_pass_counts(pkg, cols):
    """One to four passes and last digits of 0 to 8 bits, a third of the entries in one
    column, which stay in row order: bit-exact."""
    rng = np.random.default_rng(cols)
    lens = rng.integers(0, 9, 3001)
    lens[1000] = 4096
    col = rng.integers(0, cols, lens.sum()).astype(np.uint32)
    col[::3] = cols - 1
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    val = rng.standard_normal(len(col)).astype(np.float32)
    cp, ri, v = pkg.transpose(rp, col, val, cols)
    order = np.argsort(col, kind="stable")
    np.testing.assert_array_equal(cp, np.concatenate([[0], np.cumsum(np.bincount(col, minlength=cols))]).astype(np.uint64))
    np.testing.assert_array_equal(ri, np.repeat(np.arange(3001, dtype=np.uint32), lens)[order])
    np.testing.assert_array_equal(v.view(np.uint32), val[order].view(np.uint32))

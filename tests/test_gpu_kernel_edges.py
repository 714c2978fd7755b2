"""Kernels at the sizes where they can go wrong (GPU, through the public entry
points): row lengths around the widths a lane group works in, misaligned row
starts, unsorted and repeated columns, empty rows, caller buffers off a 16-byte
boundary.

Tolerances: every operand here is non-negative, so an FP32 sum of k products
lies within (k + 2) * 2^-24 of its FP64 value, relative, in any order (values
stored in 16 bits are rounded to their type before the FP64 sum).
"""
from __future__ import annotations

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

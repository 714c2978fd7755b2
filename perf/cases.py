"""The work that users of this framework have it do, as timed cases.

A case is a system matrix (a ring scanner, a voxel grid and how the matrix is
stored), one public entry point and its switches:

* ``run``    ``Matrix.run_device``: MLEM iterations on device buffers
* ``host``   ``Matrix.run``: the same on host buffers
* ``ops``    ``Matrix.forward_project`` and ``Matrix.back_project``
* ``batch``  ``Matrix.batch_run``: many sinograms, uneven iteration counts
* ``mlem``   ``mlem()``: the reference's call, host CSR in, image out

The scanners are the package's presets and others of the same kind.  A
program keeps its matrix handle and reconstructs many sinograms with it, so
handles stay in a small cache here; sinograms and images are made from the
seed.  A sinogram holds Poisson counts of the exact chord lengths of seeded
ellipsoids, so it depends on no projection code.
"""
import importlib
import math
from collections import OrderedDict

import numpy as np
import torch

pkg = importlib.import_module("bachelorarbeit-mlem_gb300")

GEO = ("det_per_ring", "n_rings", "radius", "ring_pitch", "nx", "ny", "nz", "vx", "vy", "vz", "sub_t", "sub_z",
       "width_t", "width_z", "row_stride", "row_phase")
STORED = ("value", "layout", "compress", "symmetry", "transpose")
VALUES = {"f32": pkg.VAL_F32, "f16": pkg.VAL_F16, "bf16": pkg.VAL_BF16}
SPMV = {"vector": pkg.SPMV_CSR_VECTOR, "merge": pkg.SPMV_MERGE}
BP = {"trans": pkg.BP_TRANS, "scatter": pkg.BP_SCATTER, "fused": pkg.BP_FUSED}


def _case(name, scanner, kind, iterations, value="f32", layout=pkg.LAYOUT_NATURAL, compress=False, symmetry=False,
          transpose=True, spmv="vector", bp="trans", count=1, counts=38.0, **geo):
    c = {"name": name, "kind": kind, "iterations": iterations, "value": value, "layout": layout,
         "compress": compress, "symmetry": symmetry, "transpose": transpose, "spmv": spmv, "bp": bp, "count": count,
         "counts": counts}
    c.update(dict(pkg.PRESETS[scanner], row_stride=1, row_phase=0))
    c.update(geo)
    return c


def listed():
    loc = pkg.LAYOUT_LOCALITY
    return [
        # single projections of a 2-D ring: a program with its own iteration (OSEM, MAP) around the two operators
        _case("ops_ring2d", "ring2d", "ops", 1),
        # a 2-D slice reconstruction: a matrix that fits in L2, two short kernels per iteration
        _case("run_ring2d", "ring2d", "run", 50),
        # the reference's call with host arrays, matrix uploaded and transposed inside: every seventh LOR of the
        # 3-D mid scanner, so ragged row counts
        _case("mlem_mid_7th", "cyl3d_mid", "mlem", 20, row_stride=7, row_phase=3),
        # a resident matrix in the caller's order, sinogram and image on the host: the default handle
        _case("host_mid", "cyl3d_mid", "host", 20),
        # the same scanner in the locality layout, device buffers
        _case("run_mid", "cyl3d_mid", "run", 10, layout=loc),
        # argv[8] = 0: merge-path projections
        _case("merge_mid", "cyl3d_mid", "run", 10, spmv="merge"),
        # argv[7] = 1: no transpose held, back projection by scatter; a short scan with few counts
        _case("scatter_mid", "cyl3d_mid", "run", 10, layout=loc, transpose=False, bp="scatter", counts=5.0),
        # a queue of sinograms of one scanner with uneven iteration counts
        _case("batch_mid", "cyl3d_mid", "batch", 20, layout=loc, count=24),
        # an odd scanner with short rings and a flat odd grid, half-precision storage, single projections
        _case("ops_odd_bf16", "cyl3d_mid", "ops", 1, value="bf16", layout=loc, det_per_ring=93, n_rings=11,
              radius=47.0, nx=121, ny=133, nz=37),
        # the 12 GB-class matrix, plain FP32
        _case("run_12gb", "cyl3d_12gb", "run", 10, layout=loc),
        # the same in one pass over A per iteration
        _case("fused_12gb", "cyl3d_12gb", "run", 10, layout=loc, bp="fused"),
        # the same with FP16 values and 16-bit indices
        _case("fp16_12gb", "cyl3d_12gb", "run", 10, value="f16", layout=loc, compress=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    flat = rng.random() < 0.3
    kind = rng.choice(["run", "run", "run", "host", "ops", "ops", "batch", "mlem"])
    n = _log_int(rng, 33, 160)
    ny = n if rng.random() < 0.5 else max(17, n - rng.randrange(1, 17))
    nz = 1 if flat else _log_int(rng, 3, 48)
    dpr, rings = _log_int(rng, 49, 160), 1 if flat else rng.randrange(2, 9)
    vx = round(rng.uniform(0.4, 1.0), 2)
    # rows of the scanner, thinned to what the largest listed case holds at most (one-shot calls to less)
    lors = dpr * rings * (dpr * rings - 1) // 2
    stride = max(1, -(-lors // (150_000 if kind == "mlem" else 600_000)))
    if rng.random() < 0.3:
        stride += rng.randrange(1, 6)
    value = rng.choice(["f32", "f32", "f32", "f16", "bf16"]) if kind != "mlem" else "f32"
    bp = rng.choice(["trans", "trans", "trans", "scatter", "fused"]) if kind in ("run", "host") else "trans"
    if kind == "mlem" and rng.random() < 0.4:
        bp = "scatter"
    sym = kind in ("run", "host") and bp == "trans" and rng.random() < 0.15
    if sym:  # the 16 symmetries: detectors in quarters, a square grid, every LOR
        n = ny = min(n, ny)
        dpr, rings, stride = dpr // 4 * 4, min(rings, 1000 // dpr), 1
    spmv = "merge" if not sym and kind in ("run", "ops", "mlem") and bp != "fused" and rng.random() < 0.25 else "vector"
    return {"kind": kind, "iterations": 1 if kind == "ops" else _log_int(rng, 3, 40), "value": value,
            "layout": pkg.LAYOUT_NATURAL if kind == "mlem" or sym else rng.choice([0, 1]),
            "compress": value != "f32" and kind != "batch" and rng.random() < 0.5, "symmetry": sym,
            "transpose": bp == "trans", "spmv": spmv, "bp": bp,
            "count": _log_int(rng, 3, 40) if kind == "batch" else 1, "counts": round(math.exp(rng.uniform(0, 4)), 2),
            "det_per_ring": dpr, "n_rings": rings, "radius": round(0.72 * n * vx, 1) + 2.0,
            "ring_pitch": round(1.1 * max(nz, 2) * vx / max(rings, 1), 2), "nx": n, "ny": ny, "nz": nz,
            "vx": vx, "vy": vx, "vz": vx, "sub_t": rng.randrange(1, 4), "sub_z": 1 if flat else rng.randrange(1, 3),
            "width_t": round(1.5 * vx, 2), "width_z": 0.0 if flat else round(1.5 * vx, 2),
            "row_stride": stride, "row_phase": rng.randrange(stride)}


# ------------------------------------------------------------------- matrices
_handles = OrderedDict()  # the matrices a program keeps: spec -> Matrix, or host CSR arrays and column sums
_MOST = 6


def _geometry(case):
    return pkg.geometry(**{k: case[k] for k in GEO})


def _generate(case):
    return pkg.Matrix.generate(_geometry(case), value_type=VALUES[case["value"]], build_transpose=case["transpose"],
                               compress=case["compress"], layout=case["layout"], symmetry=case["symmetry"])


def _kept(case):
    key = tuple(case[k] for k in GEO + STORED) + (case["kind"] == "mlem",)
    if key not in _handles:
        while len(_handles) >= _MOST:
            _handles.popitem(last=False)
        m = _generate(case)
        if case["kind"] == "mlem":
            rp, col, val = m.csr()
            m.close()
            norm = np.bincount(col, weights=val, minlength=case["nx"] * case["ny"] * case["nz"]).astype(np.float32)
            m = (rp, col, val, norm)
        _handles[key] = m
    _handles.move_to_end(key)
    return _handles[key]


def _sinogram(case, rng):
    """int32 counts of the kept LORs: Poisson of the chord lengths through seeded ellipsoids (float64, on the GPU)."""
    dpr, rings = case["det_per_ring"], case["n_rings"]
    d = torch.arange(dpr * rings, device="cuda")
    th = (d % dpr).double() * (2 * math.pi / dpr)
    z = ((d // dpr).double() - 0.5 * (rings - 1)) * case["ring_pitch"]
    p = torch.stack([case["radius"] * th.cos(), case["radius"] * th.sin(), z], 1)
    a, b = torch.triu_indices(dpr * rings, dpr * rings, 1, device="cuda")[:, case["row_phase"]::case["row_stride"]]
    p, q = p[a], p[b] - p[a]
    half = [0.5 * case["nx"] * case["vx"], 0.5 * case["ny"] * case["vy"], 0.5 * case["nz"] * case["vz"]]
    lam = torch.zeros(a.numel(), dtype=torch.float64, device="cuda")
    for _ in range(8):
        mid = torch.tensor([rng.uniform(-0.4, 0.4) * h for h in half], dtype=torch.float64, device="cuda")
        axes = torch.tensor([rng.uniform(0.1, 0.5) * h for h in half], dtype=torch.float64, device="cuda")
        u, v = (p - mid) / axes, q / axes
        uu, uv, vv = (u * u).sum(1), (u * v).sum(1), (v * v).sum(1)
        t = (uv * uv - vv * (uu - 1)).clamp_min(0).sqrt() * 2 / vv
        lam += float(rng.uniform(0.2, 1.0)) * t * q.norm(dim=1)
    lam = case["counts"] * (0.95 * lam / max(float(lam.mean()), 1e-30) + 0.05)
    return torch.poisson(lam, generator=torch.Generator("cuda").manual_seed(int(rng.integers(1 << 62)))).int()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kept = _kept(case)
    cols = case["nx"] * case["ny"] * case["nz"]
    s = {"case": case, "kept": kept, "kind": case["kind"], "iterations": case["iterations"],
         "opts": {"spmv": SPMV[case["spmv"]], "bp_mode": BP[case["bp"]]}}
    f0 = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    if case["kind"] == "batch":
        s["g"] = torch.stack([_sinogram(case, rng) for _ in range(case["count"])]).cpu().numpy()
        s["iterations"] = _uneven(case)
        return s
    g = _sinogram(case, rng)
    if case["kind"] in ("host", "mlem"):
        s["g"], s["f0"] = g.cpu().numpy(), f0
        return s
    s["g"], s["f0"] = g, torch.from_numpy(f0).cuda()
    if case["kind"] == "ops":
        s["ratio"] = torch.from_numpy(rng.uniform(0.0, 2.0, g.numel()).astype(np.float32)).cuda()
    return s


def _uneven(case):
    lo, hi = max(1, case["iterations"] // 4), case["iterations"]
    return [lo + 7919 * i % (hi - lo + 1) for i in range(case["count"])]


# ----------------------------------------------------------------------- runs
def run(s):
    m, kind = s["kept"], s["kind"]
    if kind == "run":
        f = s["f0"].clone()
        m.run_device(s["g"].data_ptr(), f.data_ptr(), s["iterations"], torch.cuda.current_stream().cuda_stream,
                     **s["opts"])
        return f
    if kind == "ops":
        stream = torch.cuda.current_stream().cuda_stream
        ratio, fwproj = torch.empty_like(s["ratio"]), torch.empty_like(s["ratio"])
        bp = torch.empty_like(s["f0"])
        m.forward_project(s["f0"].data_ptr(), s["g"].data_ptr(), ratio.data_ptr(), fwproj.data_ptr(), stream,
                          **s["opts"])
        m.back_project(s["ratio"].data_ptr(), bp.data_ptr(), stream, **s["opts"])
        return {"ratio": ratio, "fwproj": fwproj, "bp": bp}
    if kind == "host":
        return m.run(s["g"], s["iterations"], s["f0"], **s["opts"])
    if kind == "batch":
        return m.batch_run(s["g"], s["iterations"])
    rp, col, val, norm = m
    out = np.empty_like(s["f0"])
    c = s["case"]
    pkg.mlem(rp, col, val, None, None, None, s["g"], norm, s["f0"], out, len(rp) - 1, out.size, len(col),
             s["iterations"], 1, SPMV[c["spmv"]], 5, 5, {"trans": 0, "scatter": 1}[c["bp"]])
    return out


def _size(case):
    kept = _kept(case)
    return (len(kept[0]) - 1, len(kept[1])) if case["kind"] == "mlem" else (kept.rows, kept.nnz)


def work(case):
    rows, nnz = _size(case)
    cols = case["nx"] * case["ny"] * case["nz"]
    vb = 4 if case["value"] == "f32" else 2
    ib = 2 if case["compress"] else 4
    a = nnz * (vb + ib) + 8 * rows + 8  # A once
    t = nnz * (vb + ib) + 8 * cols + 8  # its transpose once
    if case["kind"] == "ops":
        return {"bytes": a + t + 4 * cols + 12 * rows + 4 * rows + 4 * cols, "flops": 4 * nnz}
    back = {"trans": t, "scatter": a, "fused": 0}[case["bp"]]
    one = a + back + 4 * cols + 8 * rows + (4 * rows if case["bp"] != "fused" else 0) + 12 * cols
    if case["kind"] == "batch":
        its = _uneven(case)
        # the matrix crosses once per iteration for all sinograms still running
        return {"bytes": max(its) * (a + t) + sum(its) * (16 * cols + 12 * rows), "flops": 4 * nnz * sum(its)}
    flops = 4 * nnz * case["iterations"]
    if case["kind"] == "mlem":  # the matrix in, its transpose made and read
        return {"bytes": case["iterations"] * one + 8 * nnz + (8 * nnz if case["bp"] == "trans" else 0),
                "flops": flops}
    return {"bytes": case["iterations"] * one, "flops": flops}


# ----------------------------------------------------------------- in 64 bits
def exact(case, seed):
    rows, nnz = _size(case)
    s = prepare(case, seed)
    rp, col, val = s["kept"][:3] if case["kind"] == "mlem" else s["kept"].csr()
    cols = case["nx"] * case["ny"] * case["nz"]
    rp, col = torch.from_numpy(rp.astype(np.int64)).cuda(), torch.from_numpy(col.astype(np.int32)).cuda().long()
    val = torch.from_numpy(val).cuda().double()
    a = torch.sparse_csr_tensor(rp, col, val, (rows, cols), check_invariants=False)
    rid = torch.repeat_interleave(torch.arange(rows, device="cuda"), rp[1:] - rp[:-1])
    order = torch.argsort(col, stable=True)
    cp = torch.zeros(cols + 1, dtype=torch.int64, device="cuda")
    cp[1:] = torch.bincount(col, minlength=cols).cumsum(0)
    t = torch.sparse_csr_tensor(cp, rid[order], val[order], (cols, rows), check_invariants=False)
    del rid, order

    def dev(x):
        return (torch.from_numpy(x) if isinstance(x, np.ndarray) else x).cuda().double()

    def over(g, y):
        return torch.where(y != 0, g / torch.where(y != 0, y, 1.0), 0.0)

    g = dev(s["g"])
    if case["kind"] == "ops":
        y = a @ dev(s["f0"])
        return {"ratio": over(g, y), "fwproj": y, "bp": t @ dev(s["ratio"])}
    norm = t @ torch.ones(rows, dtype=torch.float64, device="cuda")
    if case["kind"] == "mlem":
        norm = dev(s["kept"][3])
    its = s["iterations"] if case["kind"] == "batch" else [case["iterations"]]
    if case["kind"] == "batch":
        f0 = (g.sum(1) / norm.sum()).unsqueeze(1).expand(-1, cols)
    else:
        g, f0 = g.unsqueeze(0), dev(s["f0"]).unsqueeze(0)
    out = []
    for gk, f, n in zip(g, f0, its):
        f = f.clone()
        for _ in range(n):
            f = f * (t @ over(gk, a @ f))
            f = torch.where(norm != 0, f / torch.where(norm != 0, norm, 1.0), f)
        out.append(f)
    return torch.stack(out) if case["kind"] == "batch" else out[0]

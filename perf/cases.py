"""Performance cases: the calls a user of this package makes, over the range of sizes it makes them.

A case names one public call sequence (``what``), a matrix family and size (``matrix``, ``rows``), the
feature width (``feats``), the input type of the dense operand (``dtype``) and the number of column
partitions (``parts``).  The matrix families are those of ``liteform_ae_b200.synth``, drawn on the GPU:

  zipf      Zipf(1.8) row lengths, mean 16, uniform columns
  powerlaw  power-law degrees (2.1), mean 14, degree-proportional columns, row-normalised
  uniform   exactly 32 uniform columns per row
  skew      log-normal row lengths plus 64 very long rows
  banded    dense 8x8 blocks, 8 per block row, on a band of +-4096 block columns

  product   C = A B on a composed format that the program keeps     (fa.spmm / hyb.spmm_hyb)
  csr       C = A B straight from CSR, the driver's last resort      (hyb.spmm_csr)
  blocks    C = A B on 8x8 blocks that the program keeps             (bsr.spmm_bsr8)
  build     width search + format, left in device memory             (fa.search_bucket_config,
                                                                      fa.build_hyb_format_device)
  dropin    width search + format as nested NumPy arrays             (fa.build_hyb_format)
  convert   CSR to 8x8 blocks on the device                          (bsr.DeviceBsr8.from_csr_device)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from liteform_ae_b200 import bsr, hyb
from liteform_ae_b200 import format_algos as fa
from liteform_ae_b200 import width_search
from liteform_ae_b200.format_matrix_market import MTX

DEV = "cuda"
PER_ROW = 32                 # entries per row of "uniform"
BLOCKS_PER_ROW = 8           # blocks per block row of "banded"
HALF_BAND = 4096
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}


def _case(name, what, matrix, rows, feats=0, dtype="float32", parts=1):
    c = {"what": what, "matrix": matrix, "rows": rows, "feats": feats, "dtype": dtype, "parts": parts}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small graph's layer: latency and launches are all of it
        _case("product small", "product", "zipf", 2048, 32),
        # the headline workload: a million-node power-law graph at a hidden width of 128
        _case("product graph", "product", "powerlaw", 1 << 20, 128),
        # the largest: uniform rows, B far beyond the L2
        _case("product uniform", "product", "uniform", 1 << 22, 64),
        # very long rows beside short ones, 16-bit features
        _case("product skew bf16", "product", "skew", 1 << 20, 256, "bfloat16"),
        # the last layer of a classifier: as many features as classes, sizes no power of two divides
        _case("product odd width", "product", "powerlaw", 200_003, 47),
        # column partitions, the reference's own lever (its classifier picks their number)
        _case("product partitions", "product", "powerlaw", 1 << 18, 64, parts=4),
        # product without a format, as the driver falls back to
        _case("csr graph", "csr", "powerlaw", 1 << 19, 32),
        # FEM-like blocks in float32
        _case("blocks f32", "blocks", "banded", 1 << 20, 128),
        # the same in the 16-bit type the reference's block path uses, wide features
        _case("blocks f16", "blocks", "banded", 1 << 21, 256, "float16"),
        # composed format of a million-node graph: statistics, width search, construction
        _case("build graph", "build", "powerlaw", 1 << 20, 128),
        # the reference's call sequence on a small matrix: the format goes back to the host
        _case("dropin small", "dropin", "zipf", 16384, 32),
        # the driver's block branch: CSR in device memory to fp16 tiles
        _case("convert blocks", "convert", "banded", 1 << 18, 0, "float16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _gather_cost(case):
    """Bytes of one B row per stored entry plus C: what bounds a product's time from the matrix's side."""
    e = 4 if case["dtype"] == "float32" else 2
    f = case["feats"] + (case["feats"] % 4 != 0) * 2 * case["feats"]   # odd widths gather word by word
    entries = _entries(case) if case["matrix"] != "banded" else _entries(case) / 8
    return entries * (f * e + 8) * case["parts"] ** 0.5 + case["rows"] * f * 4


def draw(rng):
    biggest = _gather_cost(_case(None, "product", "uniform", 1 << 22, 64)) / 2
    while True:
        what = rng.choice(["product"] * 5 + ["csr"] * 2 + ["blocks"] * 2 + ["build", "build", "dropin", "convert"])
        dtype, parts = "float32", 1
        if what in ("blocks", "convert"):
            matrix = "banded"
            rows = 8 * _log_int(rng, 512, 1 << 18)
            dtype = rng.choice(["float32", "bfloat16", "float16"])
            step = 4 if dtype == "float32" else 8
            feats = 0 if what == "convert" else step * _log_int(rng, 1, 512 // step)
            if what == "convert":
                rows = min(rows, 1 << 19)
        else:
            matrix = rng.choice(["zipf", "powerlaw", "powerlaw", "uniform", "skew"])
            rows = _log_int(rng, 2048, 1 << 20)
            feats = _log_int(rng, 8, 512)
            if what == "product":
                dtype = rng.choice(["float32", "float32", "bfloat16"])
                parts = rng.choice([1, 1, 1, 2, 4, 8])
            elif what == "build":
                parts = rng.choice([1, 1, 2, 4, 8])
            if what == "dropin":
                rows = _log_int(rng, 2048, 1 << 17)
            if dtype == "bfloat16":
                feats = max(8, feats // 8 * 8)
            elif rng.random() < 0.6:
                feats = max(4, feats // 4 * 4)      # most programs keep feature widths even
        case = _case(None, what, matrix, rows, feats, dtype, parts)
        if _gather_cost(case) <= biggest:
            return case


# ---- matrices -----------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2 + 1)


def _csr_of_keys(keys, M):
    """Sorted distinct ``row * M + column`` keys to CSR."""
    rows = torch.div(keys, M, rounding_mode="floor")
    indices = (keys - rows * M).to(torch.int32)
    indptr = torch.zeros(M + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(rows, minlength=M), 0, out=indptr[1:])
    return indptr, indices


def _uniform_columns(lens, M, g):
    """For every row as many distinct uniform columns as ``lens`` says."""
    dense = torch.nonzero(lens * 4 > M).flatten().tolist()   # rejection would crawl: cut a permutation
    kept = [r * M + torch.randperm(M, generator=g, device=DEV)[:int(lens[r])] for r in dense]
    dense_keys = torch.cat(kept) if kept else torch.empty(0, dtype=torch.int64, device=DEV)
    want = lens.clone()
    if dense:
        want[dense] = 0
    every = torch.arange(M, device=DEV)
    keys = torch.empty(0, dtype=torch.int64, device=DEV)
    need = want
    while int(need.sum()):
        r = torch.repeat_interleave(every, need)
        c = torch.randint(0, M, (r.numel(),), generator=g, device=DEV)
        keys = torch.unique(torch.cat([keys, r * M + c]))
        need = want - torch.bincount(torch.div(keys, M, rounding_mode="floor"), minlength=M)
    return torch.sort(torch.cat([keys, dense_keys]))[0]


def _skew_heavy(M):
    return 64, min(100_000, M // 8)


def _relabelled(csr, parts, seed):
    """The same graph under other row and column numbers (columns stay in their partition): what a
    format costs and how large it gets depend on the graph alone, every entry moves."""
    M, g = csr.shape[0], _gen(seed)
    size = -(-M // parts)
    col = torch.cat([lo + torch.randperm(min(size, M - lo), generator=g, device=DEV) for lo in range(0, M, size)])
    row = torch.randperm(M, generator=g, device=DEV)
    r = torch.repeat_interleave(torch.arange(M, device=DEV), torch.diff(csr.indptr))
    keys, order = torch.sort(row[r] * M + col[csr.indices.long()])
    indptr, indices = _csr_of_keys(keys, M)
    return hyb.DeviceCsr(indptr, indices, csr.data[order], csr.shape)


def _csr(case, seed):
    M, g = case["rows"], _gen(seed)
    if case["matrix"] == "powerlaw":
        raw = (1.0 - torch.rand(M, generator=g, device=DEV, dtype=torch.float64)) ** (-1.0 / 1.1)
        deg = _scaled_degrees(raw, M, torch)
        weight = torch.cumsum((deg + 1).to(torch.float64), 0)
        r = torch.repeat_interleave(torch.arange(M, device=DEV), deg)
        u = torch.rand(r.numel(), generator=g, device=DEV, dtype=torch.float64) * weight[-1]
        c = torch.searchsorted(weight, u, right=True).clamp_(max=M - 1)
        indptr, indices = _csr_of_keys(torch.unique(r * M + c), M)
        lens = torch.diff(indptr)
        data = torch.repeat_interleave(1.0 / lens.clamp(min=1).to(torch.float32), lens)
        return hyb.DeviceCsr(indptr, indices, data, (M, M))
    if case["matrix"] == "uniform":
        cols = torch.randint(0, M, (M, PER_ROW), generator=g, device=DEV, dtype=torch.int32).sort(1)[0]
        while True:
            bad = torch.nonzero((cols[:, 1:] == cols[:, :-1]).any(1)).flatten()
            if not bad.numel():
                break
            cols[bad] = torch.randint(0, M, (bad.numel(), PER_ROW), generator=g, device=DEV, dtype=torch.int32).sort(1)[0]
        indptr = torch.arange(M + 1, device=DEV) * PER_ROW
        indices = cols.reshape(-1)
    elif case["matrix"] == "banded":
        bptr, bcol = _banded(M, g)
        Mb, n = M // 8, bcol.shape[1]
        cols = (bcol.to(torch.int32)[:, None, :, None] * 8 + torch.arange(8, device=DEV, dtype=torch.int32)).expand(Mb, 8, n, 8)
        indices = cols.reshape(-1).contiguous()
        indptr = torch.arange(M + 1, device=DEV) * (8 * n)
    else:
        if case["matrix"] == "zipf":
            raw = np.clip(np.random.default_rng(seed).zipf(1.8, M), 1, min(2048, M)).astype(np.float64)
            lens = torch.from_numpy(np.clip(np.rint(raw * (16.0 / raw.mean())), 1, min(2048, M)).astype(np.int64)).to(DEV)
        else:
            n = torch.randn(M, generator=g, device=DEV, dtype=torch.float64)
            lens = torch.exp(2.0 + 1.2 * n).round().clamp(1, M).to(torch.int64)
            rows, length = _skew_heavy(M)
            lens[torch.randperm(M, generator=g, device=DEV)[:rows]] = length
        indptr, indices = _csr_of_keys(_uniform_columns(lens, M, g), M)
    data = torch.rand(indices.numel(), generator=g, device=DEV) * 2 - 1
    return hyb.DeviceCsr(indptr, indices, data, (M, M))


def _scaled_degrees(raw, M, xp):
    """Power-law degrees rescaled to a mean of 14 and clipped to [1, 50000]."""
    cap, scale = min(50_000, M), 1.0
    for _ in range(8):
        scale *= 14.0 / float((raw * scale).round().clip(1, cap).mean())
    deg = (raw * scale).round().clip(1, cap)
    return deg.to(torch.int64) if xp is torch else deg


def _banded(M, g):
    """Block columns of a banded block matrix: int64 [M / 8, n], ascending and distinct, diagonal included."""
    Mb = M // 8
    half = min(HALF_BAND, max(1, Mb // 2))
    i = torch.arange(Mb, device=DEV)
    lo, hi = (i - half).clamp(min=0), (i + half).clamp(max=Mb - 1)
    span = (hi - lo + 1).to(torch.float64)
    todo = i
    cols = torch.empty((Mb, BLOCKS_PER_ROW), dtype=torch.int64, device=DEV)
    while todo.numel():
        u = torch.rand((todo.numel(), BLOCKS_PER_ROW - 1), generator=g, device=DEV, dtype=torch.float64)
        fresh = lo[todo, None] + (u * span[todo, None]).to(torch.int64)
        cols[todo] = torch.cat([todo[:, None], fresh], 1).sort(1)[0]
        todo = torch.nonzero((cols[:, 1:] == cols[:, :-1]).any(1)).flatten()
    return torch.arange(Mb + 1, device=DEV) * BLOCKS_PER_ROW, cols


# ---- one case -----------------------------------------------------------------------------------
def prepare(case, seed):
    what, M, N, P = case["what"], case["rows"], case["feats"], case["parts"]
    s = {"what": what, "dtype": case["dtype"], "cfg": fa.CostModelSettings(feat_size=N, num_parts=P)}
    if what == "blocks":
        g = _gen(seed)
        bptr, bcol = _banded(M, g)
        blocks = torch.rand((bcol.numel(), 8, 8), generator=g, device=DEV) * 2 - 1
        s["A"] = bsr.DeviceBsr8(bptr, bcol.reshape(-1).to(torch.int32), blocks.to(DTYPES[case["dtype"]]), (M, M))
    else:
        csr = _relabelled(_csr(case, 0), P, seed) if what in ("build", "dropin") else _csr(case, seed)
        if what == "product":
            stats, hist = hyb.hyb_stats(csr, P)
            s["A"] = hyb.build_hyb_device(csr, width_search.search_from_stats(stats, hist, N, P), with_mask=False)
        elif what in ("build", "dropin"):
            # the program loaded the matrix and has it on the device from an earlier call
            s["A"] = MTX.from_csr(csr.indptr.cpu().numpy(), csr.indices.cpu().numpy(), csr.data.cpu().numpy(), csr.shape)
            s["A"].csr_device(DEV)
        else:
            s["A"] = csr
    if what in ("product", "csr", "blocks"):
        s["B"] = torch.randn((M, N), generator=_gen(seed + 1), device=DEV).to(DTYPES[case["dtype"]])
    torch.cuda.synchronize()
    return s


def run(s):
    what, A = s["what"], s["A"]
    if what == "product":
        return hyb.spmm_hyb(A, s["B"]) if s["dtype"] == "bfloat16" else fa.spmm(A, s["B"])
    if what == "csr":
        return hyb.spmm_csr(A, s["B"])
    if what == "blocks":
        return bsr.spmm_bsr8(A, s["B"])
    if what == "convert":
        b = bsr.DeviceBsr8.from_csr_device(A, dtype=s["dtype"])
        return b.indptr, b.indices, b.blocks
    widths = fa.search_bucket_config(A, s["cfg"].num_parts, s["cfg"])
    flat = np.array([w for part in widths for w in part], dtype=np.int32)
    if what == "dropin":
        rows, cols, mask = fa.build_hyb_format(A, widths)
        return flat, rows, cols, mask
    f = fa.build_hyb_format_device(A, widths, with_mask=False)
    return flat, f.ell_rows, f.rows, f.cols, f.vals, f.zero_rows


# ---- what a pass cannot do without ------------------------------------------------------------------
def _quantile_degrees(M):
    q = (np.arange(65536) + 0.5) / 65536
    return _scaled_degrees((1.0 - q) ** (-1.0 / 1.1), M, np)


def _entries(case):
    """Expected number of stored entries."""
    M = case["rows"]
    if case["matrix"] == "banded":
        return M * 8 * BLOCKS_PER_ROW
    if case["matrix"] == "skew":
        rows, length = _skew_heavy(M)
        return M * math.exp(2.0 + 1.2 ** 2 / 2) + rows * length
    return M * {"uniform": PER_ROW, "zipf": 16, "powerlaw": 14}[case["matrix"]]


def _touched_columns(case):
    """Expected number of columns that hold an entry: rows of B that have to be read."""
    M, nnz = case["rows"], _entries(case)
    if case["matrix"] == "banded":
        return M
    if case["matrix"] == "powerlaw":
        d = _quantile_degrees(M) + 1
        return M * float((1.0 - np.exp(-nnz * d / (d.mean() * M))).mean())
    return M * (1.0 - math.exp(-nnz / M))


def work(case):
    """Each input read once, each output written once (padding of the format not counted)."""
    what, M, N = case["what"], case["rows"], case["feats"]
    e = 4 if case["dtype"] == "float32" else 2
    nnz = _entries(case)
    ptr = 8 * (M + 1)
    dense = _touched_columns(case) * N * e + M * N * 4 if what in ("product", "csr", "blocks") else 0
    if what == "product":
        return {"bytes": nnz * 8 + M * 4 + dense, "flops": 2 * nnz * N}
    if what == "csr":
        return {"bytes": nnz * 8 + ptr + dense, "flops": 2 * nnz * N}
    if what == "blocks":
        return {"bytes": nnz * e + nnz / 64 * 4 + ptr / 8 + dense, "flops": 2 * nnz * N}
    if what == "convert":
        return {"bytes": nnz * 8 + ptr + nnz * e + nnz / 64 * 4 + ptr / 8, "flops": 0}
    # statistics read the columns; the format reads columns and values and writes both and a row id each
    made = nnz * (8 if what == "build" else 9) + M * 4
    return {"bytes": nnz * (8 if what == "build" else 4) + ptr + made, "flops": 0}


def tolerance(case):
    # float32 accumulation of exact (or rounded once) inputs in any order; formats are whole numbers and copies
    return {"rel": 1e-5} if case["what"] in ("product", "csr", "blocks") else "exact"

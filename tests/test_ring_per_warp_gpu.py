"""``spmm_hyb_ring_kernel``, the ring per warp that large products take, on small matrices (slot threshold 1): ranges
and orders of the blocks, rows cut by ranges, one and three partitions, operands that are column windows, B in
float32 and bf16.  Every test asks the library that this is the kernel it runs.

Tolerance: the float32 product's (rel 1e-5 / abs 1e-4 against float64; no row has more than 2500 entries)."""
import itertools

import numpy as np
import pytest

from liteform_ae_b200 import _cabi, hyb, synth

pytestmark = pytest.mark.gpu
NAME = "spmm_hyb_ring_kernel"


@pytest.fixture(autouse=True)
def options():
    lib = _cabi.load()
    assert lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, 1) == 0
    yield lib
    lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, 1 << 20)
    lib.lf_set_option(_cabi.LF_OPT_SPMM_SLOTS_PER_GROUP, 0)
    lib.lf_set_option(_cabi.LF_OPT_SPMM_TILE_SEGMENTS, 0)
    lib.lf_set_option(_cabi.LF_OPT_SPMM_GATHER_RING, 16)


@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("N", [68, 100, 128])
def test_order_of_the_register_kernel(cuda_device, options, parts, N):
    import torch
    csr = synth.skewed_rows(M=6000, seed=8, heavy_rows=5, heavy_len=2500)
    d = hyb.DeviceCsr.from_host(csr.indptr, csr.indices, csr.data, csr.shape, cuda_device)
    fmt = hyb.build_hyb_device(d, [[1, 2, 4, 8, 16, 64]] if parts == 1 else [[1, 4, 32], [2, 8], [1, 2, 4, 8, 16]], with_mask=False)
    B = torch.from_numpy(synth.dense_features(6000, N, 3)).to(cuda_device)
    want = csr.toscipy().astype(np.float64) @ B.cpu().numpy().astype(np.float64)
    short = np.diff(csr.indptr) <= 64       # one ELL row, one range, no atomics
    for slots, segments in itertools.product((0, 8, 40, 4096), (0, 7)):
        assert options.lf_set_option(_cabi.LF_OPT_SPMM_SLOTS_PER_GROUP, slots) == 0
        assert options.lf_set_option(_cabi.LF_OPT_SPMM_TILE_SEGMENTS, segments) == 0
        assert options.lf_set_option(_cabi.LF_OPT_SPMM_GATHER_RING, 0) == 0
        base = hyb.spmm_hyb(fmt, B).cpu().numpy()
        assert options.lf_set_option(_cabi.LF_OPT_SPMM_GATHER_RING, 16) == 0
        C = torch.full((6000, N), float("nan"), device=cuda_device)
        assert hyb.spmm_hyb_kernel_name(fmt, B, C) == NAME
        got = hyb.spmm_hyb(fmt, B, out=C).cpu().numpy()
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-4, err_msg=f"{slots} {segments}")
        if parts == 1:
            assert np.array_equal(got[short], base[short])


@pytest.mark.parametrize("dtype,N", [("float32", 128), ("float32", 320), ("bfloat16", 136), ("bfloat16", 256), ("bfloat16", 264)])
def test_column_windows(cuda_device, options, dtype, N):
    """70 000 columns: at 320 features B is larger than what the group form takes."""
    import torch
    M, K, g = 9000, 70_000, torch.Generator(device=cuda_device).manual_seed(4)
    lens = torch.randint(0, 61, (M,), generator=g, device=cuda_device)
    lens[::1500] = 900
    rows = torch.repeat_interleave(torch.arange(M, device=cuda_device), lens)
    keys = torch.unique(rows * K + torch.randint(0, K, (rows.numel(),), generator=g, device=cuda_device))
    rows, cols = keys // K, keys % K
    indptr = torch.zeros(M + 1, dtype=torch.int64, device=cuda_device)
    torch.cumsum(torch.bincount(rows, minlength=M), 0, out=indptr[1:])
    vals = torch.rand(keys.numel(), generator=g, device=cuda_device) * 2 - 1
    d = hyb.DeviceCsr(indptr, cols.to(torch.int32), vals, (M, K))
    wide = torch.randn((K, N + 24), device=cuda_device, generator=g).to(getattr(torch, dtype))
    B = wide[:, 16:16 + N]
    want = torch.zeros((M, N), dtype=torch.float64, device=cuda_device)
    want.index_add_(0, rows, B[cols].double() * vals.double()[:, None])
    for widths in ([[1, 2, 8, 32]], [[1, 4, 16], [2, 64]]):
        fmt = hyb.build_hyb_device(d, widths, with_mask=False)
        C = torch.full((M, N + 8), float("nan"), device=cuda_device)
        out = C[:, 4:4 + N]
        assert hyb.spmm_hyb_kernel_name(fmt, B, out) == NAME
        hyb.spmm_hyb(fmt, B, out=out)
        torch.testing.assert_close(out.double(), want, rtol=1e-5, atol=1e-4)
        hyb.spmm_hyb(fmt, B, out=out, accumulate=True)
        torch.testing.assert_close(out.double(), 2 * want, rtol=1e-5, atol=2e-4)
        assert torch.isnan(C[:, :4]).all() and torch.isnan(C[:, 4 + N:]).all()

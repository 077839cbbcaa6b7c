"""The composed-format product on both sides of every line of the rule that picks its kernel: rows of B
around 128 and 256 bytes, a B that stays in the L2 and one that does not, more columns than 512-byte rows
are taken whole for, buckets narrower than a step, rows cut by groups, one and two partitions.

Tolerance: the float32 product's (rel 1e-5 / abs 1e-4 against float64; no row has more than 600 entries)."""
import pytest

from liteform_ae_b200 import _cabi, hyb

pytestmark = pytest.mark.gpu
M = 12000


@pytest.fixture(scope="module", params=[30_000, 300_000, (1 << 19) + 8])
def matrix(request, cuda_device):
    import torch
    K, g = request.param, torch.Generator(device=cuda_device).manual_seed(7)
    lens = torch.randint(0, 81, (M,), generator=g, device=cuda_device)
    lens[::1000], lens[5:40] = 600, 0
    rows = torch.repeat_interleave(torch.arange(M, device=cuda_device), lens)
    cols = torch.randint(0, K, (rows.numel(),), generator=g, device=cuda_device)
    keys = torch.unique(rows * K + cols)
    rows, cols = keys // K, keys % K
    indptr = torch.zeros(M + 1, dtype=torch.int64, device=cuda_device)
    torch.cumsum(torch.bincount(rows, minlength=M), 0, out=indptr[1:])
    vals = torch.rand(keys.numel(), generator=g, device=cuda_device) * 2 - 1
    csr = hyb.DeviceCsr(indptr, cols.to(torch.int32), vals, (M, K))
    lib = _cabi.load()
    assert lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, 1) == 0
    yield csr, rows, [hyb.build_hyb_device(csr, w, with_mask=False) for w in ([[1, 2, 8, 32]], [[1, 4, 16], [2, 64]])]
    lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, 1 << 20)


@pytest.mark.parametrize("dtype,N", [("float32", n) for n in (4, 28, 32, 36, 64, 68, 72, 128, 132)] +
                         [("bfloat16", n) for n in (8, 64, 72, 128, 136, 248, 256, 264)])
def test_forms(matrix, cuda_device, dtype, N):
    import torch
    csr, rows, formats = matrix
    K = csr.shape[1]
    wide = torch.randn((K, N + 8), device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(N)).to(getattr(torch, dtype))
    B = wide[:, 8:]
    want = torch.zeros((M, N), dtype=torch.float64, device=cuda_device)
    want.index_add_(0, rows, B[csr.indices.long()].double() * csr.data.double()[:, None])
    for fmt in formats:
        C = torch.full((M, N + 8), float("nan"), device=cuda_device)
        hyb.spmm_hyb(fmt, B, out=C[:, 4:4 + N])
        torch.testing.assert_close(C[:, 4:4 + N].double(), want, rtol=1e-5, atol=1e-4)
        assert torch.isnan(C[:, :4]).all() and torch.isnan(C[:, 4 + N:]).all()
        C = torch.ones((M, N), device=cuda_device)
        hyb.spmm_hyb(fmt, B, out=C, accumulate=True)
        torch.testing.assert_close(C.double(), want + 1, rtol=1e-5, atol=2e-4)
    for fmt in formats:
        row, slots = N * (4 if dtype == "float32" else 2), int(fmt.slot_off[-1])
        reach = min(K, slots)
        fits = reach * row <= (104 if row <= 128 else 80) << 20
        if fits and (row <= 128 or (dtype == "float32" and (row <= 256 or row > 512))):   # 65 to 128 features: many slots
            name = "spmm_hyb_groups_kernel"
        elif row <= 256 or (dtype == "bfloat16" and N >= 256 and reach >= 1 << 19):
            name = "spmm_hyb_ring_rows_kernel"
        else:
            name = "spmm_hyb_ring_kernel"
        assert hyb.spmm_hyb_kernel_name(fmt, B, C) == name
    if K > 1 << 19:    # both ways of a wide bf16 row are reached, with plain stores and with atomic adds
        assert min(int(f.slot_off[-1]) for f in formats) >= 1 << 19

"""Rounding error of the products against float64, beside float32 sums in a stated order computed with torch.

The order is the reference here: a row in ``chains`` interleaved chains (the forms for a B larger than the L2
keep two or four per row), or in ranges of entries added one behind the other.  The root mean square over
more than 100 000 sums is known to 0.2 %, so a product passes with up to 3 % more than the order leaves
(64 long rows, 4096 sums: known to 1.1 %, up to 8 % more)."""
import numpy as np
import pytest

from liteform_ae_b200 import _cabi, hyb

pytestmark = pytest.mark.gpu
K = 20_000


def _matrix(rows, n, device, seed):
    """``rows`` rows of ``n`` entries at random places (sorted, distinct columns)."""
    import torch
    g = torch.Generator(device=device).manual_seed(seed)
    cols = torch.stack([torch.randperm(K, generator=g, device=device)[:n].sort()[0] for _ in range(min(rows, 64))])
    cols = cols.repeat(-(-rows // len(cols)), 1)[:rows].contiguous()
    vals = torch.rand((rows, n), generator=g, device=device) * 2 - 1
    indptr = torch.arange(rows + 1, device=device) * n
    return hyb.DeviceCsr(indptr, cols.to(torch.int32).reshape(-1), vals.reshape(-1), (rows, K)), cols, vals


def _fma(acc, v, x):   # one rounding of a float32 multiply-add: the product of two float32 is exact in float64
    return (acc.double() + v.double() * x.double()).float()


def _interleaved(vals, X, chains):
    import torch
    p = [torch.zeros_like(X[:, 0]) for _ in range(chains)]
    for j in range(X.shape[1]):
        p[j % chains] = _fma(p[j % chains], vals[:, j, None], X[:, j])
    while len(p) > 1:
        p = [a + b for a, b in zip(p[:len(p) // 2], p[len(p) // 2:])]
    return p[0]


def _ranges(vals, X, length, chains=1):
    total = None
    for a in range(0, X.shape[1], length):
        s = _interleaved(vals[:, a:a + length], X[:, a:a + length], chains)
        total = s if total is None else total + s
    return total


def _rms(x, exact):
    return float(((x.double() - exact) ** 2).mean().sqrt())


def _features(N, dtype, device):
    import torch
    B = torch.randn((K, N), device=device, generator=torch.Generator(device=device).manual_seed(N))
    return B.to(getattr(torch, dtype))


@pytest.mark.parametrize("n", [4, 16, 32, 64, 256])
@pytest.mark.parametrize("dtype,N,chains", [("float32", 16, 4), ("float32", 32, 4), ("float32", 64, 2), ("float32", 128, 1),
                                            ("bfloat16", 32, 4), ("bfloat16", 64, 4), ("bfloat16", 128, 2)])
def test_rows_of_one_ell_row(cuda_device, n, dtype, N, chains):
    """2^20 slots and more, from where the forms for a larger B keep several partial sums."""
    csr, cols, vals = _matrix(max(4096, (1 << 20) // n), n, cuda_device, n)
    fmt = hyb.build_hyb_device(csr, [[n]], with_mask=False)
    B = _features(N, dtype, cuda_device)
    X = B[:, :8].float()[cols]
    exact = (X.double() * vals.double()[:, :, None]).sum(1)
    got = hyb.spmm_hyb(fmt, B)
    assert (hyb.spmm_hyb_kernel_name(fmt, B, got) == "spmm_hyb_groups_kernel") == (N <= 64)
    assert _rms(got[:, :8], exact) <= 1.03 * _rms(_interleaved(vals, X, chains), exact)


@pytest.mark.parametrize("n", [5, 32, 64])
@pytest.mark.parametrize("dtype,N", [("float32", n) for n in (12, 32, 64, 128, 260)] + [("bfloat16", n) for n in (32, 64, 128)])
def test_small_products_have_the_sums_of_the_register_kernel(cuda_device, n, dtype, N):
    csr, cols, vals = _matrix(2000, n, cuda_device, n)
    fmt = hyb.build_hyb_device(csr, [[8, 32] if n < 64 else [64]], with_mask=False)
    B = _features(N, dtype, cuda_device)
    got, lib = hyb.spmm_hyb(fmt, B), _cabi.load()
    assert hyb.spmm_hyb_kernel_name(fmt, B, got) == "spmm_hyb_groups_kernel"
    assert lib.lf_set_option(_cabi.LF_OPT_SPMM_GATHER_RING, 0) == 0
    try:
        assert (got == hyb.spmm_hyb(fmt, B)).all()
    finally:
        lib.lf_set_option(_cabi.LF_OPT_SPMM_GATHER_RING, 16)


@pytest.mark.parametrize("N", [200, 512])
def test_rows_of_eight_ell_rows_with_blocks_along_y(cuda_device, N):
    """2^20 slots: chains are the ranges of 32 slots, although longer ranges fill the chip."""
    csr, cols, vals = _matrix(4096, 256, cuda_device, 8)
    fmt = hyb.build_hyb_device(csr, [[32]], with_mask=False)
    B = _features(N, "float32", cuda_device)
    X = B[:, :8][cols]
    exact = (X.double() * vals.double()[:, :, None]).sum(1)
    got = hyb.spmm_hyb(fmt, B)
    assert hyb.spmm_hyb_kernel_name(fmt, B, got) == "spmm_hyb_groups_kernel"
    assert _rms(got[:, :8], exact) <= 1.03 * _rms(_ranges(vals, X, 32), exact)


@pytest.mark.parametrize("dtype,N,chains", [("float32", 32, 4), ("float32", 64, 2), ("bfloat16", 64, 4)])
def test_long_rows(cuda_device, dtype, N, chains):
    """Rows shared by hundreds of ranges: the sums of 32 entries a range, added one behind the other."""
    csr, cols, vals = _matrix(64, 16_384, cuda_device, 3)
    fmt = hyb.build_hyb_device(csr, [[32]], with_mask=False)
    B = _features(N, dtype, cuda_device)
    sums = [], []
    for f in range(0, 64 if N >= 64 else 32, 8):
        X = B[:, f:f + 8].float()[cols]
        exact = (X.double() * vals.double()[:, :, None]).sum(1)
        sums[0].append(_rms(hyb.spmm_hyb(fmt, B)[:, f:f + 8], exact) ** 2)
        sums[1].append(_rms(_ranges(vals, X, 32, chains), exact) ** 2)
    assert np.mean(sums[0]) ** 0.5 <= 1.08 * np.mean(sums[1]) ** 0.5


@pytest.mark.parametrize("N,lanes", [(32, 8), (64, 16), (128, 32), (200, 32), (47, 32), (9, 32)])
def test_csr_rows_of_256_entries(cuda_device, N, lanes):
    """3.7 M entries: chains of as many entries as fill the chip eight times, at 32 entries or more."""
    import torch
    csr, cols, vals = _matrix(14_336, 256, cuda_device, 5)
    chain, blocks = 256, torch.cuda.get_device_properties(cuda_device).multi_processor_count * 3 * 8
    while chain > 32 and -(-csr.nnz // (chain * (256 // lanes))) < blocks:
        chain //= 2
    B = _features(N, "float32", cuda_device)
    X = B[:, :8][cols]
    exact = (X.double() * vals.double()[:, :, None]).sum(1)
    assert _rms(hyb.spmm_csr(csr, B)[:, :8], exact) <= 1.03 * _rms(_ranges(vals, X, chain), exact)

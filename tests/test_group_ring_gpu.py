"""The gather ring for groups of 4, 8, 16 and 32 lanes at the sizes where it can go wrong: feature counts
around the capacity of a group (4 G aligned, 4 G - 4 not), row changes at every place of a strip, runs
of empty rows longer than a strip, rows cut by group boundaries, operands off the 16-byte grid.

Tolerance: the float32 product's (rel 1e-5 / abs 1e-4 against SciPy in float64; no row has more than
4096 entries)."""
import numpy as np
import pytest

from liteform_ae_b200 import _cabi, hyb, synth

pytestmark = pytest.mark.gpu
K = 3000


def _matrix():
    """Row lengths 0 .. 70 in order, runs of 7 / 8 / 33 / 100 empty rows, rows of exactly 8, 16, 32 and 256
    entries back to back, three long rows, a tail of single entries."""
    lens = list(range(71)) + [0] * 7 + [1] + [0] * 8 + [2] + [0] * 33 + [3] + [0] * 100 + [8] * 9 + [16] * 9 + [32] * 9 + \
        [256] * 3 + [2999, 5, 1500, 0, 700] + [1] * 301 + [0] * 40
    rng = np.random.default_rng(11)
    indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    indices = np.concatenate([np.sort(rng.permutation(K)[:n]) for n in lens if n]).astype(np.int32)
    return synth.Csr(indptr, indices, rng.uniform(-1, 1, len(indices)).astype(np.float32), (len(lens), K))


@pytest.fixture(scope="module", params=[1 << 20, 0], ids=["groups", "slots"])
def setup(request, cuda_device):
    """The composed-format product by groups of lanes (a small product) and, with a threshold of 0, by consecutive
    slots per step; the CSR product has the group ring alone."""
    csr = _matrix()
    d = hyb.DeviceCsr.from_host(csr.indptr, csr.indices, csr.data, csr.shape, cuda_device)
    lib = _cabi.load()
    assert lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, request.param) == 0
    yield csr, d, hyb.build_hyb_device(d, [[1, 2, 4, 16, 64]], with_mask=False), csr.toscipy().astype(np.float64)
    lib.lf_set_option(_cabi.LF_OPT_SPMM_RING_MIN_SLOTS, 1 << 20)


@pytest.mark.parametrize("N", [1, 4, 7, 28, 29, 32, 36, 47, 60, 61, 64, 65, 100, 124, 125, 128, 130, 260])
def test_products_around_the_group_capacity(setup, cuda_device, N):
    import torch
    csr, d, fmt, A = setup
    wide = torch.from_numpy(synth.dense_features(K, N + 9, 5)).to(cuda_device)
    for shift in (0, 1, 3):             # shift 0 with N + 9 columns: a leading dimension off the grid
        B = wide[:, shift:shift + N]
        for b in (B, B.contiguous()):
            want = A @ b.cpu().numpy().astype(np.float64)
            for product in (lambda out: hyb.spmm_csr(d, b, out=out), lambda out: hyb.spmm_hyb(fmt, b, out=out)):
                C = torch.full((csr.shape[0], N + 5), float("nan"), device=cuda_device)
                product(C[:, 2:2 + N])
                got = C.cpu().numpy()
                np.testing.assert_allclose(got[:, 2:2 + N], want, rtol=1e-5, atol=1e-4)
                assert np.isnan(got[:, :2]).all() and np.isnan(got[:, 2 + N:]).all()


@pytest.mark.parametrize("dtype,N", [("float32", n) for n in (4, 12, 16, 20, 28, 32, 36, 48, 60, 64, 68, 100, 124, 128, 132, 256, 260)] +
                         [("bfloat16", n) for n in (8, 32, 40, 64, 72, 120, 128)])
def test_operands_on_the_16_byte_grid(request, setup, cuda_device, dtype, N):
    """Contiguous operands and column windows of wider ones, C written and added to, next to untouched columns."""
    import torch
    csr, d, fmt, A = setup
    slots = "slots" in request.node.callspec.id.split("-")
    wide = torch.from_numpy(synth.dense_features(K, N + 16, 5)).to(cuda_device).to(getattr(torch, dtype))
    for B in (wide[:, 8:8 + N], wide[:, 8:8 + N].contiguous()):
        want = A @ B.float().cpu().numpy().astype(np.float64)
        C = torch.full((csr.shape[0], N + 8), float("nan"), device=cuda_device)
        out = C[:, 4:4 + N]
        assert hyb.spmm_hyb_kernel_name(fmt, B, out) == ("spmm_hyb_ring_rows_kernel" if slots else "spmm_hyb_groups_kernel")
        hyb.spmm_hyb(fmt, B, out=out)
        np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=1e-4)
        hyb.spmm_hyb(fmt, B, out=out, accumulate=True)
        np.testing.assert_allclose(out.cpu().numpy(), 2 * want, rtol=1e-5, atol=2e-4)
        if dtype == "float32":
            out.fill_(float("nan"))
            hyb.spmm_csr(d, B, out=out)
            np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=1e-4)
        assert torch.isnan(C[:, :4]).all() and torch.isnan(C[:, 4 + N:]).all()


@pytest.mark.parametrize("N", [32, 47, 64, 128])
def test_csr_row_ranges_and_missing_values(setup, cuda_device, N):
    import torch
    csr, d, fmt, A = setup
    B = torch.from_numpy(synth.dense_features(K, N, 6)).to(cuda_device)
    want = A @ B.cpu().numpy().astype(np.float64)
    for r0, r1 in ((0, 1), (5, 6), (70, 240), (229, csr.shape[0]), (csr.shape[0] - 10, csr.shape[0])):
        C = torch.full((r1 - r0, N), float("nan"), device=cuda_device)
        hyb.spmm_csr(d, B, out=C, row_range=(r0, r1))
        np.testing.assert_allclose(C.cpu().numpy(), want[r0:r1], rtol=1e-5, atol=1e-4)
    ones = hyb.DeviceCsr(d.indptr, d.indices, None, d.shape)
    P = csr.toscipy().astype(np.float64)
    P.data[:] = 1.0
    want = P @ B.cpu().numpy().astype(np.float64)
    # sums of up to 2999 terms of size 1 instead of 0.5: twice the absolute part
    np.testing.assert_allclose(hyb.spmm_csr(ones, B).cpu().numpy(), want, rtol=1e-5, atol=2e-4)

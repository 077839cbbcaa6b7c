"""Columns per set of width classes: pairwise sums against the definition (the bins that intersect the set)."""
import numpy as np
import pytest

from liteform_ae_b200 import hyb, synth, width_search as ws


def test_pairwise_sums_equal_the_definition():
    rng = np.random.default_rng(3)
    hist = rng.integers(0, 1 << 40, (3, ws.BINS)) * (rng.random((3, ws.BINS)) < 0.2)
    hist[2] = 0
    bins = np.arange(ws.BINS)
    got = ws.coverage_from_hist(hist)
    for c in [0, 1, 2, 1024, 2047, 2046] + rng.integers(0, ws.BINS, 40).tolist():
        np.testing.assert_array_equal(got[:, c], hist[:, (bins & c) != 0].sum(1))


@pytest.mark.gpu
@pytest.mark.parametrize("parts", [1, 2, 7])
def test_device_table_equals_the_host_table(cuda_device, parts):
    csr = synth.skewed_rows(M=4096, seed=8, heavy_rows=4, heavy_len=3000)
    d = hyb.DeviceCsr.from_host(csr.indptr, csr.indices, csr.data, csr.shape, cuda_device)
    stats, hist = hyb.hyb_stats(d, parts)
    for workspace in (None, hyb.Workspace(cuda_device)):
        stats_c, coverage = hyb.hyb_coverage(d, parts, workspace)
        np.testing.assert_array_equal(stats_c, stats)
        np.testing.assert_array_equal(coverage, ws.coverage_from_hist(hist))

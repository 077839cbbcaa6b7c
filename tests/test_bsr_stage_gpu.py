"""CSR -> 8x8 blocks where a warp's 32 rows just fit its stage in shared memory, just do not, or hold one
long row among short ones; rows with repeated columns (the last value counts); more block rows than one
step of the scan.  Whole numbers and copies: exact, against a walk over each block row in Python."""
import numpy as np
import pytest

from liteform_ae_b200 import bsr, hyb

pytestmark = pytest.mark.gpu
K = 40_000


def _blocks(indptr, indices, data):
    """Dictionary per block row: block column -> 8x8 tile, later entries over earlier ones."""
    ptr, cols, tiles = [0], [], []
    M = len(indptr) - 1
    for I in range(0, M, 8):
        found = {}
        for r in range(I, min(I + 8, M)):
            for e in range(indptr[r], indptr[r + 1]):
                t = found.setdefault(int(indices[e]) >> 3, np.zeros((8, 8), np.float32))
                t[r - I, int(indices[e]) & 7] = data[e]
        cols += sorted(found)
        tiles += [found[c] for c in sorted(found)]
        ptr.append(len(cols))
    return np.array(ptr), np.array(cols, dtype=np.int32), np.array(tiles, dtype=np.float32).reshape(-1, 8, 8)


def _check(lens, device, seed, repeat=0):
    import torch
    rng = np.random.default_rng(seed)
    indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    rows = []
    for n in lens:
        if repeat and n:
            rows.append(np.sort(rng.integers(0, max(1, n // repeat), n)))
        else:   # dense stretches and scattered columns
            rows.append(np.arange(n) + 3 if n % 3 == 0 else np.sort(rng.permutation(K)[:n]))
    indices = np.concatenate(rows).astype(np.int32)
    data = rng.uniform(0.5, 1.5, len(indices)).astype(np.float32)
    up = lambda x: torch.from_numpy(x).to(device)
    d = hyb.DeviceCsr(up(indptr), up(indices), up(data), (len(lens), K))      # unchecked: repeated columns pass
    a = bsr.DeviceBsr8.from_csr_device(d, "float32")
    ptr, cols, tiles = _blocks(indptr, indices, data)
    np.testing.assert_array_equal(a.indptr.cpu().numpy(), ptr)
    np.testing.assert_array_equal(a.indices.cpu().numpy(), cols)
    np.testing.assert_array_equal(a.blocks.cpu().numpy(), tiles)


@pytest.mark.parametrize("lens", [
    [64] * 32, [64] * 31 + [65], [2048] + [0] * 31, [2049] + [0] * 31, [0] * 31 + [2049], [3] * 13 + [5000] + [7] * 25,
    [31, 32, 33, 8, 9, 7, 0, 1] * 9, [1] * 37, [700] * 33, [0] * 40 + [5],
], ids=lambda x: f"{len(x)}rows{sum(x)}")
def test_stage_and_windows(cuda_device, lens):
    _check(lens, cuda_device, sum(lens))


@pytest.mark.parametrize("lens", [[60] * 40, [300] * 40])
@pytest.mark.parametrize("repeat", [2, 9])
def test_repeated_columns(cuda_device, lens, repeat):
    _check(lens, cuda_device, repeat, repeat)


@pytest.mark.parametrize("block_rows", [255, 8192, 8193, 20_000])
def test_scan_steps(cuda_device, block_rows):
    lens = np.zeros(block_rows * 8, dtype=np.int64)
    lens[::5] = 2
    indptr = np.concatenate([[0], np.cumsum(lens)])
    indices = np.tile(np.array([1, 77], dtype=np.int32), int(lens.sum()) // 2)
    d = hyb.DeviceCsr.from_host(indptr, indices, np.ones(len(indices), np.float32), (len(lens), K), cuda_device)
    a = bsr.DeviceBsr8.from_csr_device(d, "float16")
    has = lens.reshape(-1, 8).any(1)
    np.testing.assert_array_equal(a.indptr.cpu().numpy(), np.concatenate([[0], np.cumsum(2 * has)]))
    np.testing.assert_array_equal(a.indices.cpu().numpy(), np.tile([0, 9], int(has.sum())))

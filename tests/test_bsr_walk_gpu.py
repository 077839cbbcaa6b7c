"""CSR -> 8x8 blocks at the edges of the walk's three ways to consume a block: scattered entries (the window
of eight columns moves up by one), full tile rows on 16-byte boundaries (two 16-byte loads), anything else
(entry by entry); one long row among short ones; rows with repeated columns (the last value counts); more
block rows than one step of the scan.  Whole numbers and copies: exact, against a walk over each block row
in Python."""
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
def test_row_lengths(cuda_device, lens):
    _check(lens, cuda_device, sum(lens))


def _check_rows(rows, device, offset=0, with_data=True):
    """``rows``: list of column arrays; the arrays start ``offset`` elements behind a 16-byte boundary."""
    import torch
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    indices = np.concatenate(rows).astype(np.int32)
    data = np.arange(1, len(indices) + 1, dtype=np.float32) if with_data else np.ones(len(indices), np.float32)

    def up(x):
        buf = torch.empty(len(x) + 8, dtype=torch.from_numpy(x[:0]).dtype, device=device)[offset:offset + len(x)]
        return buf.copy_(torch.from_numpy(x))
    d = hyb.DeviceCsr(torch.from_numpy(indptr).to(device), up(indices), up(data) if with_data else None, (len(rows), K))
    a = bsr.DeviceBsr8.from_csr_device(d, "float32")
    ptr, cols, tiles = _blocks(indptr, indices, data)
    np.testing.assert_array_equal(a.indptr.cpu().numpy(), ptr)
    np.testing.assert_array_equal(a.indices.cpu().numpy(), cols)
    np.testing.assert_array_equal(a.blocks.cpu().numpy(), tiles)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("with_data", [True, False])
def test_full_blocks_and_what_follows_them(cuda_device, offset, with_data):
    """Runs of full blocks followed by 0 .. 9 further entries, on and off the 16-byte grid, some warps of full
    blocks alone, some beside scattered rows, one group of eight rows done long before its neighbours."""
    full = lambda *blocks: np.concatenate([np.arange(8) + 8 * b for b in blocks])
    rows = [full(3, 4, 9)] * 32                                                   # nothing but full blocks
    rows += [np.concatenate([full(1, 2), np.arange(k) + 40]) for k in range(10)]  # a rest of 0 .. 9
    rows += [np.concatenate([np.arange(k), full(2, 5)]) for k in range(8)]        # starts off the grid
    rows += [full(7)[1:], full(7)[:7], full(7), full(6, 7)] * 3
    rows += [full(*range(40))] * 8 + [np.array([5])] * 8 + [full(11)] * 16        # one long group
    rows += [np.arange(100) * 8 + r for r in range(8)] + [np.arange(100) * 64 for _ in range(24)]   # scattered
    _check_rows(rows, cuda_device, offset, with_data)


def test_rows_that_are_not_sorted_keep_their_meaning(cuda_device):
    """Unsorted columns are outside the contract; runs of one block still make one tile each, in order."""
    import torch
    rows = [[40, 41, 8, 9, 42]] + [[]] * 7
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    up = lambda x: torch.from_numpy(x).to(cuda_device)
    d = hyb.DeviceCsr(up(indptr), up(np.array(rows[0], np.int32)), up(np.arange(1, 6, dtype=np.float32)), (8, K))
    a = bsr.DeviceBsr8.from_csr_device(d, "float32")
    assert a.indices.cpu().tolist() == [5, 1, 5]
    assert a.blocks.cpu().numpy()[:, 0].tolist() == [[1, 2, 0, 0, 0, 0, 0, 0], [3, 4, 0, 0, 0, 0, 0, 0], [0, 0, 5, 0, 0, 0, 0, 0]]


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

"""The C view that a ``HybFormat`` keeps between products follows every change of the format."""
import copy
import pickle

import numpy as np
import pytest

from liteform_ae_b200 import hyb, synth

pytestmark = pytest.mark.gpu


def test_kept_view_follows_the_format(cuda_device):
    import torch
    csr = synth.zipf_rows(M=1024, seed=3)
    d = hyb.DeviceCsr.from_host(csr.indptr, csr.indices, csr.data, csr.shape, cuda_device)
    fmt = hyb.build_hyb_device(d, [[1, 2, 4, 8]], with_mask=False)
    B = torch.from_numpy(synth.dense_features(1024, 32, 1)).to(cuda_device)
    want = csr.toscipy().astype(np.float64) @ B.cpu().numpy().astype(np.float64)

    def check(f, scale):   # one float32 rounding more per entry than the bound of the product tests allows for
        np.testing.assert_allclose(hyb.spmm_hyb(f, B).cpu().numpy(), scale * want, rtol=1e-5, atol=1e-4 * scale)

    check(fmt, 1)
    fmt.vals.mul_(2)                       # same address
    check(fmt, 2)
    fmt.vals = fmt.vals * 2                # another array
    check(fmt, 4)
    other = copy.copy(fmt)
    other.vals = fmt.vals / 4
    check(other, 1)
    check(fmt, 4)
    check(pickle.loads(pickle.dumps(fmt)), 4)

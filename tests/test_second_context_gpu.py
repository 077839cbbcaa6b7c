"""Products in a second context of the device: a kernel's shared-memory limit is raised there too, whatever an
earlier product raised in the first one.  (A host that embeds the library may run it in a context of its own.)"""
import ctypes

import numpy as np
import pytest

from liteform_ae_b200 import _cabi, hyb, synth

pytestmark = pytest.mark.gpu


def test_csr_product_in_a_context_of_its_own(cuda_device):
    import torch
    csr = synth.zipf_rows(M=512, seed=2)
    N = 64
    B = synth.dense_features(512, N, 1)
    want = csr.toscipy().astype(np.float64) @ B.astype(np.float64)
    d = hyb.DeviceCsr.from_host(csr.indptr, csr.indices, csr.data, csr.shape, cuda_device)
    np.testing.assert_allclose(hyb.spmm_csr(d, torch.from_numpy(B).to(cuda_device)).cpu().numpy(), want, rtol=1e-5, atol=1e-4)
    torch.cuda.synchronize()

    cu, lib = ctypes.CDLL("libcuda.so.1"), _cabi.load()

    def ok(status):
        assert status == 0, f"driver call failed with {status}"
    dev, ctx = ctypes.c_int(), ctypes.c_void_p()
    ok(cu.cuDeviceGet(ctypes.byref(dev), cuda_device.index))
    ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev))      # the current context of this thread from here on
    try:
        def up(x):
            x = np.ascontiguousarray(x)
            p = ctypes.c_uint64()
            ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(x.nbytes)))
            ok(cu.cuMemcpyHtoD_v2(p, ctypes.c_void_p(x.ctypes.data), ctypes.c_size_t(x.nbytes)))
            return p.value
        C = np.zeros((512, N), np.float32)
        ptr, idx, val, b, c = (up(x) for x in (csr.indptr.astype(np.int64), csr.indices.astype(np.int32),
                                              csr.data.astype(np.float32), B.astype(np.float32), C))
        _cabi.check(lib.lf_spmm_csr_f32(ptr, idx, val, 0, 512, len(csr.indices), b, N, c, N, N, None))
        ok(cu.cuCtxSynchronize())
        ok(cu.cuMemcpyDtoH_v2(ctypes.c_void_p(C.ctypes.data), ctypes.c_uint64(c), ctypes.c_size_t(C.nbytes)))
    finally:
        ok(cu.cuCtxDestroy_v2(ctx))
    np.testing.assert_allclose(C, want, rtol=1e-5, atol=1e-4)
    # and the first context still works
    np.testing.assert_allclose(hyb.spmm_csr(d, torch.from_numpy(B).to(cuda_device)).cpu().numpy(), want, rtol=1e-5, atol=1e-4)

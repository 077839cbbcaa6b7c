"""The C view that a ``HybFormat`` keeps says at every time what a fresh one says, and refuses what it refuses."""
import numpy as np
import pytest
import torch

from liteform_ae_b200 import hyb
from liteform_ae_b200._cabi import LfHyb


def _format():
    rows, cols = [[np.array([0, 2]), np.array([2])]], [[np.array([[1], [3]]), np.array([[0, 2]])]]
    vals = [[np.ones((2, 1)), np.ones((1, 2))]]
    ell, row_off, slot_off, r, c, v, z = hyb.HybFormat.host_layout([[1, 2]], rows, cols, vals, 4)
    up = torch.from_numpy
    return hyb.HybFormat((4, 4), (0, 4), [[1, 2]], ell, row_off, slot_off, up(r), up(c), up(v), None, up(z))


def _same(fmt):
    kept, fresh = fmt._c_ref()._obj, fmt.c_struct()
    return all(getattr(kept, name) == getattr(fresh, name) for name, _ in LfHyb._fields_)


def test_kept_between_calls():
    fmt = _format()
    assert fmt._c_ref() is fmt._c_ref() and _same(fmt)


def test_rows_to_clear_shrunk_in_place():
    fmt = _format()
    assert fmt._c_ref()._obj.num_zero_rows == 3
    fmt.zero_rows.resize_(1)
    assert fmt.zero_rows.data_ptr() == fmt._c_ref()._obj.zero_rows and _same(fmt)


@pytest.mark.parametrize("name", ["row_off", "widths", "ell_rows", "mask", "zero_rows"])
def test_deleted_attribute_is_missed(name):
    fmt = _format()
    fmt._c_ref()
    delattr(fmt, name)
    with pytest.raises(AttributeError):
        fmt._c_ref()


def test_strides_changed_in_place_are_refused():
    fmt = _format()
    fmt._c_ref()
    fmt.vals.as_strided_((8, 8), (1, 8))
    with pytest.raises(AssertionError):
        fmt._c_ref()


def test_mask_and_missing_arrays():
    fmt = _format()
    fmt.mask = torch.ones(128, dtype=torch.uint8)
    assert _same(fmt)
    fmt.zero_rows = None
    assert _same(fmt)
    fmt.rows = fmt.cols = fmt.vals = None      # a format without ELL rows
    assert _same(fmt) and fmt._c_ref()._obj.vals is None

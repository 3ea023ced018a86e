"""gbds_op_autotune on the FP64 operator, which has one launch shape: fields
that the operator would refuse are refused (no device work)."""
import ctypes

import pytest


@pytest.mark.parametrize("nd", [4, 3])
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("fields", [(0, 4096, 8192), (4096, 0, 8192), (4096, 8192, 0), (4096, 8192, 12296), (4104, 8192, 12288),
                                     (4096, 8200, 12288)])
def test_fp64_autotune_refuses_bad_fields(fields, recon, nd):
    from sse_wilson_dslash_gb300 import _lib
    L = _lib.core()
    h = ctypes.c_void_p()
    assert L.gbds_op_create_ex(ctypes.byref(h), (ctypes.c_int * 4)(4, 4, 4, 4), nd, 64, recon, 1, 0) == 0
    try:
        want = L.gbds_op_dslash(h, *fields, 1, 0, None)
        assert want != 0
        assert L.gbds_op_autotune(h, *fields, None) == want
    finally:
        L.gbds_op_destroy(h)

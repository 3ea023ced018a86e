"""The default multi-RHS kernel by lattice size, count and storage (no device
work): the plain kernel (variant 0) wherever the fields make few blocks."""
import ctypes

import pytest


def default_variant(dims, nrhs, fmt, recon=18):
    from sse_wilson_dslash_gb300 import _lib
    L = _lib.core()
    h, blk, var = ctypes.c_void_p(), ctypes.c_int(), ctypes.c_int()
    assert L.gbds_op_create_ex(ctypes.byref(h), (ctypes.c_int * 4)(*dims), 4, 32, recon, nrhs, fmt) == 0
    assert L.gbds_op_get_tuning(h, ctypes.byref(blk), ctypes.byref(var)) == 0
    L.gbds_op_destroy(h)
    return var.value


FP32, BF16, HALF, PAIRS = 0, 1, 2, 3


@pytest.mark.parametrize("fmt", [BF16, HALF])
@pytest.mark.parametrize("nrhs", [3, 4, 5, 6, 7, 9, 10, 11])
def test_16_bit_storage_on_small_lattices_takes_the_plain_kernel(nrhs, fmt):
    for dims in ((4, 4, 4, 4), (6, 6, 6, 12), (10, 10, 12, 16)):
        assert default_variant(dims, nrhs, fmt) == 0
    if nrhs < 8:
        assert default_variant((12, 12, 16, 24), nrhs, fmt) == 0


@pytest.mark.parametrize("fmt,nrhs,recon,small,large,variant", [
    (HALF, 4, 18, (16, 16, 16, 32), (16, 16, 20, 32), 2),
    (HALF, 5, 18, (16, 16, 16, 32), (16, 16, 20, 32), 2),
    (HALF, 7, 18, (16, 16, 16, 24), (16, 16, 16, 32), 2),
    (HALF, 5, 12, (20, 20, 20, 24), (20, 20, 24, 24), 2),
    (HALF, 6, 18, (16, 16, 16, 16), (16, 16, 16, 24), 3),
    (BF16, 6, 18, (12, 12, 16, 24), (16, 16, 16, 24), 3),
    (BF16, 10, 18, (10, 10, 12, 16), (12, 12, 16, 16), 3),
    (BF16, 12, 18, (10, 10, 12, 16), (8, 8, 8, 32), 3),
    (HALF, 11, 18, (16, 16, 16, 16), (16, 16, 16, 24), 2),
    (BF16, 9, 18, (16, 16, 16, 16), (16, 16, 16, 24), 2),
    (FP32, 12, 18, (12, 12, 16, 24), (16, 16, 16, 32), 2),
    (PAIRS, 12, 12, (12, 12, 16, 24), (16, 16, 16, 32), 2),
])
def test_lines_between_the_kernels(fmt, nrhs, recon, small, large, variant):
    assert default_variant(small, nrhs, fmt, recon) == 0
    assert default_variant(large, nrhs, fmt, recon) == variant
    assert default_variant((24, 24, 24, 48), nrhs, fmt, recon) == variant


@pytest.mark.parametrize("nrhs", [18, 24, 30])
def test_two_rhs_a_thread_at_every_size_from_18(nrhs):
    for dims in ((4, 4, 4, 4), (10, 10, 12, 16), (24, 24, 24, 48)):
        assert default_variant(dims, nrhs, BF16) == default_variant(dims, nrhs, HALF, 12) == 3


def test_counts_without_a_line():
    for dims in ((4, 4, 4, 4), (24, 24, 24, 48)):
        for nrhs, want in ((8, (0, 0, 2, 0)), (16, (3, 4, 4, 3)), (32, (3, 4, 4, 3))):
            assert tuple(default_variant(dims, nrhs, f) for f in (FP32, BF16, HALF, PAIRS)) == want

"""Creating a solver leaves the caller's streams alone: inside a relaxed capture
of a stream that synchronises with the default stream the capture stays valid
and empty, and the solver made there solves."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

KAPPA, DIMS = 0.124, (4, 4, 4, 8)


def _runtime():
    for name in ("libcudart.so.13", "libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            continue
    pytest.skip("no shared CUDA runtime")


@pytest.mark.parametrize("make", ["single32", "single16", "batched"])
def test_create_inside_a_capture(make):
    import torch
    from sse_wilson_dslash_gb300.device import BatchedWilsonSolver, WilsonSolver
    torch.zeros(1, device="cuda")
    rt = _runtime()
    stream, graph, n = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_size_t(99)
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
    try:
        if make == "batched":
            s = BatchedWilsonSolver(DIMS, 4, KAPPA, tol=1e-10)
        else:
            s = WilsonSolver(DIMS, KAPPA, tol=1e-10, inner_prec=int(make[6:]))
    finally:
        ended = rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    assert ended == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0 and n.value == 0
    rt.cudaGraphDestroy(graph)
    rt.cudaStreamDestroy(stream)
    u, b = O.make_inputs(DIMS, 11, 12, kind="near_unit")
    s.set_gauge(torch.from_numpy(u.ravel()).cuda())
    bs = torch.from_numpy(np.tile(b.ravel(), 4 if make == "batched" else 1)).cuda()
    x = torch.zeros_like(bs)
    st = s.solve(bs, x)
    assert all(t["converged"] == 1 for t in (st if make == "batched" else [st]))
    s.close()

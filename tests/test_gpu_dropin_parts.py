"""The reference's call on pinned host arrays, where it goes through the lattice
in parts (results of one part while the links of the next come in): the same
bits as the operator on resident fields, and nothing else written."""
import pytest

from sse_wilson_dslash_gb300 import _lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (dims, nd): two and three parts of uneven slices (parts^2 x 8 MB of links), one
# slice a part, and lattices that go in one
SHAPES = [((16, 16, 16, 32), 4), ((12, 16, 20, 33), 3), ((32, 32, 36, 4), 4), ((48, 48, 48, 2), 4), ((4, 6, 4, 8), 4)]


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("dims,nd", SHAPES)
def test_parts_match_operator(dims, nd, prec):
    from sse_wilson_dslash_gb300.device import DslashOperator
    from sse_wilson_dslash_gb300.legacy import SSEDslash
    V = dims[0] * dims[1] * dims[2] * dims[3]
    dt = torch.float32 if prec == 32 else torch.float64
    gen = torch.Generator().manual_seed(V + prec)
    u = torch.randn(V * 72, dtype=dt, generator=gen).pin_memory()
    psi = torch.randn(V * 24, dtype=dt, generator=gen).pin_memory()
    op = DslashOperator(dims, nd=nd, prec=prec)
    gauge = op.pack_gauge(u.cuda())
    api, suffix = SSEDslash(prec), "_3d" if nd == 3 else ""
    getattr(api, "init_sse_su3dslash" + suffix)(dims, *_lib.canonical_callbacks(nd, dims))
    try:
        for isign, cb in ((1, 0), (-1, 1), (1, 0)):
            res = torch.full((V * 24,), 7.0, dtype=dt).pin_memory()
            getattr(api, "sse_su3dslash_wilson" + suffix)(u, psi, res, isign, cb)
            want = torch.full((V * 24,), 7.0, dtype=dt, device="cuda")
            op.unpack_spinor(op.apply(gauge, op.pack_spinor(psi.cuda(), cb), isign, cb), 1 - cb, want)
            assert torch.equal(res, want.cpu())
    finally:
        getattr(api, "free_sse_su3dslash" + suffix)()

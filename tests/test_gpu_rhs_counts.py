"""The fully packed multi-RHS kernels at counts of right-hand sides that do not
divide a CTA: one rhs a thread (variant 2, any count), two adjacent rhs a
thread with 256-bit loads (variant 3, 16-bit storage, even counts) and the
default choice, every rhs and target site against the oracle.  The lattice's
120 sites a checkerboard leave the last CTA partly idle, and counts such as 3,
7, 12 and 24 leave threads of every CTA idle.  Bounds: tests/formats.py."""
import numpy as np
import pytest

import oracle as O
from formats import TOL, site_err, stored

pytestmark = pytest.mark.gpu

DIMS = (6, 2, 2, 10)


@pytest.mark.parametrize("fmt", ["native", "f32_pairs", "bf16", "f16"])
@pytest.mark.parametrize("nrhs", [2, 3, 4, 5, 6, 7, 8, 10, 12, 24, 31])
def test_counts_match_oracle(nrhs, fmt):
    import torch
    from sse_wilson_dslash_gb300.device import DslashOperator
    V, lol = O.volume(DIMS), O.layout_table(O.LAYOUT_CB2, DIMS)
    rng = np.random.default_rng(900 + nrhs)
    u = O.random_gauge(rng, V).astype(np.float32)
    psi = np.stack([O.gaussian_spinor(rng, V) for _ in range(nrhs)]).astype(np.float32).reshape(nrhs, V, 24)
    src = stored(psi, fmt)
    packed = torch.from_numpy(psi.ravel()).cuda()
    for recon, isign, cb in ((18, 1, 0), (12, -1, 1)):
        ts = O.target_sites(4, DIMS, lol, cb)
        ref = np.stack([np.asarray(O.dslash_plain(4, DIMS, lol, u, src[r].reshape(V, 4, 3, 2), isign, cb)).reshape(V, 24)
                        for r in range(nrhs)])
        for variant in (None, 2, 3):
            op = DslashOperator(DIMS, recon=recon, nrhs=nrhs, spinor_format=fmt)
            if variant is not None:
                op.set_tuning(0, variant)
            gauge = op.pack_gauge(torch.from_numpy(u.ravel()).cuda())
            # fields at a 16-byte boundary that is no 32-byte one, and at one that is
            for shift in (0, 16):
                a = torch.zeros(op.spinor_bytes + 16, dtype=torch.uint8, device="cuda")
                b = torch.zeros_like(a)
                field = op.pack_spinor(packed, cb, out=a[shift:shift + op.spinor_bytes])
                out = op.apply(gauge, field, isign, cb, out=b[shift:shift + op.spinor_bytes])
                res = torch.zeros(nrhs * V * 24, dtype=torch.float32, device="cuda")
                op.unpack_spinor(out, 1 - cb, res)
                assert site_err(res.cpu().numpy().reshape(nrhs, V, 24), ref, ts) <= TOL[fmt], (recon, variant, shift)
            op.close()

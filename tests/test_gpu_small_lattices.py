"""The FP32 single-rhs kernels that differ by lattice size (csrc/dslash_f32.cu):
four warps a site, and every register cap, against the oracle at the FP32
per-site tolerance, at sizes that leave the last CTA partly idle (fewer sites
than one CTA; 120 and 129 sites), 4D and 3D, 18- and 12-real links; the default
choice on both sides of its first two lines (228 and 512 CTAs of 128 sites)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _errors(nd, dims, recon, tunings, combos):
    import torch
    from sse_wilson_dslash_gb300.device import DslashOperator
    lol = O.layout_table(O.LAYOUT_CB2 if nd == 4 else O.LAYOUT_CB3D, dims)
    u, psi = (a.astype(np.float32) for a in O.make_inputs(dims, 61, 62))
    op = DslashOperator(dims, nd=nd, prec=32, recon=recon)
    gauge = op.pack_gauge(torch.from_numpy(u.ravel()).cuda())
    pd = torch.from_numpy(psi.ravel()).cuda()
    for isign, cb in combos:
        ref = O.dslash_plain(nd, dims, lol, u, psi, isign, cb)
        ts = O.target_sites(nd, dims, lol, cb)
        src = op.pack_spinor(pd, cb)
        for tuning in tunings(op):
            if tuning is not None:
                op.set_tuning(*tuning)
            res = torch.zeros(op.volume * 24, dtype=torch.float32, device="cuda")
            op.unpack_spinor(op.apply(gauge, src, isign, cb), 1 - cb, res)
            yield tuning, isign, cb, O.site_rel_err(res.cpu().numpy(), ref, ts)
    op.close()


@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("nd,dims", [(4, (2, 2, 2, 2)), (4, (6, 2, 2, 10)), (4, (4, 6, 8, 4)), (3, (2, 2, 2, 1)),
                                      (3, (4, 6, 4, 5)), (3, (2, 6, 2, 43))])
def test_every_variant_matches_oracle(nd, dims, recon):
    def tunings(op):
        return [None, (32, 0), (256, 0)] + [(0, v) for v in range(op.num_variants)]
    for what in _errors(nd, dims, recon, tunings, ((1, 0), (1, 1), (-1, 0), (-1, 1))):
        assert what[-1] <= TOL, what


@pytest.mark.parametrize("dims", [(12, 12, 12, 32), (16, 16, 16, 16), (16, 16, 16, 32), (16, 16, 16, 36)])
def test_default_choice_matches_oracle(dims):
    for recon in (18, 12):
        for what in _errors(4, dims, recon, lambda op: [None], ((1, 0),)):
            assert what[-1] <= TOL, (recon, what)

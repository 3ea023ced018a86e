"""The solvers on lattices that leave the last CTA of their launches partly idle,
on those whose FP32 operator launches use uncapped registers (with and without
their own sums), and for iteration counts that mix recorded and single steps;
against the oracle's Dslash and a conjugate gradient in FP64 numpy on it."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

KAPPA = 0.124


class System:
    """M = 1 - kappa^2 D_eo D_oe on the even sites of a smooth random field."""

    def __init__(self, dims, nrhs=1):
        self.dims, self.lol = dims, O.layout_table(O.LAYOUT_CB2, dims)
        self.u, _ = O.make_inputs(dims, 91, 92, kind="near_unit")
        rng = np.random.default_rng(93)
        self.b = [O.gaussian_spinor(rng, O.volume(dims)) for _ in range(nrhs)]
        self.even = O.target_sites(4, dims, self.lol, 1)

    def M(self, x, sign):
        t = O.dslash_plain(4, self.dims, self.lol, self.u, x, sign, 0)
        y = O.dslash_plain(4, self.dims, self.lol, self.u, t, sign, 1)
        out = np.zeros_like(x)
        out[self.even] = x[self.even] - KAPPA * KAPPA * y[self.even]
        return out

    def residual(self, x, q=0):
        r = self.M(x, 1)[self.even] - self.b[q][self.even]
        return np.linalg.norm(r) / np.linalg.norm(self.b[q][self.even])

    def cg(self, iterations, q=0):
        """x after so many iterations on M^+ M x = M^+ b from x = 0."""
        b = np.zeros_like(self.b[q])
        b[self.even] = self.b[q][self.even]
        r = self.M(b, -1)
        x, p, rr = np.zeros_like(r), r.copy(), (r ** 2).sum()
        for _ in range(iterations):
            Mp = self.M(p, 1)
            alpha = rr / (Mp ** 2).sum()
            r = r - alpha * self.M(Mp, -1)
            x = x + alpha * p
            new = (r ** 2).sum()
            p, rr = r + new / rr * p, new
        return x


def _single(sys, prec, recon, max_iter=2000, tol=1e-10):
    import torch
    from sse_wilson_dslash_gb300.device import WilsonSolver
    s = WilsonSolver(sys.dims, KAPPA, tol=tol, max_iter=max_iter, inner_prec=prec, inner_recon=recon,
                     inner_tol=1e-5 if prec >= 32 else 1e-3)
    s.set_gauge(torch.from_numpy(sys.u.ravel()).cuda())
    x = torch.zeros(sys.u.size // 3, dtype=torch.float64, device="cuda")
    st = s.solve(torch.from_numpy(sys.b[0].ravel()).cuda(), x)
    s.close()
    return st, x.cpu().numpy().reshape(sys.b[0].shape)


def _batched(sys, nrhs, recon, max_iter=2000):
    import torch
    from sse_wilson_dslash_gb300.device import BatchedWilsonSolver
    s = BatchedWilsonSolver(sys.dims, nrhs, KAPPA, tol=1e-10, max_iter=max_iter, inner_recon=recon)
    s.set_gauge(torch.from_numpy(sys.u.ravel()).cuda())
    b = torch.from_numpy(np.stack(sys.b).ravel()).cuda()
    x = torch.zeros_like(b)
    st = s.solve(b, x)
    s.close()
    return st, x.cpu().numpy().reshape((nrhs,) + sys.b[0].shape)


# sites a checkerboard: 120 (less than a CTA), 1080, 37240 (290.9 CTAs of 128:
# uncapped registers and sums in the launch), 32768 (256 CTAs, the same)
SMALL = [(6, 2, 2, 10), (6, 6, 6, 10), (10, 14, 14, 38), (16, 16, 16, 16)]


@pytest.mark.parametrize("prec,recon", [(64, 18), (32, 18), (32, 12), (16, 12), (16, 18), (17, 12)])
@pytest.mark.parametrize("dims", SMALL)
def test_solve_on_uneven_lattices(dims, prec, recon):
    sys = System(dims)
    st, x = _single(sys, prec, recon)
    assert st["converged"] == 1 and st["residual"] <= 1e-10, st
    res = sys.residual(x)
    # the normal equations' residual is at most 1e-10 of |M^+ b|; |M^-1| < 100 here
    assert res < 1e-8 and abs(res - st["true_residual"]) <= 1e-3 * res + 1e-14


@pytest.mark.parametrize("recon", [12, 18])
def test_solve_with_uncapped_registers_and_separate_sums(recon):
    """18^3x50: 1139.1 CTAs, where the 12-real launches are uncapped again."""
    sys = System((18, 18, 18, 50))
    st, x = _single(sys, 32, recon)
    assert st["converged"] == 1 and sys.residual(x) < 1e-8


@pytest.mark.parametrize("nrhs,recon", [(2, 12), (4, 18), (8, 12), (16, 18), (32, 12)])
@pytest.mark.parametrize("dims", SMALL[:2])
def test_batched_solve_on_uneven_lattices(dims, nrhs, recon):
    sys = System(dims, nrhs)
    st, x = _batched(sys, nrhs, recon)
    for q in range(nrhs):
        assert st[q]["converged"] == 1 and sys.residual(x[q], q) < 1e-8, q


# FP32 rounds each of an iteration's fields by 6e-8; CG carries such errors on
# with factors of the order of the operator's condition number (< 100 here)
CG_TOL = {64: 1e-11, 32: 1e-4}


@pytest.mark.parametrize("max_iter", [1, 3, 4, 5, 7, 8, 11])
@pytest.mark.parametrize("dims", [(6, 6, 6, 10), (16, 16, 16, 16)])
def test_iterations_before_and_after_the_recorded_ones(dims, max_iter):
    """Stopped after 1, 3 (no group of four), 4, 8 (whole groups) or 5, 7, 11
    iterations (groups, then single steps): the iterate is CG's."""
    sys = System(dims)
    want = sys.cg(max_iter)[sys.even]
    for prec, recon in ((64, 18), (32, 18), (32, 12)):
        st, x = _single(sys, prec, recon, max_iter, tol=1e-14)
        assert st["iterations"] == max_iter and st["converged"] == 0
        assert np.linalg.norm(x[sys.even] - want) <= CG_TOL[prec] * np.linalg.norm(want), (prec, recon)


@pytest.mark.parametrize("max_iter", [3, 4, 6])
@pytest.mark.parametrize("nrhs", [2, 8, 16])
def test_batched_iterations_before_and_after_the_recorded_ones(nrhs, max_iter):
    sys = System((6, 6, 6, 10), nrhs)
    st, x = _batched(sys, nrhs, 18, max_iter)
    for q in (0, nrhs - 1):
        want = sys.cg(max_iter, q)[sys.even]
        assert st[q]["iterations"] == max_iter and st[q]["converged"] == 0
        assert np.linalg.norm(x[q][sys.even] - want) <= CG_TOL[32] * np.linalg.norm(want), q

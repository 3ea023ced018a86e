"""Accuracy of the FP64 Dslash component by component: every real of a result
against the sum of its own terms' moduli, not against its site's norm.

The fixed-point sums (csrc/fixpoint.cuh) share a scale among the outputs of a
colour; an output whose own terms are small against it is left to FP64
arithmetic.  On the CPU: that rule, on the sums as the kernel forms them,
against exact rational arithmetic.  On the GPU: the operator with spins, colours,
real and imaginary parts of spinors and links at scales of their own, and with
some of them exactly zero, against extended precision."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import oracle as O

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
EPS = 2.0 ** -53

# FP64 arithmetic: one projection, six multiply-adds and eight sums round a
# component, each by at most 2^-53 of a partial sum, which the terms' moduli bound
COMP_TOL = 15 * EPS
# those roundings at random, uniform within +-2^-53 of partial sums no larger
# than the result typically is: rms over a field
RMS_TOL = (15 / 3) ** 0.5 * EPS
# 12-real links: the third row's products round three times more
COMP_TOL_12 = 18 * EPS
TINY = 64 * 2.0 ** -1074  # results below FP64's normal range


# ---------------------------------------------------------------------------
# The rule on the CPU
# ---------------------------------------------------------------------------

@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    """One output of eight hops as the kernel sums it: in, per hop and colour,
    (ur, ui, hr, hi) and the exponent of the spinor's scale; out, the two sums,
    whether each is resolved, and the exponent of their unit."""
    d = tmp_path_factory.mktemp("sums")
    src = d / "sums.cc"
    src.write_text(r'''
#include "fixpoint.cuh"
#include <cstring>
using namespace gbds;
static uint32_t hw(double v) { uint64_t b; memcpy(&b, &v, 8); return (uint32_t)(b >> 32); }
static uint32_t lw(double v) { uint64_t b; memcpy(&b, &v, 8); return (uint32_t)b; }
static fix2 fx(double v, uint32_t t) { return fix_convert(hw(v), lw(v), t); }
extern "C" int sums(const double *v, const unsigned *eh, const int *dag, long long *acc_out, int *resolved) {
    int64_t acc[2] = {0, 0};
    uint32_t seen[2] = {0, 0}, e = 0;
    for (int hop = 0; hop < 8; hop++) {
        const double *q = v + hop * 12;
        const unsigned *sc = eh + hop * 3;
        uint32_t et = 0;
        for (int j = 0; j < 3; j++)
            for (int p = 0; p < 2; p++) {
                const uint32_t x = fix_exponent(hw(q[4 * j + p])) + sc[j];
                if (x > et) et = x;
            }
        if (et > e) {
            for (int p = 0; p < 2; p++) {
                acc[p] = fix_sar(acc[p], et - e);
                seen[p] = fix_shr(seen[p], et - e);
            }
            e = et;
        }
        int64_t W[2] = {0, 0}, X[2] = {kFixHalf, kFixHalf};
        for (int j = 0; j < 3; j++) {
            const uint32_t t0 = e - sc[j] + 3;
            const fix2 ur = fx(q[4 * j], t0 - fix_exponent(hw(q[4 * j]))), ui = fx(q[4 * j + 1], t0 - fix_exponent(hw(q[4 * j + 1])));
            const fix2 hr = fx(q[4 * j + 2], sc[j] + 3 - fix_exponent(hw(q[4 * j + 2])));
            const fix2 hi = fx(q[4 * j + 3], sc[j] + 3 - fix_exponent(hw(q[4 * j + 3])));
            if (dag[hop]) fix_cmad<true>(W, X, ur, ui, hr, hi);
            else fix_cmad<false>(W, X, ur, ui, hr, hi);
        }
        for (int p = 0; p < 2; p++) {
            W[p] += X[p] >> 32;
            acc[p] += W[p];
            seen[p] += fix_modulus_hi(W[p]);
        }
    }
    for (int p = 0; p < 2; p++) { acc_out[p] = acc[p]; resolved[p] = fix_resolved(seen[p]); }
    return (int)e - 2 * 1023 - kFixUnit;
}
''')
    so = d / "sums.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "sse_wilson_dslash_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    L = ctypes.CDLL(str(so))

    def run(v, eh, dag):
        v, eh = np.ascontiguousarray(v, dtype=np.float64), np.ascontiguousarray(eh, dtype=np.uint32)
        dag = np.ascontiguousarray(dag, dtype=np.int32)
        acc, res = (ctypes.c_longlong * 2)(), (ctypes.c_int * 2)()
        unit = L.sums(v.ctypes.data_as(ctypes.c_void_p), eh.ctypes.data_as(ctypes.c_void_p),
                      dag.ctypes.data_as(ctypes.c_void_p), acc, res)
        return [int(a) for a in acc], [bool(r) for r in res], unit

    return run


def _exact(v, dag):
    s, t = [Fraction(0)] * 2, [Fraction(0)] * 2
    for hop in range(8):
        for j in range(3):
            ur, ui, hr, hi = (Fraction(float(x)) for x in v[hop, j])
            ui = -ui if dag[hop] else ui
            for p, (x, y) in enumerate([(ur * hr, -ui * hi), (ur * hi, ui * hr)]):
                s[p] += x + y
                t[p] += abs(x) + abs(y)
    return s, t


@pytest.mark.parametrize("shift", [0, 3, 6, 10, 20, 40, 56, 200])
def test_resolved_sums_keep_fp64_accuracy(sums, shift):
    """Sums whose operands lie 2^shift below the scale (another spin's), or
    whose imaginary parts do: one that counts as resolved is within the bound of
    FP64 arithmetic of its own terms; at the scale itself nearly all are."""
    rng = np.random.default_rng(shift)
    own = counted = 0
    for k in range(400):
        v = rng.standard_normal((8, 3, 4))
        v[..., :2] /= np.sqrt((v[..., :2] ** 2).sum(axis=(1, 2), keepdims=True))  # rows of unitary links
        if k % 2:
            v[..., 2:] *= 2.0 ** -shift
        else:
            v[..., [1, 3]] *= 2.0 ** -shift
        dag = np.arange(8) % 2
        # the scale: the largest of four reals, two of them another spin's
        other = rng.standard_normal((8, 3, 2))
        eh = np.frexp(np.maximum(np.abs(other).max(-1), np.abs(v[..., 2:]).max(-1)))[1] - 1 + 1023
        acc, res, unit = sums(v, eh, dag)
        s, t = _exact(v, dag)
        for p in range(2):
            if res[p]:
                counted += 1
                assert abs(Fraction(acc[p]) * Fraction(2) ** unit - s[p]) <= Fraction(COMP_TOL) * t[p], (k, p)
        own += sum(res) if shift == 0 else 0
    if shift == 0:
        assert own == 800  # one thread (eight outputs) in 4 million is left to FP64
    if shift >= 40:
        assert counted <= 400  # the imaginary parts' and the small spins' are not


def test_exact_zeros_add_up_to_zero(sums):
    """Every product with a factor +-0: the sum is 0 but for the shifts of -1, and
    does not count as resolved."""
    rng = np.random.default_rng(5)
    for k in range(200):
        v = rng.standard_normal((8, 3, 4))
        z = 0.0 if k % 2 else -0.0
        if k % 3 == 0:
            v[..., 2:] = z                 # a spin of zeros beside others
        elif k % 3 == 1:
            v[..., [1, 3]] = z             # real operands: the imaginary sum
        else:
            v[..., [0, 3]] = z             # ... the real one
        acc, res, _ = sums(v, rng.integers(1024, 1027, (8, 3)), np.arange(8) % 2)
        for p, zero in enumerate([k % 3 in (0, 2), k % 3 in (0, 1)]):
            if zero:
                assert abs(acc[p]) <= 8 and not res[p]


# ---------------------------------------------------------------------------
# The operator
# ---------------------------------------------------------------------------

def _reference(nd, dims, lol, u, psi, isign, cb, recon):
    """(result, sum of its terms' moduli), [V][4][3][2] in extended precision."""
    R = np.longdouble
    V = O.volume(dims)
    Lx, Ly, Lz, Lt = dims
    axis = {0: 3, 1: 2, 2: 1, 3: 0}
    grid = (Lt, Lz, Ly, Lx)
    p = psi.reshape(V, 4, 3, 2)[lol].astype(R).reshape(grid + (4, 3, 2))
    m = np.swapaxes(u.reshape(V, 4, 3, 3, 2)[lol].astype(R), 2, 3)  # [V][mu][i][j][2], U_ij
    mm = np.abs(m)

    def mul(x, y):
        return np.stack([x[..., 0] * y[..., 0] - x[..., 1] * y[..., 1], x[..., 0] * y[..., 1] + x[..., 1] * y[..., 0]], -1)

    def mulabs(x, y):
        return np.stack([x[..., 0] * y[..., 0] + x[..., 1] * y[..., 1], x[..., 0] * y[..., 1] + x[..., 1] * y[..., 0]], -1)

    if recon == 12:
        m, mm = m.copy(), mm.copy()
        for j in range(3):
            k, l = (j + 1) % 3, (j + 2) % 3
            m[:, :, 2, j] = mul(m[:, :, 0, k], m[:, :, 1, l]) - mul(m[:, :, 0, l], m[:, :, 1, k])
            m[:, :, 2, j, 1] *= -1
            mm[:, :, 2, j] = mulabs(mm[:, :, 0, k], mm[:, :, 1, l]) + mulabs(mm[:, :, 0, l], mm[:, :, 1, k])
    m, mm = m.reshape(grid + (4, 3, 3, 2)), mm.reshape(grid + (4, 3, 3, 2))
    gam = O.gamma_matrices()
    res, mod = np.zeros_like(p), np.zeros_like(p)

    def times(code, x):  # one of 0, +-1, +-i
        re, im = R(code.real), R(code.imag)
        return np.stack([re * x[..., 0] - im * x[..., 1], re * x[..., 1] + im * x[..., 0]], -1)

    def hop(mat, matabs, src, sg, mu):
        # half spinors h_k = psi_k + (partner), w = mat h, lower spins from w
        n = -sg * gam[mu]
        out, outabs = np.zeros_like(src), np.zeros_like(src)
        w, wabs = [], []
        for k in range(2):
            h = src[..., k, :, :].copy()
            for t in (2, 3):
                h = h + times(n[k, t], src[..., t, :, :])
            w.append(sum(mul(mat[..., :, j, :], h[..., None, j, :]) for j in range(3)))
            wabs.append(sum(mulabs(matabs[..., :, j, :], np.abs(h[..., None, j, :])) for j in range(3)))
            out[..., k, :, :], outabs[..., k, :, :] = w[k], wabs[k]
        for t in (2, 3):
            for k in range(2):
                if n[t, k] != 0:
                    out[..., t, :, :] = times(n[t, k], w[k])
                    outabs[..., t, :, :] = np.abs(times(n[t, k], wabs[k]))
        return out, outabs

    for mu in range(nd):
        M, A = m[..., mu, :, :, :], mm[..., mu, :, :, :]
        o, oa = hop(M, A, np.roll(p, -1, axis=axis[mu]), isign, mu)
        res, mod = res + o, mod + oa
        D, DA = np.swapaxes(M, -3, -2).copy(), np.swapaxes(A, -3, -2)
        D[..., 1] *= -1
        o, oa = hop(D, DA, p, -isign, mu)
        res, mod = res + np.roll(o, 1, axis=axis[mu]), mod + np.roll(oa, 1, axis=axis[mu])
    sel = (O.parity_of_lex(dims, nd) == 1 - cb).ravel()
    return res.reshape(V, 4, 3, 2)[sel], mod.reshape(V, 4, 3, 2)[sel], lol[sel]


def _apply(nd, dims, recon, u, psi, isign, cb):
    import torch
    from sse_wilson_dslash_gb300.device import DslashOperator
    op = DslashOperator(dims, nd=nd, prec=64, recon=recon)
    gauge = op.pack_gauge(torch.from_numpy(np.ascontiguousarray(u)).cuda())
    src = op.pack_spinor(torch.from_numpy(np.ascontiguousarray(psi)).cuda(), cb)
    res = torch.zeros(op.volume * 24, dtype=torch.float64, device="cuda")
    op.unpack_spinor(op.apply(gauge, src, isign, cb), 1 - cb, res)
    out = res.cpu().numpy().reshape(psi.shape)
    op.close()
    return out


def test_reference_is_the_oracle():
    for nd, dims in ((4, (4, 2, 6, 4)), (3, (4, 2, 4, 3))):
        lol = O.layout_table(O.LAYOUT_CB2 if nd == 4 else O.LAYOUT_CB3D, dims)
        u, psi = O.make_inputs(dims, 3, 4)
        for isign, cb, recon in ((1, 0, 18), (-1, 1, 12)):
            ref, mod, sites = _reference(nd, dims, lol, u, psi, isign, cb, recon)
            want = O.dslash_plain(nd, dims, lol, u, psi, isign, cb)[sites]
            assert np.all(np.abs(want - ref) <= 64 * EPS * mod)


def _check(nd, dims, recon, u, psi, combos=((1, 0), (-1, 1)), rms=True):
    lol = O.layout_table(O.LAYOUT_CB2 if nd == 4 else O.LAYOUT_CB3D, dims)
    tol = COMP_TOL if recon == 18 else COMP_TOL_12
    for isign, cb in combos:
        ref, mod, sites = _reference(nd, dims, lol, u, psi, isign, cb, recon)
        err = np.abs(_apply(nd, dims, recon, u, psi, isign, cb)[sites] - ref)
        assert np.all(err <= tol * mod + np.where(mod > 0, TINY, 0)), (isign, cb, float((err / np.maximum(mod, np.finfo(np.longdouble).tiny)).max()))
        if rms:  # each spin and colour, real and imaginary parts apart
            e, r = np.sqrt((err ** 2).mean(0)), np.sqrt((ref ** 2).mean(0))
            assert np.all(e <= RMS_TOL * r), (isign, cb, float((e / r).max()))


SIZES = [(4, (4, 6, 8, 4)), (4, (6, 2, 2, 10)), (3, (4, 6, 4, 5))]


@pytest.mark.gpu
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("nd,dims", SIZES)
def test_components_of_ordinary_fields(nd, dims, recon):
    u, psi = O.make_inputs(dims, 71, 72)
    _check(nd, dims, recon, u, psi, ((1, 0), (1, 1), (-1, 0), (-1, 1)), rms=recon == 18)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [2, 3, 4, 7, 10, 20, 40, 60, 300])
@pytest.mark.parametrize("large", [(0,), (1,), (2,), (3,), (0, 2), (0, 1)])
def test_spins_of_different_size(large, k):
    """All spins but `large` 2^k smaller."""
    nd, dims = SIZES[k % 3]
    u, psi = O.make_inputs(dims, 73, 74)
    f = np.full(4, 2.0 ** -k)
    f[list(large)] = 1
    _check(nd, dims, 18, u, psi * f[:, None, None])


@pytest.mark.gpu
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("most", [4, 12, 40, 100])
def test_every_component_at_a_scale_of_its_own(most, recon):
    """Each spin, colour and part of the spinors, and each entry and part of the
    links (of the first two rows with 12 reals), at a power of two of its own."""
    nd, dims = SIZES[most % 3]
    rng = np.random.default_rng(most + recon)
    for _ in range(4):
        u, psi = O.make_inputs(dims, 75, 76)
        psi = psi * np.exp2(-rng.integers(0, most + 1, (4, 3, 2)))
        u = u * np.exp2(-rng.integers(0, most // 2 + 1, (1, 4, 3, 3, 2)))
        _check(nd, dims, recon, u, psi, rms=False)


@pytest.mark.gpu
@pytest.mark.parametrize("tiny", [0.0, -0.0, 1e-310, 1e-290])
def test_zeros_and_subnormals_beside_ordinary_components(tiny):
    """Diluted sources (one spin, one colour, chiral halves, one part), cold and
    diagonal links: exact zeros stay exact, the smallest numbers survive."""
    dims, nd = (4, 6, 8, 4), 4
    u, psi = O.make_inputs(dims, 77, 78)
    unit = np.zeros_like(u)
    unit[..., np.arange(3), np.arange(3), 0] = 1
    keep = np.zeros((5, 4, 3, 2), dtype=bool)
    keep[0, 1], keep[1, :, 2], keep[2, :2], keep[3, ..., 0], keep[4, 2, 0] = True, True, True, True, True
    for mask in keep:
        p = np.where(mask, psi, tiny * (1 + np.abs(psi)))
        for links in (u, unit):
            _check(nd, dims, 18, links, p, rms=False)


@pytest.mark.gpu
def test_solver_operator_keeps_small_components():
    """M = 1 - kappa^2 D_eo D_oe on FP64 fields (the epilogue launches): a spin
    2^-40 of the others, judged on its own."""
    import torch
    from sse_wilson_dslash_gb300.device import WilsonSolver
    dims, kappa = (6, 2, 2, 10), 0.124
    lol = O.layout_table(O.LAYOUT_CB2, dims)
    u, psi = O.make_inputs(dims, 79, 80)
    # directions 0 and 1 switched off: D then maps spins 0, 2 and 1, 3 to themselves
    u[:, :2] = 0
    psi = psi * np.array([1, 2.0 ** -40, 1, 2.0 ** -40])[:, None, None]
    s = WilsonSolver(dims, kappa, inner_prec=64)
    s.set_gauge(torch.from_numpy(u.ravel()).cuda())
    y = torch.zeros(psi.size, dtype=torch.float64, device="cuda")
    s.apply(torch.from_numpy(np.ascontiguousarray(psi).ravel()).cuda(), y)
    s.close()
    t, _, odd = _reference(4, dims, lol, u, psi, 1, 0, 18)
    mid = np.zeros(psi.shape, dtype=np.longdouble)
    mid[odd] = t
    d, _, ev = _reference(4, dims, lol, u, mid, 1, 1, 18)
    want = psi[ev].astype(np.longdouble) - np.longdouble(kappa) ** 2 * d
    got = y.cpu().numpy().reshape(psi.shape)[ev]
    e = np.sqrt(((got - want) ** 2).mean((0, 2, 3)))
    r = np.sqrt((want ** 2).mean((0, 2, 3)))
    # two operators and the sum
    assert np.all(e <= 3 * RMS_TOL * r), e / r

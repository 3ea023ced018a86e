"""The fixed-point numbers of the FP64 Dslash (csrc/fixpoint.cuh).

On the CPU: the conversion against exact rational arithmetic.  On the GPU: the
FP64 operator, 18- and 12-real links, 4D and 3D, at lattices that leave the
last group of 32 sites partly idle, with operands spread over many powers of
two, and beyond the fixed-point range (where it falls back to FP64), against
the oracle."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import oracle as O

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

# 8 hops of one projection, six multiply-adds and one sum, each rounded once
# (2^-53), on terms whose moduli sum to at most four times the result's norm
SITE_TOL = 8 * 8 * 4 * 2.0 ** -53


@pytest.fixture(scope="module")
def convert(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixpoint")
    src = d / "fix.cc"
    src.write_text('#include "fixpoint.cuh"\n'
                   'extern "C" void conv(unsigned hi, unsigned lo, unsigned t, int *out) {\n'
                   "    gbds::fix2 f = gbds::fix_convert(hi, lo, t); out[0] = f.n; out[1] = f.g; }\n"
                   'extern "C" unsigned expo(unsigned hi) { return gbds::fix_exponent(hi); }\n')
    so = d / "fix.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "sse_wilson_dslash_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    L = ctypes.CDLL(str(so))
    out = (ctypes.c_int * 2)()

    def conv(v, e):
        """(n, g) of the double v against the biased scale exponent e."""
        b = int(np.float64(v).view(np.uint64))
        hi, lo = b >> 32, b & 0xFFFFFFFF
        L.conv(hi, lo, e + 3 - L.expo(hi), out)
        return out[0], out[1]

    return conv


def test_conversion_is_the_nearest_multiple(convert):
    rng = np.random.default_rng(11)
    for k in range(4000):
        v = float(rng.standard_normal() * 2.0 ** rng.integers(-40, 40))
        if k % 7 == 0:
            v = float(np.ldexp(np.sign(v) * (1 + (k % 3 - 1) * 2.0 ** -52), int(rng.integers(-30, 30))))
        own = np.frexp(abs(v))[1] - 1 + 1023
        for d in (0, 1, 2, 5, 27, 28, 29, 31, 32, 40, 58):
            n, g = convert(v, int(own) + d)
            assert abs(n) <= 1 << 28 and -(1 << 31) <= g < 1 << 31
            exact = Fraction(v) * Fraction(2) ** (27 - (int(own) + d - 1023) + 32)
            # one unit of the shifted-out end, and one of the one's complement
            assert abs(n * (1 << 32) + g - exact) <= 2, (v, d)


def test_conversion_of_what_lies_below_the_scale(convert):
    for e in (64, 1023, 1200):
        assert convert(0.0, e) == (0, 0)
        assert convert(-0.0, e) in ((0, 0), (0, -1))
    assert convert(2.0 ** -70, 1023) == (0, 0)
    assert convert(-2.0 ** -70, 1023) in ((0, 0), (0, -1))


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


def _layout(nd, dims):
    return O.layout_table(O.LAYOUT_CB2 if nd == 4 else O.LAYOUT_CB3D, dims)


@pytest.mark.gpu
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("nd,dims", [(4, (2, 2, 2, 2)), (4, (6, 2, 2, 10)), (4, (4, 6, 8, 4)), (3, (4, 6, 4, 5)), (3, (2, 2, 2, 1))])
def test_fp64_operator_matches_oracle(nd, dims, recon):
    lol = _layout(nd, dims)
    u, psi = O.make_inputs(dims, 41, 42)
    for isign in (1, -1):
        for cb in (0, 1):
            got = _apply(nd, dims, recon, u, psi, isign, cb)
            ref = O.dslash_plain(nd, dims, lol, u, psi, isign, cb)
            assert O.site_rel_err(got, ref, O.target_sites(nd, dims, lol, cb)) <= SITE_TOL, (isign, cb)


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0, 1, 20, 60, 300])
def test_operands_spread_over_powers_of_two(spread):
    """Sites, and links, scaled by random powers of two: the error stays within
    the rounding of each site's largest term."""
    dims, nd = (4, 4, 6, 4), 4
    lol, rng = _layout(nd, dims), np.random.default_rng(spread + 1)
    u, psi = O.make_inputs(dims, 43, 44)
    V = O.volume(dims)
    psi = psi * np.exp2(rng.integers(-spread, spread + 1, V))[:, None, None, None]
    u = u * np.exp2(rng.integers(-spread // 4, spread // 4 + 1, (V, 4)))[:, :, None, None, None]
    for isign, cb in ((1, 0), (-1, 1)):
        got = _apply(nd, dims, 18, u, psi, isign, cb)
        ref = O.dslash_plain(nd, dims, lol, u, psi, isign, cb)
        assert O.site_rel_err(got, ref, O.target_sites(nd, dims, lol, cb)) <= SITE_TOL, (isign, cb)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [600, -600, -900])
def test_outside_the_fixed_point_range(k):
    """Fields scaled by 2^k give the unscaled result scaled by 2^k: exactly
    where neither run leaves FP64's normal range, up to rounding otherwise."""
    dims, nd = (4, 4, 2, 6), 4
    lol = _layout(nd, dims)
    u, psi = O.make_inputs(dims, 45, 46)
    got = _apply(nd, dims, 18, u, np.ldexp(psi, k), 1, 0)
    ref = O.dslash_plain(nd, dims, lol, u, psi, 1, 0)
    assert O.site_rel_err(np.ldexp(got, -k), ref, O.target_sites(nd, dims, lol, 0)) <= SITE_TOL


@pytest.mark.gpu
def test_zeros_infinities_and_nan():
    dims, nd = (4, 4, 4, 4), 4
    lol, V = _layout(nd, dims), O.volume((4, 4, 4, 4))
    u, psi = O.make_inputs(dims, 47, 48)
    tgt = O.target_sites(nd, dims, lol, 0)
    # a zero source; a point source, with every other site exactly zero
    assert not _apply(nd, dims, 18, u, np.zeros_like(psi), 1, 0).any()
    point = np.zeros_like(psi)
    point[3] = psi[3]
    got, ref = _apply(nd, dims, 18, u, point, 1, 0), O.dslash_plain(nd, dims, lol, u, point, 1, 0)
    hit = np.abs(ref).reshape(V, -1).max(1) > 0
    assert hit.sum() == 8 and not got[~hit].any()
    assert O.site_rel_err(got, ref, np.nonzero(hit)[0]) <= SITE_TOL
    # links switched off in one direction (a Dirichlet boundary), unit links
    cut = u.copy()
    cut[:, 3] = 0
    assert O.site_rel_err(_apply(nd, dims, 18, cut, psi, 1, 0), O.dslash_plain(nd, dims, lol, cut, psi, 1, 0), tgt) <= SITE_TOL
    unit = np.zeros_like(u)
    unit[..., np.arange(3), np.arange(3), 0] = 1
    assert O.site_rel_err(_apply(nd, dims, 18, unit, psi, -1, 0), O.dslash_plain(nd, dims, lol, unit, psi, -1, 0), tgt) <= SITE_TOL
    # a non-finite source spinor or link reaches its neighbours and nobody else
    for bad in (np.inf, np.nan):
        p = psi.copy()
        p[3, 1, 2, 0] = bad
        got, ref = _apply(nd, dims, 18, u, p, 1, 0), O.dslash_plain(nd, dims, lol, u, p, 1, 0)
        fin = np.isfinite(ref).reshape(V, -1).all(1)
        assert (np.isfinite(got).reshape(V, -1).all(1) == fin).all() and (~fin).sum() == 8
        assert O.site_rel_err(got, ref, tgt[fin[tgt]]) <= SITE_TOL
        w = u.copy()
        w[tgt[5], 2, 0, 1, 1] = bad
        got, ref = _apply(nd, dims, 18, w, psi, 1, 0), O.dslash_plain(nd, dims, lol, w, psi, 1, 0)
        fin = np.isfinite(ref).reshape(V, -1).all(1)
        assert (np.isfinite(got).reshape(V, -1).all(1) == fin).all() and (~fin).sum() == 1

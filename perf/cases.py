"""The work that users of this library have it do, as measurable cases.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (fields on the GPU, the operator handle), ``run`` makes one
call through the public entry points and returns its whole output, ``work``
says what the call cannot do without, and ``exact`` gives the same output in
64 bits from plain torch.

Kinds of case:

  apply   one Dslash application on resident fields (DslashOperator.apply), the
          inner step of every solver: 4D and 3D, FP32, FP64 and FP64 in
          double-float, 18- and 12-real links, one to 32 right-hand sides, the
          16-bit and spin-pair storage formats
  batch   several lattices of different sizes in one launch (DslashBatch)
  force   the fermion force of a molecular-dynamics step (DslashOperator.force)
  solve   an even-odd mixed-precision solve (WilsonSolver.solve)
  bsolve  several right-hand sides solved together (BatchedWilsonSolver.solve)
  dropin  the reference's own call on host arrays (SSEDslash), a full
          host-to-host round trip
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sse_wilson_dslash_gb300 import _lib
from sse_wilson_dslash_gb300.device import BatchedWilsonSolver, DslashBatch, DslashOperator, WilsonSolver
from sse_wilson_dslash_gb300.legacy import SSEDslash

DEV = "cuda"
KAPPA = 0.124


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def _apply(name, dims, nd=4, prec=32, recon=18, nrhs=1, fmt="native", isign=1, cb=0):
    c = {"kind": "apply", "dims": dims, "nd": nd, "prec": prec, "recon": recon, "nrhs": nrhs, "fmt": fmt, "isign": isign,
         "cb": cb}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a test lattice, or one level of a multigrid; launch latency counts
        _apply("apply_f32_8x8x8x8", "8x8x8x8"),
        # an ordinary lattice of uneven extents with compressed links
        _apply("apply_f32_r12_12x20x28x36", "12x20x28x36", recon=12, isign=-1, cb=1),
        # the production lattice
        _apply("apply_f32_32x32x32x64", "32x32x32x64"),
        # the FP64 operator: final residuals, FP64 solvers, the 64-bit build of the reference
        _apply("apply_f64_24x24x24x48", "24x24x24x48", prec=64),
        # the spatial operator (smearing, anisotropic even-odd schemes), at an odd time extent
        _apply("apply_3d_f32_24x24x24x47", "24x24x24x47", nd=3, isign=-1),
        # a propagator's twelve spin-colour sources on one gauge field
        _apply("apply_f32_12rhs_16x16x16x32", "16x16x16x32", nrhs=12),
        # many stochastic sources with 16-bit storage
        _apply("apply_bf16_32rhs_24x24x24x48", "24x24x24x48", nrhs=32, fmt="bf16", cb=1),
        # lattices of several sizes with their own gauge fields and source counts
        {"name": "batch_f32_uneven", "kind": "batch", "fmt": "native", "recon": 18,
         "items": "16x16x16x16*8,20x20x20x40*4,24x24x24x48*2,32x32x32x64*1"},
        # the backward direction: the force on every link
        {"name": "force_f32_32x32x32x64", "kind": "force", "dims": "32x32x32x64", "prec": 32, "mode": 1, "isign": 1, "cb": 0},
        # a whole solve: FP32 inner CG, FP64 defect correction
        {"name": "solve_f32_24x24x24x48", "kind": "solve", "dims": "24x24x24x48", "inner_prec": 32, "df": False},
        # sixteen solves on one gauge field
        {"name": "bsolve_16rhs_16x16x16x32", "kind": "bsolve", "dims": "16x16x16x32", "nrhs": 16, "df": False},
        # the reference's call on the caller's (pinned) host arrays
        {"name": "dropin_f32_24x24x24x48", "kind": "dropin", "dims": "24x24x24x48", "nd": 4, "prec": 32, "isign": 1, "cb": 0},
    ]


def _extent(rng, lo, hi, even=True):
    """An extent between lo and hi, spread over its logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    v = min(max(v, lo), hi)
    return v - v % 2 if even else v


def _dims(rng, spatial=(4, 32), temporal=(4, 64), odd_t=False):
    e = [_extent(rng, *spatial) for _ in range(3)] + [_extent(rng, *temporal, even=not odd_t)]
    return "x".join(str(v) for v in e)


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "multi", "multi", "batch", "force", "solve", "bsolve", "dropin"])
    isign, cb = rng.choice([1, -1]), rng.choice([0, 1])
    if kind == "apply":
        nd = rng.choice([4, 4, 3])
        prec, fmt = rng.choice([(32, "native"), (32, "native"), (64, "native"), (64, "double_float")])
        return _apply(None, _dims(rng, odd_t=nd == 3), nd, prec, rng.choice([18, 12]), 1, fmt, isign, cb)
    if kind == "multi":
        fmt = rng.choice(["native", "native", "bf16", "f16", "f32_pairs"])
        nrhs = rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 24, 32])
        if nrhs == 1 and fmt == "native":
            nrhs = 2
        return _apply(None, _dims(rng, (4, 24), (4, 48)), 4, 32, rng.choice([18, 12]), nrhs, fmt, isign, cb)
    if kind == "batch":
        items = ",".join("%s*%d" % (_dims(rng, (4, 24), (4, 48)), rng.randint(1, 8)) for _ in range(rng.randint(2, 6)))
        return {"kind": "batch", "fmt": rng.choice(["native", "bf16"]), "recon": rng.choice([18, 12]), "items": items}
    if kind == "force":
        return {"kind": "force", "dims": _dims(rng), "prec": rng.choice([32, 32, 64]), "mode": rng.choice([0, 1]),
                "isign": isign, "cb": cb}
    if kind == "solve":
        return {"kind": "solve", "dims": _dims(rng, (6, 24), (8, 48)), "inner_prec": rng.choice([32, 32, 16]),
                "df": rng.choice([False, False, True])}
    if kind == "bsolve":
        return {"kind": "bsolve", "dims": _dims(rng, (6, 16), (8, 32)), "nrhs": rng.choice([4, 8, 16]),
                "df": rng.choice([False, False, True])}
    nd = rng.choice([4, 4, 3])
    return {"kind": "dropin", "dims": _dims(rng, (4, 24), (4, 48), odd_t=nd == 3), "nd": nd, "prec": rng.choice([32, 64]),
            "isign": isign, "cb": cb}


# ---------------------------------------------------------------------------
# Inputs, from the seed alone
# ---------------------------------------------------------------------------

def _shape(text):
    return tuple(int(v) for v in text.split("x"))


def _volume(dims):
    return dims[0] * dims[1] * dims[2] * dims[3]


def _items(case):
    out = []
    for it in case["items"].split(","):
        d, n = it.split("*")
        out.append((_shape(d), int(n)))
    return out


def _unitarise(a):
    """[n][2][3] complex rows -> [n][3][3] SU(3): Gram-Schmidt, row 2 = conj(row0 x row1)."""
    r0 = a[:, 0] / a[:, 0].abs().square().sum(-1, keepdim=True).sqrt()
    r1 = a[:, 1] - (r0.conj() * a[:, 1]).sum(-1, keepdim=True) * r0
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([r0, r1, torch.linalg.cross(r0, r1).conj()], dim=1)


def _links(V, gen, near_unit=False):
    """Random SU(3) links in the packed layout [V][4][j][i][2] (U_ij), FP64:
    Haar-like, or scattered around the unit matrix as on a smooth field."""
    out = torch.empty(V * 4, 3, 3, 2, dtype=torch.float64, device=DEV)
    for s in range(0, V * 4, 1 << 21):
        m = min(1 << 21, V * 4 - s)
        if near_unit:
            h = torch.view_as_complex(torch.randn(m, 3, 3, 2, dtype=torch.float64, device=DEV, generator=gen))
            a = (0.5 * 0.3j) * (h + h.conj().transpose(1, 2)) + torch.eye(3, dtype=torch.complex128, device=DEV)
            a = a[:, :2]
        else:
            a = torch.view_as_complex(torch.randn(m, 2, 3, 2, dtype=torch.float64, device=DEV, generator=gen))
        out[s:s + m] = torch.view_as_real(_unitarise(a).transpose(1, 2).contiguous())
    return out.reshape(-1)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _spinor(V, nrhs, gen, dtype, fmt="native"):
    psi = torch.randn(nrhs * V * 24, dtype=dtype, device=DEV, generator=gen)
    # 16-bit storage holds values that were rounded to it when they were stored
    return psi.to(torch.bfloat16).to(dtype) if fmt == "bf16" else psi


def _fields(case, seed, dims, nrhs, nd, prec, fmt):
    gen, dt = _gen(seed), torch.float32 if prec == 32 else torch.float64
    u = _links(_volume(dims), gen).to(dt)
    return u, _spinor(_volume(dims), nrhs, gen, dt, fmt)


class _DropIn:
    """The reference API's init .. free around the calls of one program."""

    def __init__(self, dims, nd, prec):
        self.api, self.nd = SSEDslash(prec), nd
        getattr(self.api, "init_sse_su3dslash" + ("_3d" if nd == 3 else ""))(dims, *_lib.canonical_callbacks(nd, dims))
        self.call = self.api.sse_su3dslash_wilson_3d if nd == 3 else self.api.sse_su3dslash_wilson

    def __del__(self):
        getattr(self.api, "free_sse_su3dslash" + ("_3d" if self.nd == 3 else ""))()


def _host(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "apply":
        dims = _shape(case["dims"])
        op = DslashOperator(dims, nd=case["nd"], prec=case["prec"], recon=case["recon"], nrhs=case["nrhs"],
                            spinor_format=case["fmt"])
        u, psi = _fields(case, seed, dims, case["nrhs"], case["nd"], case["prec"], case["fmt"])
        s.update(op=op, gauge=op.pack_gauge(u), psi=op.pack_spinor(psi, case["cb"]), out=op.new_spinor().zero_())
        if case["fmt"] == "double_float":
            s["res"] = torch.zeros(op.volume * 24, dtype=torch.float64, device=DEV)
        else:
            s["view"] = _views(s["out"], case["fmt"], case["prec"], op.stride * op.nrhs)
    elif kind == "batch":
        items, gen = [], _gen(seed)
        for k, (dims, nrhs) in enumerate(_items(case)):
            op = DslashOperator(dims, recon=case["recon"], nrhs=nrhs, spinor_format=case["fmt"])
            u = _links(op.volume, gen).to(torch.float32)
            psi = _spinor(op.volume, nrhs, gen, torch.float32, case["fmt"])
            items.append(dict(op=op, gauge=op.pack_gauge(u), psi=op.pack_spinor(psi, k % 2), res=op.new_spinor().zero_(),
                              isign=1 - 2 * (k % 2), cb=k % 2))
        s["batch"] = DslashBatch(items, recon=case["recon"], spinor_format=case["fmt"])
        s["batch"].autotune()
        s["view"] = [_views(it["res"], case["fmt"], 32, it["op"].stride * it["op"].nrhs) for it in items]
    elif kind == "force":
        dims = _shape(case["dims"])
        op = DslashOperator(dims, prec=case["prec"])
        u, psi = _fields(case, seed, dims, 1, 4, case["prec"], "native")
        chi = _spinor(op.volume, 1, _gen(seed + 7919), psi.dtype)
        s.update(op=op, gauge=op.pack_gauge(u), psi=op.pack_spinor(psi, case["cb"]),
                 chi=op.pack_spinor(chi, 1 - case["cb"]), out=torch.zeros(op.volume * 72, dtype=psi.dtype, device=DEV))
    elif kind in ("solve", "bsolve"):
        dims = _shape(case["dims"])
        gen, nrhs = _gen(seed), case.get("nrhs", 1)
        u = _links(_volume(dims), gen, near_unit=True)
        if kind == "solve":
            s["solver"] = WilsonSolver(dims, KAPPA, tol=1e-11, inner_prec=case["inner_prec"],
                                       inner_tol=1e-5 if case["inner_prec"] == 32 else 1e-3, outer_double_float=case["df"])
        else:
            s["solver"] = BatchedWilsonSolver(dims, nrhs, KAPPA, tol=1e-11, outer_double_float=case["df"])
        s["solver"].set_gauge(u)
        s["b"] = _spinor(_volume(dims), nrhs, gen, torch.float64)
        s["x"] = torch.zeros_like(s["b"])
    else:
        dims = _shape(case["dims"])
        u, psi = _fields(case, seed, dims, 1, case["nd"], case["prec"], "native")
        s.update(u=_host(u), psi=_host(psi), res=_host(torch.zeros_like(psi)), api=_DropIn(dims, case["nd"], case["prec"]))
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "apply":
        s["op"].apply(s["gauge"], s["psi"], case["isign"], case["cb"], out=s["out"])
        if case["fmt"] == "double_float":
            return s["op"].unpack_spinor(s["out"], 1 - case["cb"], s["res"])
        return s["view"]
    if kind == "batch":
        s["batch"].launch()
        return s["view"]
    if kind == "force":
        return s["op"].force(s["gauge"], s["psi"], s["chi"], case["isign"], case["cb"], s["out"], mode=case["mode"])
    if kind in ("solve", "bsolve"):
        s["solver"].solve(s["b"], s["x"])
        return s["x"]
    s["api"].call(s["u"], s["psi"], s["res"], case["isign"], case["cb"])
    return s["res"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

_SPINOR_BYTES = {"native": 96, "bf16": 48, "f16": 52, "f32_pairs": 96, "double_float": 192}


def _dslash_work(dims, nd, prec, recon, nrhs, fmt):
    """One application: every source spinor and every link read once, every output written once."""
    V, real = _volume(dims), 4 if prec == 32 else 8
    sp = 192 if prec == 64 else _SPINOR_BYTES[fmt]
    return {"bytes": V * nrhs * sp + V * nd * recon * real, "flops": (1320 if nd == 4 else 984) * (V // 2) * nrhs}


def work(case):
    kind = case["kind"]
    if kind == "apply":
        return _dslash_work(_shape(case["dims"]), case["nd"], case["prec"], case["recon"], case["nrhs"], case["fmt"])
    if kind == "batch":
        w = [_dslash_work(d, 4, 32, case["recon"], n, case["fmt"]) for d, n in _items(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    V = _volume(_shape(case["dims"]))
    if kind == "force":
        real = 4 if case["prec"] == 32 else 8
        # psi and chi, the links (mode 1) and the force; two 3x3 outer products a link, and one 3x3 product
        return {"bytes": V * real * (24 + 72 + (72 if case["mode"] else 0)),
                "flops": V * 4 * (24 + 2 * 72 + (216 if case["mode"] else 0))}
    if kind in ("solve", "bsolve"):
        # about 44 iterations of M^+ M at this kappa: four applications each; links, sources and solutions once
        n = case.get("nrhs", 1)
        return {"bytes": V * (4 * 18 * 8 + n * 24 * 8), "flops": 44 * 4 * 1320 * (V // 2) * n}
    return _dslash_work(_shape(case["dims"]), case["nd"], case["prec"], 18, 1, "native")


# ---------------------------------------------------------------------------
# The same outputs in 64 bits, from plain torch
# ---------------------------------------------------------------------------

def _views(buf, fmt, prec, cs):
    """The real numbers of an internal field (a byte tensor)."""
    if fmt == "bf16":
        return buf.view(torch.bfloat16)
    if fmt == "f16":
        return [buf[:48 * cs].view(torch.float16), buf[48 * cs:].view(torch.float32)]
    return buf.view(torch.float32 if prec == 32 else torch.float64)


def _stored(psi, fmt, dims, nd, cb, stride):
    """[nrhs][Vh][4][3] complex -> the reals of the internal field, laid out like _views."""
    nrhs, Vh = psi.shape[:2]
    v = torch.view_as_real(psi).reshape(nrhs, Vh, 24)
    norm = None
    if fmt == "f16":
        norm = v.abs().amax(-1)
        v = v / norm.clamp_min(1e-300)[..., None]
    if fmt == "f32_pairs":
        p = v.reshape(nrhs, Vh, 2, 2, 3, 2)                      # spin half, spin, colour, part
        v = p.permute(0, 1, 2, 4, 5, 3).reshape(nrhs, Vh, 24)    # half, colour, part, spin
    per = {"native": 4, "f32_pairs": 4, "bf16": 8, "f16": 8, "f64": 2}[fmt]
    out = torch.zeros(24 // per, stride, nrhs, per, dtype=torch.float64, device=psi.device)
    out[:, :Vh] = v.reshape(nrhs, Vh, 24 // per, per).permute(2, 1, 0, 3)
    if norm is None:
        return out.reshape(-1)
    n = torch.zeros(stride, nrhs, dtype=torch.float64, device=psi.device)
    n[:Vh] = norm.T
    return [out.reshape(-1), n.reshape(-1)]


class _Lattice:
    """Checkerboarded neighbour tables (QDP++ cb2 order for nd 4, cb3d for 3)."""

    def __init__(self, dims, nd):
        Lx, Ly, Lz, Lt = dims
        self.nd, self.Vh = nd, _volume(dims) // 2
        i = torch.arange(self.Vh, device=DEV)
        if nd == 4:
            xh, y, z, t = i % (Lx // 2), i // (Lx // 2) % Ly, i // (Lx // 2 * Ly) % Lz, i // (Lx // 2 * Ly * Lz)
        else:
            t, xh, y, z = i % Lt, i // Lt % (Lx // 2), i // (Lt * (Lx // 2)) % Ly, i // (Lt * (Lx // 2) * Ly)

        def index(c):
            c = [v % L for v, L in zip(c, dims)]
            if nd == 4:
                return ((c[3] * Lz + c[2]) * Ly + c[1]) * (Lx // 2) + c[0] // 2
            return c[3] + Lt * (c[0] // 2 + Lx // 2 * (c[1] + Ly * c[2]))

        self.nbr = []  # [target parity][mu][forward, backward] -> source index
        for p in (0, 1):
            x = 2 * xh + (p + y + z + (t if nd == 4 else 0)) % 2
            rows = []
            for mu in range(nd):
                f, b = [x, y, z, t], [x, y, z, t]
                f[mu], b[mu] = f[mu] + 1, b[mu] - 1
                rows.append((index(f), index(b)))
            self.nbr.append(rows)


def _gammas():
    """DeGrand-Rossi gamma matrices."""
    i = 1j
    g = [[[0, 0, 0, i], [0, 0, i, 0], [0, -i, 0, 0], [-i, 0, 0, 0]],
         [[0, 0, 0, -1], [0, 0, 1, 0], [0, 1, 0, 0], [-1, 0, 0, 0]],
         [[0, 0, i, 0], [0, 0, 0, -i], [-i, 0, 0, 0], [0, i, 0, 0]],
         [[0, 0, 1, 0], [0, 0, 0, 1], [1, 0, 0, 0], [0, 1, 0, 0]]]
    return [torch.tensor(m, dtype=torch.complex128, device=DEV) for m in g]


def _spin(m, psi):
    """Spin matrix m (one entry a row) times psi [..., 4, 3]."""
    out = torch.zeros_like(psi)
    for a in range(4):
        for b in range(4):
            if m[a, b] != 0:
                out[..., a, :] += m[a, b] * psi[..., b, :]
    return out


def _colour(U, h):
    """U [Vh][3][3] times h [nrhs][Vh][4][3]."""
    out = torch.zeros_like(h)
    for j in range(3):
        out += U[:, None, :, j] * h[..., j, None]
    return out


def _matrices(u, recon=18):
    """Packed links -> [V][4][3][3] complex128 U_ij, the third row rebuilt for recon 12."""
    U = torch.view_as_complex(u.double().reshape(-1, 4, 3, 3, 2)).transpose(2, 3).contiguous()
    if recon == 12:
        U[:, :, 2] = torch.linalg.cross(U[:, :, 0], U[:, :, 1]).conj()
    return U


def _dslash(lat, U, psi, isign, cb):
    """[nrhs][Vh][4][3] on checkerboard cb -> the other one."""
    pt, Vh = 1 - cb, lat.Vh
    out = torch.zeros_like(psi)
    for mu, g in enumerate(_gammas()[:lat.nd]):
        f, b = lat.nbr[pt][mu]
        h = psi[:, f]
        out += _colour(U[pt * Vh:(pt + 1) * Vh, mu], h - isign * _spin(g, h))
        h = psi[:, b]
        out += _colour(U[cb * Vh + b, mu].conj().transpose(1, 2), h + isign * _spin(g, h))
    return out


def _half(psi, dims, nrhs, cb):
    """Packed [nrhs][V][4][3][2] -> checkerboard cb, complex128."""
    Vh = _volume(dims) // 2
    return torch.view_as_complex(psi.double().reshape(nrhs, 2, Vh, 4, 3, 2)[:, cb].contiguous())


def _exact_apply(dims, nd, recon, u, psi, nrhs, isign, cb, fmt):
    lat, U = _Lattice(dims, nd), _matrices(u, recon)
    src = _half(psi, dims, nrhs, cb)
    if fmt == "f16":  # the stored values: halves of the largest component, and that one
        v = torch.view_as_real(src).reshape(nrhs, lat.Vh, 24).float()
        n = v.abs().amax(-1, keepdim=True)
        v = (v * (1.0 / n)).half().double() * n.double()
        src = torch.view_as_complex(v.reshape(nrhs, lat.Vh, 4, 3, 2).contiguous())
    return torch.cat([_dslash(lat, U, src[r:r + 1], isign, cb) for r in range(nrhs)])


def _packed(res, dims, nrhs, cb):
    out = torch.zeros(nrhs, 2, _volume(dims) // 2, 24, dtype=torch.float64, device=res.device)
    out[:, cb] = torch.view_as_real(res).reshape(nrhs, -1, 24)
    return out.reshape(-1)


def _exact_force(case, seed):
    dims = _shape(case["dims"])
    u, psi = _fields(case, seed, dims, 1, 4, case["prec"], "native")
    chi = _spinor(_volume(dims), 1, _gen(seed + 7919), psi.dtype)
    lat, U = _Lattice(dims, 4), _matrices(u)
    cb, isign, Vh = case["cb"], case["isign"], lat.Vh
    pt = 1 - cb
    p, c = _half(psi, dims, 1, cb)[0], _half(chi, dims, 1, pt)[0]
    out = torch.empty(2 * Vh, 4, 3, 3, dtype=torch.complex128, device=DEV)
    for mu, g in enumerate(_gammas()):
        # links of pt: chi(x) (1 - isign g) psi(x + mu); links of cb: the backward hop into y = x + mu
        f = p[lat.nbr[pt][mu][0]]
        f = f - isign * _spin(g, f)
        out[pt * Vh:(pt + 1) * Vh, mu] = torch.einsum("vsi,vsj->vij", c, f.conj())
        h = p + isign * _spin(g, p)
        out[cb * Vh:(cb + 1) * Vh, mu] = torch.einsum("vsi,vsj->vij", h, c[lat.nbr[cb][mu][0]].conj())
    if case["mode"] == 1:
        for mu in range(4):
            m = out[:, mu] @ U[:, mu].conj().transpose(1, 2)
            m = (m - m.conj().transpose(1, 2)) / 2
            tr = m.diagonal(dim1=1, dim2=2).sum(-1) / 3
            out[:, mu] = m - tr[:, None, None] * torch.eye(3, dtype=torch.complex128, device=DEV)
    return torch.view_as_real(out.transpose(2, 3).contiguous()).reshape(-1)


def _exact_solve(case, seed):
    """CG on M^+ M, all in 64 bits, to 1e-14."""
    dims, nrhs, gen = _shape(case["dims"]), case.get("nrhs", 1), _gen(seed)
    u = _links(_volume(dims), gen, near_unit=True)
    b = _half(_spinor(_volume(dims), nrhs, gen, torch.float64), dims, nrhs, 0)
    lat, U = _Lattice(dims, 4), _matrices(u)
    del u

    def M(v, sign):
        return v - KAPPA ** 2 * _dslash(lat, U, _dslash(lat, U, v, sign, 0), sign, 1)

    def norm(v):
        return torch.view_as_real(v).square().sum((1, 2, 3, 4))

    def over(a):
        return a[:, None, None, None]

    x, r = torch.zeros_like(b), M(b, -1)
    p, rr = r.clone(), norm(r)
    goal = rr * 1e-28
    for k in range(400):
        if k % 4 == 0 and bool((rr <= goal).all()):
            break
        q = M(p, 1)
        a = rr / norm(q)
        x += over(a) * p
        r -= over(a) * M(q, -1)
        new = norm(r)
        p = r + over(new / rr) * p
        rr = new
    return _packed(x, dims, nrhs, 0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        dims, fmt, nrhs = _shape(case["dims"]), case["fmt"], case["nrhs"]
        u, psi = _fields(case, seed, dims, nrhs, case["nd"], case["prec"], fmt)
        res = _exact_apply(dims, case["nd"], case["recon"], u, psi, nrhs, case["isign"], case["cb"], fmt)
        if fmt == "double_float":
            return _packed(res, dims, 1, 1 - case["cb"])
        stride = -(-(_volume(dims) // 2) // 64) * 64
        return _stored(res, "f64" if case["prec"] == 64 else fmt, dims, case["nd"], 1 - case["cb"], stride)
    if kind == "batch":
        out, gen = [], _gen(seed)
        for k, (dims, nrhs) in enumerate(_items(case)):
            V = _volume(dims)
            u = _links(V, gen).to(torch.float32)
            psi = _spinor(V, nrhs, gen, torch.float32, case["fmt"])
            res = _exact_apply(dims, 4, case["recon"], u, psi, nrhs, 1 - 2 * (k % 2), k % 2, case["fmt"])
            out.append(_stored(res, case["fmt"], dims, 4, 1 - k % 2, -(-(V // 2) // 64) * 64))
        return out
    if kind == "force":
        return _exact_force(case, seed)
    if kind in ("solve", "bsolve"):
        return _exact_solve(case, seed)
    dims = _shape(case["dims"])
    u, psi = _fields(case, seed, dims, 1, case["nd"], case["prec"], "native")
    res = _exact_apply(dims, case["nd"], 18, u, psi, 1, case["isign"], case["cb"], "native")
    return _packed(res, dims, 1, 1 - case["cb"])

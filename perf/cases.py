"""Performance cases: what a user of the FFT-VIE framework has it compute.

A case is a dict of plain values.  ``kind`` names the call:

* ``apply`` / ``adjoint``: the VIE operator and its Hermitian adjoint on body
  vectors (``VieOperator.apply`` / ``apply_adjoint``), the call every GMRES
  iteration makes;
* ``grid``: the raw N operator on full grids (``apply_N``), as MATLAB's
  ``func.mvp_N`` and the coupled coil/body product call it;
* ``fields``: total E and H fields of solved currents (``fields``);
* ``solve``: a whole ``gmres`` call;
* ``assemble``: the Green's tensor of a grid (``assemble_green``);
* ``loops``: incident fields of coil loops (``incident_loops``).

``prec`` is the arithmetic: ``c64`` (complex64), ``ff`` (complex128 held as
pairs of FP32 numbers) or ``c128`` (native complex128).

The operators here are built by this file: N and K moments of the free-space
dyadic Green's function by the two-point Gauss rule per axis, with the point
term of N at the self offset, and a seeded ellipsoid phantom.  A program keeps
its operator handle while it applies it to many vectors, so one handle is kept
for the case at hand and the states of a case share it; their vectors,
currents and coil positions come from the seed.
"""
import json
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marie-tools_gb300"))

import marie_gb300 as mg  # noqa: E402
from marie_gb300 import operator as mgop  # noqa: E402

C0 = 299792458.0
MU0 = 4e-7 * math.pi
EPS0 = 1.0 / (C0 * C0 * MU0)
RES, F7T, F3T = 2e-3, 297.2e6, 128e6

# (l, l') of the ten PWL moment pairs; mirror signs of the six N and three K
# components and of the ten pairs along each axis; block of (row, column)
PAIRS = [(0, 0), (1, 1), (2, 2), (3, 3), (0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
SIGN_N = [(1, -1, -1, 1, 1, 1), (1, -1, 1, 1, -1, 1), (1, 1, -1, 1, -1, 1)]
SIGN_K = [(-1, 1, 1), (1, -1, 1), (1, 1, -1)]
SIGN_L = [(1, 1, 1, 1, -1, 1, 1, -1, -1, 1), (1, 1, 1, 1, 1, -1, 1, -1, 1, -1), (1, 1, 1, 1, 1, 1, -1, 1, -1, -1)]
PQ_N = [[1, 2, 3], [2, 4, 5], [3, 5, 6]]
PQ_K = [[0, -3, 2], [3, 0, -1], [-2, 1, 0]]
LLP = [[1, 5, 6, 7], [-5, 2, 8, 9], [-6, 8, 3, 10], [-7, 9, 10, 4]]
SLP = [[1, -1, -1, -1], [-1, 1, 1, 1], [-1, 1, 1, 1], [-1, 1, 1, 1]]


def _case(name, kind, n1, n2, n3, pwl, prec, nrhs, **more):
    return dict(name=name, kind=kind, n1=n1, n2=n2, n3=n3, pwl=pwl, prec=prec, nrhs=nrhs, res=RES, freq=F7T) | more


def listed():
    return [
        # the smallest call: one product on the 32^3 PWC sphere-sized body, as a solver driven from outside makes it
        _case("apply-32-pwc-c64", "apply", 32, 32, 32, False, "c64", 1, res=5e-3, freq=F3T),
        # one product of the single-loop head phantom at 2 mm, PWL
        _case("apply-96-pwl-c64", "apply", 96, 96, 96, True, "c64", 1),
        # the largest call: the block product of 64 loop ports on the 128^3 PWL phantom
        _case("apply-128-pwl-c64-64", "apply", 128, 128, 128, True, "c64", 64),
        # one body of the uneven PWC batch: 112^3 with 7 loops
        _case("apply-112-pwc-c64-7", "apply", 112, 112, 112, False, "c64", 7),
        # a body cut to its bounding box: no edge is a multiple of 16
        _case("apply-odd-pwl-c64-3", "apply", 60, 77, 90, True, "c64", 3),
        # the adjoint product of the refinement loop and the gradient: complex128 in FP32 pairs
        _case("adjoint-96-pwl-ff", "adjoint", 96, 96, 96, True, "ff", 1),
        # mvp_N of a MATLAB caller on its full double grid, the default handle
        _case("grid-48-pwl-c128", "grid", 48, 56, 40, True, "c128", 1),
        # E and H of four solved ports for maps, in single precision
        _case("fields-96-pwl-c64-4", "fields", 96, 96, 96, True, "c64", 4),
        # a whole solve of a small PWC body to 1e-6, the drop-in is_gmres_vie
        _case("solve-32-pwc-ff", "solve", 32, 32, 32, False, "ff", 1, res=5e-3, freq=F3T, mode="fp64", tol=1e-6, body="sphere"),
        # a whole multi-port solve by block GMRES, to a tolerance that finite differences of the fields need
        _case("solve-48-pwl-block-8", "solve", 48, 48, 48, True, "ff", 8, res=4e-3, mode="block", tol=1e-10),
        # the Green's tensor of a new grid
        _case("assemble-48-pwl", "assemble", 48, 48, 48, True, "c128", 1),
        # the right-hand sides of four loop ports
        _case("loops-64-pwl-4", "loops", 64, 64, 64, True, "c128", 4, res=3e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """n, or the next smaller edge without a prime factor above 31."""
    while True:
        m = n
        for p in range(2, 32):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n -= 1


def draw(rng):
    """Any of the calls, edges 16-128 (any integer; multiples of 16 half the time), 1-64 right-hand sides."""
    kind, prec = rng.choice([("apply", "c64")] * 5 + [("apply", "ff"), ("apply", "c128"), ("adjoint", "c64"), ("adjoint", "ff"),
                                                     ("grid", "c64"), ("grid", "c128"), ("fields", "c64"), ("fields", "c128"),
                                                     ("solve", "ff"), ("assemble", "c128"), ("loops", "c128")])
    pwl = rng.random() < 0.6
    top = {"c64": 128, "ff": 112, "c128": 64}[prec]
    if kind in ("solve", "assemble", "loops"):
        top = {"solve": 48, "assemble": 56, "loops": 96}[kind]
    even = prec == "ff" or (rng.random() < 0.5 and kind not in ("assemble", "loops"))
    edges = []
    for _ in range(3):
        e = _log_int(rng, 16, top)
        edges.append(max(16, 16 * int(round(e / 16))) if even else e)
    if kind in ("grid", "solve"):
        edges = [_smooth(e) for e in edges]
    nvox = edges[0] * edges[1] * edges[2] * (12 if pwl else 3)
    cost = {"c64": 1.0, "ff": 8.0, "c128": 30.0}[prec]
    most = int(128 ** 3 * 12 * 64 / (2 * cost * nvox))
    nrhs = _log_int(rng, 1, max(1, min({"apply": 64, "loops": 8, "solve": 4}.get(kind, 16), most)))
    c = dict(kind=kind, n1=edges[0], n2=edges[1], n3=edges[2], pwl=pwl, prec=prec, nrhs=1 if kind == "assemble" else nrhs, res=RES,
             freq=rng.choice([F3T, F7T]))
    if kind == "solve":
        c |= dict(mode="fp64", tol=1e-6, res=4e-3, body="sphere")
    return c


# ---------------------------------------------------------------------------
# Operands
# ---------------------------------------------------------------------------

def _dims(case):
    return case["n1"], case["n2"], case["n3"]


def _ce(freq):
    return 1j * 2 * math.pi * freq * EPS0


def _moments(case, kernel):
    """I_V (n1, n2, n3, pairs, components), complex128 on the GPU: two Gauss points per axis and voxel."""
    n, res, k0 = _dims(case), case["res"], 2 * math.pi * case["freq"] / C0
    nc = 6 if kernel == "N" else 3
    pairs = PAIRS if case["pwl"] else PAIRS[:1]
    g, h = 1 / math.sqrt(3), res / 2
    # weights of the differences (-2g, 0, 2g): [l is linear][l' is linear]
    axis = [[(1, 2, 1), (g / 2, 0, -g / 2)], [(-g / 2, 0, g / 2), (-g * g / 4, g * g / 2, -g * g / 4)]]
    dev = dict(dtype=torch.float64, device="cuda")
    out = torch.zeros((*n, len(pairs), nc), dtype=torch.complex128, device="cuda")
    r = [res * torch.arange(m, **dev) for m in n]
    for iu in range(27):
        u = (iu % 3, iu // 3 % 3, iu // 9)
        X = (r[0] + (u[0] - 1) * 2 * g * h)[:, None, None]
        Y = (r[1] + (u[1] - 1) * 2 * g * h)[None, :, None]
        Z = (r[2] + (u[2] - 1) * 2 * g * h)[None, None, :]
        R2 = X * X + Y * Y + Z * Z
        zero = R2 == 0
        R = torch.where(zero, torch.ones_like(R2), R2).sqrt()
        Ge = torch.polar(torch.where(zero, torch.zeros_like(R), 1 / (4 * math.pi * R ** 3)), -k0 * R)
        if kernel == "N":
            a = torch.complex(3 / (R * R) - k0 * k0, 3 * k0 / R) * Ge
            b = torch.complex(torch.ones_like(R), k0 * R) * Ge
            xx, yy, zz = a * (X * X) - b, a * (Y * Y) - b, a * (Z * Z) - b
            f = [-(yy + zz), a * (X * Y), a * (X * Z), -(xx + zz), a * (Y * Z), -(xx + yy)]
        else:
            b = torch.complex(torch.ones_like(R), k0 * R) * Ge
            f = [-(b * X), -(b * Y), -(b * Z)]
        for j, (l, lp) in enumerate(pairs):
            w = h ** 6
            for d in range(3):
                w *= axis[int(l == d + 1)][int(lp == d + 1)][u[d]]
            if w:
                for c in range(nc):
                    out[..., j, c] += w * f[c]
    signs = SIGN_N if kernel == "N" else SIGN_K
    for j in range(len(pairs)):
        for c in range(nc):
            for d in range(3):
                if signs[d][c] * SIGN_L[d][j] < 0:
                    out.select(d, 0)[..., j, c] = 0   # odd blocks vanish on their zero-offset plane
    if kernel == "N":
        for j in range(min(4, len(pairs))):
            for c in (0, 3, 5):
                out[0, 0, 0, j, c] += 2 / 3 * (res ** 3 if j == 0 else res ** 3 / 12)
    return out


def _phantom(case):
    """(body mask, Mr) on the grid, numpy: an ellipsoid with twelve seeded inner ellipsoids, or a homogeneous sphere (ellipsoid)."""
    n = _dims(case)
    rng = np.random.RandomState(n[0] * 10007 + n[1] * 101 + n[2])
    ax = [np.linspace(-1, 1, m + 2)[1:-1] for m in n]
    X, Y, Z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    if case.get("body") == "sphere":
        mask = X ** 2 + Y ** 2 + Z ** 2 <= 0.75 ** 2
        return mask, np.where(mask, 50.0, 1.0) + np.where(mask, 0.6, 0.0) / _ce(case["freq"])
    mask = (X / 0.84) ** 2 + (Y / 0.68) ** 2 + (Z / 0.94) ** 2 <= 1
    er, se = np.where(mask, 40.0, 1.0), np.where(mask, 0.5, 0.0)
    for _ in range(12):
        c, s = rng.uniform(-0.4, 0.4, 3), rng.uniform(0.15, 0.4, 3)
        inner = mask & (((X - c[0]) / s[0]) ** 2 + ((Y - c[1]) / s[1]) ** 2 + ((Z - c[2]) / s[2]) ** 2 <= 1)
        er[inner], se[inner] = rng.uniform(5, 80), rng.uniform(0.02, 2.0)
    return mask, er + se / _ce(case["freq"])


def _body(case):
    mask, Mr = _phantom(case)
    idx = np.nonzero(mask.reshape(-1, order="F"))[0].astype(np.int64)
    return idx, Mr


def _ql(case):
    return 12 if case["pwl"] else 3


_kept = {}   # the operator handle of the case at hand


def _operator(case):
    key = json.dumps({k: v for k, v in case.items() if k not in ("name", "kind", "mode", "tol")} | {"K": case["kind"] == "fields"}, sort_keys=True)
    if key not in _kept:
        for op in _kept.values():
            op.close()
        _kept.clear()
        idx, Mr = _body(case)
        nD = int(np.prod(_dims(case)))
        idx_solution = np.concatenate([c * nD + idx for c in range(_ql(case))])
        if case["kind"] == "solve":
            dense = {"N": mgop.assemble_green(_dims(case), case["res"], case["freq"], case["pwl"])}
        else:
            dense = {k: _moments(case, k).cpu().numpy() for k in (("N", "K") if case["kind"] == "fields" else ("N",))}
        torch.cuda.empty_cache()
        bits = {"c64": 2, "ff": 4, "c128": 3}[case["prec"]]
        if case["kind"] == "solve":
            bits |= 2
        _kept[key] = mg.VieOperator(_dims(case), case["res"], case["freq"], idx_solution, Mr, dense["N"], dense.get("K"), pwl=case["pwl"],
                                    precisions=bits, max_rhs=case["nrhs"])
    return _kept[key]


def _vector(case, length, seed):
    """Krylov-like vectors: unit norm per right-hand side, the linear PWL moments a tenth of the constant ones."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    dt = torch.complex64 if case["prec"] == "c64" else torch.complex128
    x = torch.randn((case["nrhs"], _ql(case), length), dtype=dt, device="cuda", generator=gen)
    if case["pwl"]:
        x *= torch.tensor([1.0, 0.1, 0.1, 0.1] * 3, device="cuda", dtype=dt)[None, :, None]
    x /= torch.linalg.vector_norm(x, dim=(1, 2), keepdim=True)
    return x.reshape(-1)


def _loops(case, seed):
    """(origin, loops): 5 cm loops on a cylinder around the body, centres and normals seeded."""
    rng, n, res = np.random.RandomState(seed % (1 << 31)), np.asarray(_dims(case)), case["res"]
    origin = -0.5 * res * (n - 1)
    t, z = rng.uniform(0, 2 * math.pi, case["nrhs"]), rng.uniform(-0.3, 0.3, case["nrhs"]) * res * n[2]
    rad = 0.5 * res * max(n[0], n[1]) + 0.04
    nrm = np.stack([np.cos(t), np.sin(t), rng.uniform(-0.17, 0.17, case["nrhs"])], 1)
    return origin, np.concatenate([np.stack([rad * np.cos(t), rad * np.sin(t), z], 1), nrm], 1)


def _loop_moments(case, origin, loops, idx, radius=0.025, nseg=64):
    """The field of unit currents along regular 64-gons, tested onto the body's basis with three Gauss points per axis; complex128."""
    n, res, k0 = _dims(case), case["res"], 2 * math.pi * case["freq"] / C0
    q, w = (torch.from_numpy(v).cuda() for v in np.polynomial.legendre.leggauss(3))
    centre = torch.from_numpy(origin + res * np.stack([idx % n[0], idx // n[0] % n[1], idx // (n[0] * n[1])], 1)).cuda()
    L = 4 if case["pwl"] else 1
    out = torch.zeros((len(loops), 3, L, len(idx)), dtype=torch.complex128, device="cuda")
    for i, lp in enumerate(loops):
        m = lp[3:] / np.linalg.norm(lp[3:])
        e1 = np.cross(m, [1.0, 0, 0] if abs(m[0]) < 0.9 else [0, 1.0, 0])
        e1 /= np.linalg.norm(e1)
        t = 2 * math.pi * np.arange(nseg + 1) / nseg
        p = lp[:3] + radius * (np.cos(t)[:, None] * e1 + np.sin(t)[:, None] * np.cross(m, e1))
        mid, dl = (torch.from_numpy(v).cuda() for v in (0.5 * (p[1:] + p[:-1]), p[1:] - p[:-1]))
        for a in range(27):
            s = torch.stack([q[a % 3], q[a // 3 % 3], q[a // 9]])
            wt = float(w[a % 3] * w[a // 3 % 3] * w[a // 9]) / 8
            at = centre + 0.5 * res * s
            E = torch.zeros((3, len(idx)), dtype=torch.complex128, device="cuda")
            for k in range(nseg):
                R = torch.linalg.vector_norm(at - mid[k], dim=1)
                E += torch.polar(1 / (4 * math.pi * R), -k0 * R)[None, :] * dl[k][:, None]
            E *= -1j * 2 * math.pi * case["freq"] * MU0 * wt
            for l in range(L):
                out[i, :, l] += E * (1.0 if l == 0 else 12.0 * float(s[l - 1]) / 2)
    return out.reshape(len(loops), -1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        # another seed is another voxel edge
        return dict(kind=kind, dims=_dims(case), res=case["res"] * (1 + (seed % 1009) * 1e-4), freq=case["freq"], pwl=case["pwl"])
    op = _operator(case)
    idx, Mr = _body(case)
    st = dict(kind=kind, op=op)
    if kind == "loops":
        origin, loops = _loops(case, seed)
        return st | dict(origin=origin, loops=loops)
    if kind == "solve":
        origin, loops = _loops(case, seed)
        mr = torch.from_numpy(Mr.reshape(-1, order="F")[idx]).cuda()
        b = _ce(case["freq"]) * (1 - 1 / mr)[None, None, :] * _loop_moments(case, origin, loops, idx, nseg=8).reshape(len(loops), _ql(case), -1)
        return st | dict(b=b.reshape(-1).contiguous(), mode=case["mode"], tol=case["tol"])
    st["x"] = _vector(case, int(np.prod(_dims(case))) if kind == "grid" else len(idx), seed)
    if kind == "fields":
        st["Ue"], st["Ub"] = (_vector(case, len(idx), seed + k) for k in (1001, 2003))
    return st


def run(state):
    kind, op = state["kind"], state.get("op")
    if kind == "apply":
        return op.apply(state["x"])
    if kind == "adjoint":
        return op.apply_adjoint(state["x"])
    if kind == "grid":
        return op.apply_N(state["x"])
    if kind == "fields":
        return op.fields(state["x"], state["Ue"], state["Ub"])
    if kind == "solve":
        x, _report = op.gmres(state["b"], restart=50, tol=state["tol"], maxit=200, mode=state["mode"])
        return x
    if kind == "loops":
        return op.incident_loops(state["origin"], state["loops"], 0.025)
    return mgop.assemble_green(state["dims"], state["res"], state["freq"], state["pwl"])


def work(case):
    """Bytes: vectors in and out and each distinct Green's-tensor value once.  Operations: the zero-padded transforms along each axis (rows
    that are not zero by construction), the block product at every frequency; kernel values for the two generators."""
    n, C, kind = _dims(case), _ql(case), case["kind"]
    nD, nrhs, s = n[0] * n[1] * n[2], case["nrhs"], 8 if case["prec"] == "c64" else 16
    Ns = len(_body(case)[0])
    pairs = 10 if case["pwl"] else 1
    if kind == "assemble":
        # per offset a 4-point rule in each of six dimensions has 13 distinct differences per axis; about 60 operations a kernel value
        return dict(bytes=16 * nD * pairs * 6, flops=13 ** 3 * 60 * nD)
    if kind == "loops":
        # 27 points, 64 segments, about 40 operations each
        return dict(bytes=16 * C * Ns * nrhs, flops=27 * 64 * 40 * Ns * nrhs)
    m = [2 * v for v in n]
    fft = 5 * (n[1] * n[2] * m[0] * math.log2(m[0]) + m[0] * n[2] * m[1] * math.log2(m[1]) + m[0] * m[1] * m[2] * math.log2(m[2]))
    product = 8 * 8 * nD * 9 * (16 if case["pwl"] else 1)
    one = 2 * C * fft + product
    green = 6 * pairs * nD * s
    vec = (C * nD if kind == "grid" else C * Ns) * nrhs * s
    if kind == "fields":
        return dict(bytes=5 * vec + 1.5 * green, flops=nrhs * (2 * one - product / 3))
    if kind == "solve":
        # the residual alone decides how many products a solve takes; sixty is what a body of this kind needs at the least
        return dict(bytes=60 * (2 * vec + green), flops=60 * nrhs * one)
    return dict(bytes=2 * vec + green, flops=nrhs * one)


# ---------------------------------------------------------------------------
# The same results in 64 bits, plain torch
# ---------------------------------------------------------------------------

def _spectra(case, kernel):
    """FFT of the circulant extension of each block, {block: tensor on the (2n1, 2n2, 2n3) grid}."""
    iv = _moments(case, kernel)
    n, signs = _dims(case), SIGN_N if kernel == "N" else SIGN_K
    out = {}
    for j in range(iv.shape[3]):
        for c in range(iv.shape[4]):
            t = iv[..., j, c]
            for d in range(3):
                gap = torch.zeros_like(t.narrow(d, 0, 1))
                t = torch.cat([t, gap, signs[d][c] * SIGN_L[d][j] * t.narrow(d, 1, n[d] - 1).flip(d)], d)
            out[(j, c)] = torch.fft.fftn(t)
    return out


def _entries(case, kernel, adjoint):
    for p in range(3):
        for q in range(3):
            if kernel == "K" and p == q:
                continue
            k = (PQ_N if kernel == "N" else PQ_K)[p][q]
            sk = 1 if k > 0 else -1
            for l in range(4 if case["pwl"] else 1):
                for lp in range(4 if case["pwl"] else 1):
                    j = LLP[l][lp] if case["pwl"] else 1
                    s = sk * (1 if j > 0 else -1)
                    if adjoint:
                        s *= (SLP[l][lp] if case["pwl"] else 1) * (-1 if kernel == "K" else 1)
                    L = 4 if case["pwl"] else 1
                    yield L * p + l, L * q + lp, (abs(j) - 1, abs(k) - 1), s


def _circulant(case, kernel, spectra, J, adjoint=False):
    """N or K (or its adjoint) on J (C, n1, n2, n3)."""
    n, m = _dims(case), [2 * v for v in _dims(case)]
    F = [torch.fft.fftn(J[c], s=m) for c in range(J.shape[0])]
    Y = [torch.zeros_like(F[0]) for _ in F]
    for p, q, blk, s in _entries(case, kernel, adjoint):
        G = spectra[blk]
        Y[p] += s * (G.conj() if adjoint else G) * F[q]
    return torch.stack([torch.fft.ifftn(y)[: n[0], : n[1], : n[2]] for y in Y])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "assemble"):
        return None   # a solve stops at its tolerance; the near zone is a cubature of its own
    n, C, res = _dims(case), _ql(case), case["res"]
    idx, Mr = _body(case)
    if kind == "loops":
        origin, loops = _loops(case, seed)
        return _loop_moments(case, origin, loops, idx).reshape(-1)
    at = torch.from_numpy(idx).cuda()
    gram = torch.tensor([res ** 3] + ([res ** 3 / 12] * 3 if case["pwl"] else []), dtype=torch.float64, device="cuda").repeat(3)[:, None]
    mr = torch.from_numpy(Mr.reshape(-1, order="F")[idx]).cuda()
    chi = (1 - 1 / mr)[None, :]

    def on_grid(v):
        J = torch.zeros((C, n[2] * n[1] * n[0]), dtype=torch.complex128, device="cuda")
        J[:, at] = v
        return J.reshape(C, n[2], n[1], n[0]).permute(0, 3, 2, 1)

    def on_body(J):
        return J.permute(0, 3, 2, 1).reshape(C, -1)[:, at]

    N = _spectra(case, "N")
    K = _spectra(case, "K") if kind == "fields" else None
    rows = lambda v: v.to(torch.complex128).reshape(case["nrhs"], C, -1)  # noqa: E731
    x = rows(_vector(case, int(np.prod(n)) if kind == "grid" else len(idx), seed))
    if kind == "fields":
        Ue, Ub = (rows(_vector(case, len(idx), seed + k)) for k in (1001, 2003))
        E = [Ue[r] + (on_body(_circulant(case, "N", N, on_grid(x[r]))) / gram - x[r]) / _ce(case["freq"]) for r in range(case["nrhs"])]
        H = [Ub[r] + on_body(_circulant(case, "K", K, on_grid(x[r]))) / gram for r in range(case["nrhs"])]
        return torch.cat([e.reshape(-1) for e in E]), torch.cat([h.reshape(-1) for h in H])
    out = []
    for r in range(case["nrhs"]):
        if kind == "apply":
            out.append(x[r] - chi * on_body(_circulant(case, "N", N, on_grid(x[r]))) / gram)
        elif kind == "adjoint":
            out.append(x[r] - on_body(_circulant(case, "N", N, on_grid(chi.conj() * x[r] / gram), adjoint=True)))
        else:
            J = x[r].reshape(C, n[2], n[1], n[0]).permute(0, 3, 2, 1)
            out.append(_circulant(case, "N", N, J).permute(0, 3, 2, 1).reshape(C, -1))
    return torch.cat([o.reshape(-1) for o in out])

"""Rounding of the coil-loop kernel: its error against the same sums in extended
precision is no larger than that of the plain FP64 evaluation, point by point
(sqrt, division, sin and cos of numpy), over all moments and over the constant ones
with a factor of two: a voxel's 27 points are summed for each segment here, where
the plain form averages their rounding.  Voxel edge and radius are powers of two
and the normal is an axis, so both sides start from the same coordinates.  One voxel
size on each side of the short phase series."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _field(dt, at, res, segs, k0, wmu):
    """(voxels, 3, 4) moments of the field of segments (mid, dl), in dtype dt."""
    one = dt(1)
    q = np.float64(np.sqrt(np.longdouble(3) / 5))
    x = np.array([-q, 0.0, q]).astype(dt)
    w = np.array([5 / 9, 8 / 9, 5 / 9]).astype(dt)
    out = np.zeros((len(at), 3, 4, 2), dt)
    for a in range(27):
        i = (a % 3, a // 3 % 3, a // 9)
        wt = w[i[0]] * w[i[1]] * w[i[2]] / 8
        p = at.astype(dt) + np.array([x[j] for j in i]) * dt(res) / 2
        E = np.zeros((len(at), 3, 2), dt)
        for mid, dl in segs:
            d = p - mid.astype(dt)
            R = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
            ph = dt(k0) * R
            g = one / (4 * dt(math.pi) * R) if dt is np.float64 else one / (4 * np.arccos(-one) * R)
            E[..., 0] += (np.cos(ph) * g)[:, None] * dl.astype(dt)
            E[..., 1] -= (np.sin(ph) * g)[:, None] * dl.astype(dt)
        for m in range(4):
            f = wt * (one if m == 0 else 12 * x[i[m - 1]] / 2) * dt(wmu)
            out[:, :, m, 0] += f * E[..., 1]
            out[:, :, m, 1] -= f * E[..., 0]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("res,freq", [(2.0 ** -7, 128e6), (2.0 ** -6, 297.2e6)])
def test_no_worse_than_plain_fp64(res, freq):
    from marie_gb300 import VieOperator, phantoms
    n, nseg, radius = 24, 64, 2.0 ** -5
    body = phantoms.sphere(n, res, 0.45 * n * res, 30.0, 0.5)
    assert np.array_equal(body.origin, np.full(3, -0.5 * res * (n - 1)))
    op = VieOperator(body.n, res, freq, body.idx_solution(True), body.Mr(freq), np.zeros((n, n, n, 10, 6), complex), pwl=True,
                     precisions=2)
    c = 0.5 * res * n + 0.0625
    loops = np.array([[c, 0.25 * res, 0.125, 1.0, 0.0, 0.0], [-c, -0.0625, 0.0, -1.0, 0.0, 0.0]])
    got = op.incident_loops(body.origin, loops, radius, nseg=nseg).cpu().numpy().reshape(2, 3, 4, -1)
    pick = np.random.default_rng(3).choice(op.Ns, 150, replace=False)
    lin = body.idxS[pick]
    at = body.origin + res * np.stack([lin % n, lin // n % n, lin // (n * n)], 1).astype(np.float64)
    k0 = 2 * math.pi / (299792458.0 / freq)
    wmu = 2 * math.pi * freq * (4e-7 * math.pi)
    err, ref = {}, []
    for l, L in enumerate(loops):
        e1, e2 = (np.array([0.0, 0.0, L[3]]), np.array([0.0, -1.0, 0.0]))     # n x y, n x e1 for n = +-x
        pts = [L[:3] + radius * (math.cos(t) * e1 + math.sin(t) * e2) for t in (2 * math.pi * i / nseg for i in range(nseg + 1))]
        segs = [(0.5 * (a + b), b - a) for a, b in zip(pts, pts[1:])]
        ref.append(_field(np.longdouble, at, res, segs, k0, wmu))
        plain = _field(np.float64, at, res, segs, k0, wmu)
        mine = np.stack([got[l].real, got[l].imag], -1)[..., pick, :].transpose(2, 0, 1, 3)
        for name, v in (("plain", plain), ("gpu", mine)):
            err.setdefault(name, []).append(v.astype(np.longdouble) - ref[-1])
    ref = np.stack(ref)
    rel = {k: (float(np.linalg.norm(np.float64(np.stack(v)))) / float(np.linalg.norm(np.float64(ref))),
               float(np.linalg.norm(np.float64(np.stack(v)[:, :, :, 0]))) / float(np.linalg.norm(np.float64(ref[:, :, :, 0]))))
           for k, v in err.items()}
    print(rel)
    assert rel["gpu"][0] <= rel["plain"][0] and rel["gpu"][1] <= 2 * rel["plain"][1], rel
    op.close()


@pytest.mark.gpu
@pytest.mark.parametrize("res,freq", [(2.0 ** -7, 128e6), (2.0 ** -6, 297.2e6)])
def test_segment_through_a_voxel_centre(res, freq):
    """The first segment's mid-point 1e-9 voxels from a voxel's centre: the linear
    moments, in which the centre point has no weight, stay those of plain sums (a few
    hundred units of 2^-53 of the voxel's largest, for the cancellation of the dl)."""
    from marie_gb300 import VieOperator, phantoms
    n, nseg, radius = 16, 64, 2.0 ** -5
    body = phantoms.sphere(n, res, 0.45 * n * res, 30.0, 0.5)
    op = VieOperator(body.n, res, freq, body.idx_solution(True), body.Mr(freq), np.zeros((n, n, n, 10, 6), complex), pwl=True,
                     precisions=2)
    lin = int(body.idxS[op.Ns // 2])
    at = body.origin + res * np.array([[lin % n, lin // n % n, lin // (n * n)]], np.float64)
    e1, e2 = np.array([0.0, 0.0, 1.0]), np.array([0.0, -1.0, 0.0])     # normal +x
    mid = 0.5 * radius * ((1 + math.cos(2 * math.pi / nseg)) * e1 + math.sin(2 * math.pi / nseg) * e2)
    L = at[0] - mid + 1e-9 * res * np.array([1.0, 0.0, 0.0])
    got = op.incident_loops(body.origin, np.concatenate([L, [1.0, 0.0, 0.0]])[None], radius, nseg=nseg).cpu().numpy()
    got = got.reshape(3, 4, -1)[..., op.Ns // 2]
    pts = [L + radius * (math.cos(t) * e1 + math.sin(t) * e2) for t in (2 * math.pi * i / nseg for i in range(nseg + 1))]
    k0 = 2 * math.pi / (299792458.0 / freq)
    ref = _field(np.longdouble, at, res, [(0.5 * (a + b), b - a) for a, b in zip(pts, pts[1:])], k0,
                 2 * math.pi * freq * (4e-7 * math.pi))[0]
    want = np.float64(ref[..., 0]) + 1j * np.float64(ref[..., 1])
    assert np.isfinite(got).all()
    err = np.abs(got - want)[:, 1:].max() / np.abs(want[:, 1:]).max()
    assert err < 1e-13, err
    op.close()

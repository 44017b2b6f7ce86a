"""Rounding of the Green's-tensor assembly: far-zone offsets against the same
four-point Gauss sums in extended precision (nodes and weights rounded to FP64 on
both sides).  The sums over all 4096 point pairs of an offset give 2.4e-16 of an
offset's values in the 2-norm, mostly the rounding of the kernel values and of
(res/2)^6; the kernel sums 729 distinct differences and has to stay within that,
2.4e-16 = 2.2 units of 2^-53."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

L = [0, 1, 2, 3, 0, 0, 0, 1, 1, 2]
LP = [0, 1, 2, 3, 1, 2, 3, 2, 3, 3]


def _rule():
    """Four-point Gauss rule in extended precision, rounded to FP64."""
    q = np.longdouble
    r = q(2) * np.sqrt(q(6) / 5) / 7
    x = [np.sqrt(q(3) / 7 - r), np.sqrt(q(3) / 7 + r)]
    w = [(18 + np.sqrt(q(30))) / 36, (18 - np.sqrt(q(30))) / 36]
    return (np.array([-x[1], -x[0], x[0], x[1]]).astype(np.float64).astype(q),
            np.array([w[1], w[0], w[0], w[1]]).astype(np.float64).astype(q))


def _sum(m, res, k0):
    q = np.longdouble
    x, w = _rule()
    g = np.stack(np.meshgrid(x, x, x, indexing="ij"), -1).reshape(-1, 3)
    wg = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1)
    h = q(res) / 2
    d = np.asarray(m).astype(q) * q(res) + h * (g[:, None, :] - g[None, :, :])
    R = np.sqrt((d * d).sum(-1))
    k = q(k0)
    pi4 = 4 * np.arccos(q(-1))
    gx, gy = np.cos(k * R) / pi4, -np.sin(k * R) / pi4

    def dd(a, b):
        u, v = d[..., a] * d[..., b] * (3 / R ** 5 - k * k / R ** 3), d[..., a] * d[..., b] * 3 * k / R ** 4
        if a == b:
            u, v = u - 1 / R ** 3, v - k / R ** 2
        return np.stack([gx * u - gy * v, gx * v + gy * u], -1)
    xx, yy, zz = dd(0, 0), dd(1, 1), dd(2, 2)
    f = [-yy - zz, dd(0, 1), dd(0, 2), -xx - zz, dd(1, 2), -xx - yy]
    T = np.concatenate([np.ones((len(g), 1), q), g / 2], 1)
    W = wg[:, None] * wg[None, :] * h ** 6
    return np.array([[(W * T[:, None, L[j]] * T[None, :, LP[j]])[..., None] * fc for fc in f] for j in range(10)]).sum((2, 3))


@pytest.mark.gpu
@pytest.mark.parametrize("res,freq", [(2e-3, 297.2e6), (5e-3, 128e6)])
def test_far_zone(res, freq):
    from marie_gb300 import assemble_green
    n = (40, 36, 33)
    iv = assemble_green(n, res, freq, True, "N")
    k0 = 2 * math.pi / (299792458.0 / freq)
    rng = np.random.default_rng(8)
    err = []
    while len(err) < 24:
        m = tuple(int(v) for v in rng.integers(0, n))
        if max(m) < 8:
            continue
        want = _sum(m, res, k0)
        got = np.stack([iv[m].real, iv[m].imag], -1).astype(np.longdouble)
        err.append(float(np.linalg.norm(np.float64(got - want)) / np.linalg.norm(np.float64(want))))
    rms = float(np.sqrt(np.mean(np.square(err))))
    print(rms)
    assert rms <= 2.4e-16

"""The Green's-tensor assembly kernel at the edges of its rules: offsets of the
medium (8 points per axis) and far (4 points) zones of grids with unequal
edges, where an offset's values come from a permuted one, against the plain
six-dimensional Gauss sum in numpy.  Tolerance: both sides sum up to 2.6e5
FP64 terms whose magnitudes add up to at most a few times the largest entry,
so 1e-12 of it leaves a factor of ten over 2.6e5 * 1.1e-16 / sqrt(...)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

L = [0, 1, 2, 3, 0, 0, 0, 1, 1, 2]
LP = [0, 1, 2, 3, 1, 2, 3, 2, 3, 3]


def gauss_sum(m, n, res, k0, pwl, kernel):
    x, w = np.polynomial.legendre.leggauss(n)
    g = np.stack(np.meshgrid(x, x, x, indexing="ij"), -1).reshape(-1, 3)
    wg = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1)
    h = res / 2
    d = np.asarray(m) * res + h * (g[:, None, :] - g[None, :, :])
    R = np.sqrt((d ** 2).sum(-1))
    Ge = np.exp(-1j * k0 * R) / (4 * np.pi)
    dd = lambda p, q: Ge * (d[..., p] * d[..., q] * (3 / R ** 5 + 3j * k0 / R ** 4 - k0 ** 2 / R ** 3)  # noqa: E731
                            - (p == q) * (1 / R ** 3 + 1j * k0 / R ** 2))
    if kernel == "N":
        xx, yy, zz = dd(0, 0), dd(1, 1), dd(2, 2)
        f = [-yy - zz, dd(0, 1), dd(0, 2), -xx - zz, dd(1, 2), -xx - yy]
    else:
        f = [-d[..., p] * Ge * (1 / R ** 3 + 1j * k0 / R ** 2) for p in range(3)]
    T = np.concatenate([np.ones((len(g), 1)), g / 2], 1)
    W = wg[:, None] * wg[None, :] * h ** 6
    return np.array([[(W * T[:, None, L[j]] * T[None, :, LP[j]] * fc).sum() for fc in f] for j in range(10 if pwl else 1)])


@pytest.mark.gpu
@pytest.mark.parametrize("pwl,kernel", [(False, "N"), (True, "N"), (True, "K")], ids=["pwc-N", "pwl-N", "pwl-K"])
@pytest.mark.parametrize("n", [(6, 9, 11), (10, 6, 6), (6, 6, 6)], ids=str)
def test_rules_and_permutations(n, pwl, kernel):
    from marie_gb300 import assemble_green
    res, freq = 2e-3, 297.2e6
    k0 = 2 * np.pi * freq / 299792458.0
    iv = assemble_green(n, res, freq, pwl, kernel)
    rng = np.random.default_rng(sum(n))
    offs = {(2, 0, 0), (0, 2, 1), (1, 1, 2), (3, 3, 3), tuple(v - 1 for v in n)} | {tuple(rng.integers(0, n)) for _ in range(4)}
    for m in offs:
        if max(m) < 2:
            continue
        want = gauss_sum(m, 8 if max(m) < 8 else 4, res, k0, pwl, kernel)
        assert np.abs(iv[m] - want).max() <= 1e-12 * np.abs(iv[2, 0, 0]).max(), m

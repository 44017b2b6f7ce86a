"""1/sqrt, sqrt, sin and cos of the FP64 Green's-function kernels over their whole
ranges and on both sides of each switch (1e-30 and 1e30; 1e4), against numpy in
extended precision.

Bounds, u = 2^-53, relative for the roots and absolute for sin and cos (whose
results are at most one).  1/sqrt: x*y of the Newton step rounds by u, which half
goes into the result, and the last FMA rounds by u: 1.5 u; sqrt: that and one more
rounding, 2.5 u; a tenth for the FP32 estimate's cube and the products beside them.
sin, cos: the reduced argument rounds twice (2 u), the polynomial's first left-out
term is below 5e-17 = 0.45 u, its steps round by u in the last and a third of that
in the one before: 4 u; of the short series 1.5 u."""
import ctypes as ct
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")
U = 2.0 ** -53
HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = tmp_path_factory.mktemp("fp64math") / "probe.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    str(HERE / "fp64math_probe.cu"), "-o", str(so)], check=True)
    lib = ct.CDLL(str(so))

    def run(what, x):
        x = np.ascontiguousarray(x, np.float64)
        a, b = np.empty_like(x), np.empty_like(x)
        p = lambda v: v.ctypes.data_as(ct.POINTER(ct.c_double))
        assert lib.fp64math_probe(what, p(x), p(a), p(b), x.size) == 0
        return a, b
    return run


@pytest.mark.gpu
def test_inverse_and_square_root(probe):
    rng = np.random.default_rng(1)
    near = [np.nextafter(v, d) for v in (1e-30, 1e30, 1.0, 4.0, 2.0 ** -60) for d in (0.0, np.inf)]
    edge = np.concatenate([v * (1 + np.linspace(-1e-5, 1e-5, 401)) for v in (1e-30, 1e30)])
    x = np.concatenate([10.0 ** rng.uniform(-29.9, 29.9, 200000), 1 + rng.uniform(0, 3, 100000), 10.0 ** rng.uniform(-300, 300, 4000),
                        edge, near])
    r, s = probe(0, x)
    xl = x.astype(np.longdouble)
    root = np.sqrt(xl)
    assert float(np.max(np.abs(s / root - 1))) <= 2.6 * U
    assert float(np.max(np.abs(r * root - 1))) <= 1.6 * U
    far = (x < 0.9e-30) | (x > 1.1e30)          # the library's, correctly rounded
    assert np.array_equal(s[far], np.sqrt(x[far]))
    r, s = probe(0, [0.0, np.inf, np.nan, -1.0])
    assert r[0] == np.inf and s[0] == 0 and r[1] == 0 and s[1] == np.inf and np.isnan(r[2:]).all() and np.isnan(s[2:]).all()


@pytest.mark.gpu
def test_sine_and_cosine(probe):
    rng = np.random.default_rng(2)
    k = np.arange(1, 6367)
    x = np.concatenate([rng.uniform(-1e4, 1e4, 200000), rng.uniform(-10, 10, 200000), 10.0 ** rng.uniform(-20, 0, 20000),
                        k * (np.pi / 2), k * (np.pi / 4), np.nextafter(k * (np.pi / 4), np.inf),
                        1e4 * (1 + np.linspace(-1e-3, 1e-3, 2001)), [0.0, -0.0]])
    sn, cs = probe(1, x)
    xl = x.astype(np.longdouble)
    assert float(np.max(np.abs(sn - np.sin(xl)))) <= 4 * U
    assert float(np.max(np.abs(cs - np.cos(xl)))) <= 4 * U
    sn, cs = probe(1, [np.inf, np.nan])
    assert np.isnan(sn).all() and np.isnan(cs).all()


@pytest.mark.gpu
def test_short_series(probe):
    x = np.concatenate([np.linspace(-0.05, 0.05, 200001), 10.0 ** np.random.default_rng(3).uniform(-20, -1.31, 20000)])
    sn, cs = probe(2, x)
    xl = x.astype(np.longdouble)
    assert float(np.max(np.abs(sn - np.sin(xl)))) <= 1.5 * U
    assert float(np.max(np.abs(cs - np.cos(xl)))) <= 1.5 * U

"""Which grids' complex64 transforms are padded to multiples of 16 (embed.h,
pad_dims): the rule is one of the grid and the basis alone, and grids on both sides
of each of its lines as they were measured."""
import ctypes as ct
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
I3 = ct.c_int * 3


@pytest.fixture(scope="module")
def pad(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("pad") / "libpad_shim.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(HERE / "pad_shim.cpp")], check=True)
    lib = ct.CDLL(str(so))

    def run(n, pwl):
        m = I3()
        return bool(lib.shim_pad_dims(I3(*n), 12 if pwl else 3, m)), tuple(m)
    return run


PADDED = [((60, 77, 90), False), ((60, 77, 90), True), ((100, 100, 100), True), ((24, 24, 24), True), ((24, 24, 20), True),
          ((20, 40, 40), False), ((96, 96, 6), False), ((64, 64, 8), True), ((34, 34, 34), False), ((11, 30, 30), False),
          ((22, 22, 30), False), ((127, 128, 128), True), ((13, 30, 45), False), ((20, 24, 24), True),
          ((18, 20, 32), False), ((16, 16, 12), False), ((32, 32, 6), False)]
OWN = [((64, 64, 64), True), ((16, 32, 128), False), ((8, 64, 64), False), ((8, 64, 64), True), ((6, 96, 96), True),
       ((16, 8, 16), False), ((16, 16, 8), False), ((17, 17, 17), True), ((18, 18, 18), False), ((20, 20, 20), True),
       ((129, 64, 64), False), ((144, 150, 150), True), ((10, 10, 10), False), ((16, 16, 5), True)]


@pytest.mark.parametrize("n,pwl", PADDED, ids=str)
def test_padded(pad, n, pwl):
    yes, m = pad(n, pwl)
    assert yes and m == tuple(-(-v // 16) * 16 for v in n)


@pytest.mark.parametrize("n,pwl", OWN, ids=str)
def test_own_lengths(pad, n, pwl):
    assert not pad(n, pwl)[0]

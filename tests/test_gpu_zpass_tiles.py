"""complex64 four-step passes over the ways a tile is filled: bundles of one to
sixteen right-hand sides (mirrored columns inside the tile or as tiles of their
own), odd counts that leave lanes of a bundle empty, every z-tile width, short
and long axes (tiles of 8 to 128 elements in the x and y passes), N, its adjoint
and both operators' body forms, against the generic mixed-radix passes on the
same handle.  Tolerance: 1e-5 of the 2-norm, the complex64 parity bound of the
matvec tests (both paths round at about 2e-7)."""
import numpy as np
import pytest

from helpers import Problem, rel_err

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("n", [(16, 48, 32), (32, 16, 80), (64, 32, 48)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("width", [0, 1, 2, 4, 8], ids=lambda w: f"w{w}")
def test_tiles_and_bundles(n, pwl, width, monkeypatch):
    if width:
        monkeypatch.setenv("MARIE_Z_TILE", str(width))
    P = Problem(n, pwl, seed=3 + pwl)
    op = P.gpu_operator(precisions=2, max_rhs=17, dense=True)
    gen = torch.Generator(device="cuda").manual_seed(5)
    for nrhs in (1, 2, 3, 7, 16, 17):
        x = torch.randn(nrhs * op.Nb, dtype=torch.complex64, device="cuda", generator=gen)
        g = torch.randn(2 * op.C * op.nD, dtype=torch.complex64, device="cuda", generator=gen) if nrhs == 2 else None
        for fn, v in ((op.apply, x), (op.apply_adjoint, x), (op.apply_N, g), (op.apply_N_adj, g)):
            if v is None:
                continue
            y = fn(v).cpu().numpy()
            monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
            want = fn(v).cpu().numpy()
            monkeypatch.delenv("MARIE_GENERIC_FFT")
            assert rel_err(y.astype(np.complex128), want.astype(np.complex128)) <= 1e-5, (fn.__name__, nrhs)
    op.close()

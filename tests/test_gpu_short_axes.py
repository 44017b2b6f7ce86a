"""complex64 four-step passes on short z edges: z tiles narrower than the widest, PWC
tiles of n3 = 16 in CTAs of their own size, y tiles that begin inside a column (ragged
edges beside 16) or take several, bundles wider than the right-hand sides they hold;
N, its adjoint, K and the body forms against the mixed-radix passes of the same
handle or, on padded grids, of one made for them.  Tolerance: 1e-5 of the 2-norm, the
complex64 parity bound of the matvec tests."""
import numpy as np
import pytest

from helpers import Problem, rel_err

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("n", [(16, 16, 16), (64, 16, 16), (16, 48, 16), (96, 16, 16), (16, 16, 12), (30, 16, 13), (48, 32, 15),
                               (16, 32, 27), (31, 15, 33)], ids=lambda n: "x".join(map(str, n)))
def test_short_axes(n, pwl, monkeypatch):
    P = Problem(n, pwl, seed=7 + pwl, box=((0, n[0]), (1, n[1]), (2, n[2] - 1)))
    op = P.gpu_operator(precisions=2, max_rhs=16, dense=True)
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    ref = P.gpu_operator(precisions=2, max_rhs=16, dense=True)
    gen = torch.Generator(device="cuda").manual_seed(5)
    for nrhs in (1, 2, 3, 5, 7, 8, 11, 16):
        x = torch.randn(nrhs * op.Nb, dtype=torch.complex64, device="cuda", generator=gen)
        calls = [("apply", x), ("apply_adjoint", x)]
        if nrhs in (1, 3):
            g = torch.randn(nrhs * op.C * op.nD, dtype=torch.complex64, device="cuda", generator=gen)
            calls += [("apply_N", g), ("apply_K", g), ("apply_K_adj", g)]
        for name, v in calls:
            monkeypatch.delenv("MARIE_GENERIC_FFT", raising=False)
            y = getattr(op, name)(v).cpu().numpy()
            monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
            want = getattr(ref, name)(v).cpu().numpy()
            assert rel_err(y.astype(np.complex128), want.astype(np.complex128)) <= 1e-5, (name, nrhs)
    op.close()
    ref.close()

"""complex64 grids whose edges are no multiples of 16 run the four-step passes on
padded transform lengths, and K / K^H run them as N does: every operator and
field form on such grids (edges just above and just below multiples of 16, one
multiple among them, a partial body, operands dense and as Tucker blocks) against
the generic passes on the grid's own lengths (a handle made under
MARIE_GENERIC_FFT), and K on a 16*NB grid against the generic passes of the same
handle.  Tolerance: 1e-5 of the 2-norm, the complex64 parity bound of the matvec
tests."""
import numpy as np
import pytest

from helpers import Problem, rel_err

torch = pytest.importorskip("torch")


def _forms(op, gen, nrhs=3):
    c = dict(dtype=torch.complex64, device="cuda", generator=gen)
    x = torch.randn(nrhs * op.Nb, **c)
    u = torch.randn(nrhs * op.Nb, **c)
    g = torch.randn(2 * op.C * op.nD, **c)
    for fn, v in ((op.apply, x), (op.apply_adjoint, x), (op.apply_hfield_adjoint, x), (op.apply_N, g), (op.apply_N_adj, g),
                  (op.apply_K, g), (op.apply_K_adj, g)):
        yield fn.__name__, fn(v)
    E, H = op.fields(x, u, x)
    yield "E", E
    yield "H", H


def _compare(got, want):
    for (name, a), (_, b) in zip(got, want):
        assert rel_err(a.cpu().numpy().astype(np.complex128), b.cpu().numpy().astype(np.complex128)) <= 1e-5, name


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("n,dense", [((15, 33, 30), True), ((20, 16, 27), False), ((31, 14, 48), True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else ("dense" if v else "tucker"))
def test_padded_grid(n, dense, pwl, monkeypatch):
    P = Problem(n, pwl, seed=9 + pwl, box=tuple((1, m - 1) for m in n))
    op = P.gpu_operator(precisions=2, dense=dense)
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    ref = P.gpu_operator(precisions=2, dense=dense)
    monkeypatch.delenv("MARIE_GENERIC_FFT")
    gens = [torch.Generator(device="cuda").manual_seed(2) for _ in range(2)]
    _compare(list(_forms(op, gens[0])), list(_forms(ref, gens[1])))
    op.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("n", [(32, 16, 48), (16, 32, 112)], ids=lambda n: "x".join(map(str, n)))
def test_k_on_the_four_step_path(n, pwl, monkeypatch):
    P = Problem(n, pwl, seed=4 + pwl)
    op = P.gpu_operator(precisions=2, dense=True)
    gens = [torch.Generator(device="cuda").manual_seed(3) for _ in range(2)]
    got = list(_forms(op, gens[0]))
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    _compare(got, list(_forms(op, gens[1])))
    op.close()

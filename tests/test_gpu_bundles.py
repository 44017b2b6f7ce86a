"""Batches of every size from 2 to 17 (bundles of 1, 2, 4, 8 and 16 right-hand sides,
with and without empty places, more than a chunk) on four-step, padded and
mixed-radix grids: each product against the same vector's product alone.  The
arithmetic of a right-hand side does not depend on its bundle but for the order in
which the compiler contracts it, so they agree within a few roundings of the
result: 1e-6 in complex64, 1e-13 in float-float, 1e-14 in complex128."""
import numpy as np
import pytest

from helpers import Problem

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n,pwl,precisions,tol", [((16, 32, 16), False, 2, 1e-6), ((17, 12, 20), True, 2, 1e-6),
                                                  ((16, 16, 32), True, 4, 1e-13), ((7, 6, 10), True, 1, 1e-14)])
def test_batches_equal_single(n, pwl, precisions, tol):
    P = Problem(n, pwl, seed=3)
    op = P.gpu_operator(precisions=precisions, max_rhs=16)
    dt = torch.complex64 if precisions == 2 else torch.complex128
    X = torch.from_numpy(P.random_body_vec(seed=6, nrhs=17)).to("cuda", dt)
    single = torch.stack([op.apply(X[r].contiguous()) for r in range(17)])
    adj = torch.stack([op.apply_adjoint(X[r].contiguous()) for r in range(17)])
    for nrhs in range(2, 18):
        for f, want in ((op.apply, single), (op.apply_adjoint, adj)):
            y = f(X[:nrhs].reshape(-1)).reshape(nrhs, -1)
            d = (y - want[:nrhs]).norm(dim=1) / want[:nrhs].norm(dim=1)
            assert float(d.max()) <= tol, nrhs
    op.close()


@pytest.mark.gpu
def test_chunks_of_large_grids():
    """A grid whose odd counts go in several chunks (three as two and one, seven as
    four, two and one)."""
    from marie_gb300 import VieOperator, assemble_green, phantoms
    n, res, freq = 112, 2e-3, 3e8
    body = phantoms.sphere(n, res, 0.3 * n * res, 50.0, 0.6)
    iv = assemble_green(body.n, res, freq, False, "N")
    op = VieOperator(body.n, res, freq, body.idx_solution(False), body.Mr(freq), iv, pwl=False, precisions=2, max_rhs=8)
    rng = np.random.default_rng(1)
    X = torch.from_numpy(rng.normal(size=(7, op.Nb)) + 1j * rng.normal(size=(7, op.Nb))).to("cuda", torch.complex64)
    for f in (op.apply, op.apply_adjoint):
        want = torch.stack([f(X[r].contiguous()) for r in range(7)])
        for nrhs in (3, 7):
            y = f(X[:nrhs].reshape(-1)).reshape(nrhs, -1)
            assert float(((y - want[:nrhs]).norm(dim=1) / want[:nrhs].norm(dim=1)).max()) <= 1e-6
    op.close()

"""GMRES vector kernels on both sides of the short-vector rule (131072 unknowns)
and with cycles of less than a warp of rows, more than one, and the most the
solver keeps: the residual that the recurrence reports against b - A x computed
afterwards, and each solution of a batch against its solve alone, bit for bit.
The recurrence is FP64 throughout and the operator's condition number is of order
ten, so the two residuals differ by rounding, a few hundred products of 1e-16
each: 1e-12 of b at the most."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n,pwl,restart,tol", [(9, False, 5, 1e-8), (9, True, 33, 1e-10), (10, False, 128, 1e-11),
                                               (32, True, 20, 1e-6), (34, True, 40, 1e-6)])
def test_short_and_long_vectors(n, pwl, restart, tol):
    from marie_gb300 import VieOperator, assemble_green, phantoms
    res, freq = 1e-2, 1e8
    body = phantoms.sphere(n, res, 0.42 * n * res, 10.0, 0.1)
    iv = assemble_green(body.n, res, freq, pwl, "N")
    op = VieOperator(body.n, res, freq, body.idx_solution(pwl), body.Mr(freq), iv, pwl=pwl, precisions=1, max_rhs=2)
    assert (op.Nb > 131072) == (n == 34)
    rng = np.random.default_rng(n)
    b = torch.from_numpy(rng.normal(size=(2, op.Nb)) + 1j * rng.normal(size=(2, op.Nb))).cuda()
    x, rep = op.gmres(b.reshape(-1), restart=restart, tol=tol, maxit=200, mode="fp64")
    assert rep.ok
    r = (b.reshape(-1) - op.apply(x)).reshape(2, -1)
    true = (r.norm(dim=1) / b.norm(dim=1)).cpu().numpy()
    for k in range(2):
        assert true[k] <= tol * 1.01 and abs(true[k] - rep.resvec[k][-1]) <= 1e-12
        xs, _ = op.gmres(b[k].contiguous(), restart=restart, tol=tol, maxit=200, mode="fp64")
        assert torch.equal(xs, x.reshape(2, -1)[k])
    op.close()

"""Block GMRES with up to sixteen right-hand sides (the tall-product kernels of the
block solver) and just above (GEMMs), block widths 4 / 8 / 16 and counts between
them, restarted cycles, a row count that is no multiple of a warp: each solution
against the complex128 GMRES of the same handle.  Both are converged to 1e-8
relative residual or better, and a sphere of eps_r = 10 gives an operator of a
condition number of order ten, so they agree within 1e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _case(n, pwl, nrhs):
    from marie_gb300 import VieOperator, assemble_green, phantoms
    res, freq = 1e-2, 1e8
    body = phantoms.sphere(n, res, 0.42 * n * res, 10.0, 0.1)
    iv = assemble_green(body.n, res, freq, pwl, "N")
    op = VieOperator(body.n, res, freq, body.idx_solution(pwl), body.Mr(freq), iv, pwl=pwl, precisions=3, max_rhs=nrhs)
    rng = np.random.default_rng(4)
    b = rng.normal(size=(nrhs, op.Nb)) + 1j * rng.normal(size=(nrhs, op.Nb))
    return op, torch.from_numpy(b.reshape(-1)).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("nrhs,steps", [(1, 30), (3, 7), (5, 30), (8, 5), (13, 30), (16, 4), (17, 30)])
def test_block_widths(pwl, nrhs, steps):
    op, b = _case(9, pwl, nrhs)
    x, rep = op.gmres(b, tol=1e-8, mode="block", block_steps=steps)
    want, _ = op.gmres(b, tol=1e-10, mode="fp64")
    assert rep.ok and np.all(rep.true_resid <= 1e-8)
    d = (x - want).reshape(nrhs, -1)
    assert float((d.norm(dim=1) / want.reshape(nrhs, -1).norm(dim=1)).max()) <= 1e-6
    op.close()


@pytest.mark.gpu
def test_non_finite_operator_output_is_reported():
    op, b = _case(6, False, 2)
    b[3] = float("nan")
    with pytest.raises(Exception, match="finite"):
        op.gmres(b, tol=1e-8, mode="block")
    op.close()

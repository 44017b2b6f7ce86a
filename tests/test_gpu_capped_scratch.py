"""GMRES and block GMRES on a handle with a memory cap, where the solvers keep to
their smallest partial sums: the solutions of an uncapped handle, both converged to
1e-8 on an operator of condition number about ten (1e-6 between them)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["fp64", "block"])
@pytest.mark.parametrize("nrhs", [1, 8])
def test_capped_equals_uncapped(mode, nrhs):
    from marie_gb300 import VieOperator, assemble_green, phantoms
    n, res, freq = 16, 1e-2, 1e8
    body = phantoms.sphere(n, res, 0.42 * n * res, 10.0, 0.1)
    iv = assemble_green(body.n, res, freq, True, "N")
    x = []
    for cap in (0, 1 << 30):
        op = VieOperator(body.n, res, freq, body.idx_solution(True), body.Mr(freq), iv, pwl=True, precisions=3,
                         max_rhs=nrhs, mem_cap_bytes=cap)
        rng = np.random.default_rng(5)
        b = torch.from_numpy(rng.normal(size=nrhs * op.Nb) + 1j * rng.normal(size=nrhs * op.Nb)).cuda()
        y, rep = op.gmres(b, tol=1e-8, mode=mode)
        assert rep.ok and np.all(rep.true_resid <= 1.01e-8)
        x.append(y.reshape(nrhs, -1))
        op.close()
    assert float(((x[0] - x[1]).norm(dim=1) / x[0].norm(dim=1)).max()) <= 1e-6

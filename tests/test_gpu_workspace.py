"""Device memory that a complex128 GMRES solve takes on its first call, at the
longest vectors of the short-vector kernels: the Krylov basis, the Hessenberg
matrix and its rotated copy, the partial sums of the projections (one per CTA of
256 unknowns) and a handful of vectors and small arrays, two vectors and 32 MB
here.  The Green's tensor is zero, so the solve ends after one step."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_partial_sums_of_short_vectors():
    from marie_gb300 import VieOperator, phantoms
    n, nrhs, m = 35, 64, 128
    body = phantoms.sphere(n, 1e-2, 10.0, 10.0, 0.1)     # the whole grid
    op = VieOperator(body.n, 1e-2, 1e8, body.idx_solution(False), body.Mr(1e8), np.zeros((n, n, n, 6), complex), pwl=False,
                     precisions=1, max_rhs=nrhs)
    assert 120000 < op.Nb <= 131072
    b = torch.ones(nrhs * op.Nb, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()

    def taken():
        return torch.cuda.mem_get_info()[1] - torch.cuda.mem_get_info()[0] - torch.cuda.memory_reserved()

    before = taken()
    _, rep = op.gmres(b, restart=m, tol=1e-8, maxit=1, mode="fp64")
    assert rep.ok
    basis = nrhs * (m + 1) * op.Nb * 16
    hess = 2 * nrhs * (m + 1) * m * 16
    parts = nrhs * (m + 1) * ((op.Nb + 255) // 256) * 16
    assert taken() - before <= basis + hess + parts + 2 * nrhs * op.Nb * 16 + (32 << 20)
    op.close()

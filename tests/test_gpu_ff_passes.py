"""Float-float passes on every edge 16*NB, NB = 1 .. 8, each axis, with tile widths
from one right-hand side to more than a bundle and bodies that leave rows and
slices empty, against the oracle.  A float-float operation is good to 2^-45; a
product makes six transforms of up to eight binary levels and a sum of twelve
terms, some sixty operations in a row: 60 * 2^-45 = 1.7e-12 at the very worst,
1e-12 in the 2-norm."""
import numpy as np
import pytest

from oracle import marie_oracle as O
from helpers import Problem, flat_F, unflat_F, rel_err

torch = pytest.importorskip("torch")
TOL = 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("n,pwl,nrhs", [((16, 16, 32), True, 1), ((32, 48, 16), True, 3), ((48, 16, 64), False, 5),
                                        ((16, 64, 48), True, 2), ((64, 16, 80), False, 1), ((16, 80, 16), False, 17),
                                        ((80, 16, 96), False, 2), ((16, 96, 16), True, 1), ((96, 16, 112), False, 1),
                                        ((16, 112, 16), False, 3), ((112, 16, 16), True, 1), ((16, 16, 128), True, 1),
                                        ((128, 16, 16), False, 4), ((16, 128, 16), False, 1)])
def test_edges(n, pwl, nrhs):
    P = Problem(n, pwl, seed=n[0] + n[2])
    op = P.gpu_operator(precisions=4, max_rhs=max(4, nrhs))
    assert op.tiles(0)["float_float"]
    J = P.random_grid(seed=8)
    x = torch.from_numpy(flat_F(J[0])).to("cuda", torch.complex128)
    for name, adj, f in (("N", False, op.apply_N), ("N", True, op.apply_N_adj)):
        assert rel_err(unflat_F(f(x).cpu().numpy(), n, P.C), O.mvp_op_tucker(J[0], P.TN, name, adj, cache={})) <= TOL
    X = P.random_body_vec(seed=6, nrhs=nrhs)
    xb = torch.from_numpy(X.reshape(-1)).to("cuda", torch.complex128)
    yb = op.apply(xb).cpu().numpy().reshape(nrhs, -1)
    ya = op.apply_adjoint(xb).cpu().numpy().reshape(nrhs, -1)
    for r in (0, nrhs - 1):
        assert rel_err(yb[r], O.mvp_vie(X[r], P.Mr, P.Mc, P.dims, P.TN, cache={})) <= TOL
        assert rel_err(ya[r], O.mvp_vie_adjoint(X[r], P.Mr, P.Mc, P.dims, P.TN, cache={})) <= TOL
    op.close()

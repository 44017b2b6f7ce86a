"""complex128 PWL on grids of the mixed-radix passes, where the z pass gives each
output group of a frequency to a thread: frequencies fewer than a round of 85,
just over one, no multiple of it, one slice, a prime edge; N, N^H, K and K^H
against the oracle with the native path's 1e-12."""
import numpy as np
import pytest

from oracle import marie_oracle as O
from helpers import Problem, flat_F, unflat_F, rel_err

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n,nrhs", [((3, 2, 1), 1), ((2, 3, 11), 5), ((5, 1, 31), 1), ((2, 5, 30), 3), ((4, 3, 17), 16)])
def test_output_groups(n, nrhs):
    P = Problem(n, True, seed=sum(n))
    op = P.gpu_operator(precisions=1, max_rhs=nrhs)
    J = P.random_grid(seed=2, nrhs=nrhs)
    x = torch.from_numpy(np.concatenate([flat_F(J[r]) for r in range(nrhs)])).to("cuda", torch.complex128)
    for name, adj, f in (("N", False, op.apply_N), ("N", True, op.apply_N_adj), ("K", False, op.apply_K),
                         ("K", True, op.apply_K_adj)):
        y = f(x).cpu().numpy().reshape(nrhs, -1)
        for r in (0, nrhs - 1):
            ref = O.mvp_op_tucker(J[r], P.TN if name == "N" else P.TK, name, adj, cache={})
            assert rel_err(unflat_F(y[r], n, P.C), ref) <= 1e-12
    op.close()

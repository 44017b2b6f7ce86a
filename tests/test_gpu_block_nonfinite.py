"""A finite right-hand side whose block operator output is not finite: one voxel
with a permittivity of 1e-40 has a finite contrast in FP64 and an infinite one in
complex64.  The block solver has to report the operator's output, in each width of
the kernel that checks it while it projects (4, 8, 16 right-hand sides) and above,
where a kernel of its own checks."""
import numpy as np
import pytest

from test_gpu_block_small import _case

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [1, 3, 7, 13, 17])
def test_operator_output_is_checked(nrhs):
    from marie_gb300 import _lib
    op, b = _case(8, False, nrhs)
    mr = np.full(op.Nb // 3, 10.0 - 1j)
    mr[5] = 1e-40
    op.set_materials(mr)
    with pytest.raises(_lib.MarieError, match="non-finite operator output") as ei:
        op.gmres(b, tol=1e-8, mode="block")
    assert ei.value.status == 3
    mr[5] = 10.0
    op.set_materials(mr)
    _, rep = op.gmres(b, tol=1e-8, mode="block")      # the handle is usable afterwards
    assert rep.ok
    op.close()

"""The coil-loop kernel where its steps change: voxels small and large against the
wavelength (the phase of a voxel's points from its centre's, or each its own), far
and near segments, segment counts around its tile of 64, PWC and PWL, against the
oracle's projection in numpy.  Tolerance 1e-12: both sides evaluate the same sums
in FP64, in another order."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_rhs import _centres, _op, _oracle_loops

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("pwl", [False, True], ids=["pwc", "pwl"])
@pytest.mark.parametrize("res,freq,nseg", [(2e-3, 297.2e6, 64), (1.1e-2, 297.2e6, 65), (1.25e-2, 297.2e6, 3), (0.2, 1.2e9, 130),
                                           (1e-3, 1e5, 63)])
def test_loops(res, freq, nseg, pwl):
    from marie_gb300 import phantoms
    n = 9
    body = phantoms.sphere(n, res, 0.45 * n * res, 30.0, 0.5)
    loops = np.array([[0.7 * n * res, 0.1 * res, 0.3 * res, 1.0, 0.2, 0.1], [0.0, 0.0, 5.0 * n * res, 0.0, 0.1, 1.0]])
    op = _op(body, res, freq, pwl, 2)
    got = op.incident_loops(body.origin, loops, 1.5 * res, nseg=nseg).cpu().numpy().reshape(2, -1)
    ref = _oracle_loops(_centres(body, res), res, pwl, loops, 1.5 * res, nseg, freq)
    for l in range(2):
        assert rel_err(got[l], ref[l]) <= 1e-12, l
    op.close()

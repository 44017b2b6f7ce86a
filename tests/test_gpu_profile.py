"""marie_vie_profile over applications that run in several chunks of right-hand
sides: an odd count on a large complex64 grid (powers of two), more right-hand
sides than the work arrays hold, the mixed-radix passes, complex128.  The five
pass times follow each other on one stream, so they add up to the time of the
whole application but for the gaps between launches: a few microseconds of some
hundred a launch, less than a tenth.  A time that leaves a chunk out falls short
by a third (three as two and one) or more; the bound lies between, at a fifth."""
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("n,precisions,max_rhs,nrhs", [(112, 2, 7, 3), (112, 2, 7, 7), (112, 2, 2, 8), (132, 2, 2, 6),
                                                       (48, 1, 2, 6), (64, 4, 2, 5)])
def test_passes_add_up(n, precisions, max_rhs, nrhs):
    from marie_gb300 import VieOperator, assemble_green, phantoms
    res, freq = 2e-3, 3e8
    body = phantoms.sphere(n, res, 0.45 * n * res, 50.0, 0.6)
    iv = assemble_green(body.n, res, freq, False, "N", near="standin")
    op = VieOperator(body.n, res, freq, body.idx_solution(False), body.Mr(freq), iv, pwl=False, precisions=precisions,
                     max_rhs=max_rhs)
    x = torch.randn(nrhs * op.Nb, dtype=torch.complex64 if precisions == 2 else torch.complex128, device="cuda")
    op.profile(x, reps=3)
    ms = op.profile(x, reps=10)
    assert 0.8 * ms[5] <= ms[:5].sum() <= 1.02 * ms[5], ms
    op.close()

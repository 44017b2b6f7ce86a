"""Systematic error of the complex64 four-step products: the moduli of their FP32
twiddles are the same in the transforms and their inverses, and the spectrum is
divided by the gain they make.  On every length 16*NB, N and its adjoint against
complex128 on a random full grid: the mean gain <ref, y - ref> / <ref, ref> is left
with what the rounding of some ten thousand values or more averages to, 1e-7 over the
root of their number, and the positions' gains about their mean (2.5e-8 an axis)
weighted by random data: 5e-9 bounds it (1e-7 to 1.7e-7 where the spectrum does not
carry the gain).  On padded grids the whole error is no larger than that of the
mixed-radix passes on the grid's own lengths, whose twiddles round to other
lengths' moduli; and a Tucker operator expanded per application has the same gain."""
import numpy as np
import pytest

from helpers import Problem, flat_F

torch = pytest.importorskip("torch")


def _pair(P, prec=2, **kw):
    op = P.gpu_operator(precisions=prec, max_rhs=1, **kw)
    ref = P.gpu_operator(precisions=1, max_rhs=1, **kw)
    return op, ref


@pytest.mark.gpu
@pytest.mark.parametrize("n,pwl", [((16, 32, 48), True), ((48, 16, 64), False), ((32, 64, 16), True), ((64, 48, 32), False),
                                   ((80, 16, 96), False), ((16, 96, 80), False), ((96, 80, 16), False), ((112, 16, 128), False),
                                   ((16, 128, 112), False), ((128, 112, 16), False)])
def test_mean_gain(n, pwl):
    P = Problem(n, pwl, seed=sum(n))
    op, ref = _pair(P, dense=True)
    x = torch.from_numpy(flat_F(P.random_grid(seed=1)[0])).to("cuda", torch.complex64)
    for f, g in ((op.apply_N, ref.apply_N), (op.apply_N_adj, ref.apply_N_adj), (op.apply_K, ref.apply_K)):
        want = g(x.to(torch.complex128))
        d = f(x).to(torch.complex128) - want
        gain = float((want.conj() * d).sum().real / want.norm() ** 2)
        assert abs(gain) <= 5e-9, (f.__name__, gain)
    op.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,pwl", [((20, 24, 24), False), ((21, 25, 27), True), ((12, 40, 60), False), ((40, 40, 18), True),
                                   ((50, 52, 54), False)])
def test_padded_error(n, pwl, monkeypatch):
    P = Problem(n, pwl, seed=sum(n), physical=False)
    op, ref = _pair(P, dense=True)
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    own = P.gpu_operator(precisions=2, max_rhs=1, dense=True)
    monkeypatch.delenv("MARIE_GENERIC_FFT")
    x = torch.from_numpy(P.random_body_vec(seed=2)[0]).to("cuda", torch.complex64)
    for name in ("apply", "apply_adjoint"):
        want = getattr(ref, name)(x.to(torch.complex128))
        err = [float((getattr(o, name)(x).to(torch.complex128) - want).norm() / want.norm()) for o in (op, own)]
        assert err[0] <= err[1], (name, err)
    for o in (op, ref, own):
        o.close()


@pytest.mark.gpu
def test_expanded_per_application():
    P = Problem((16, 32, 48), False, seed=2)
    op, ref = _pair(P, prec=2 | 8)
    x = torch.from_numpy(flat_F(P.random_grid(seed=1)[0])).to("cuda", torch.complex64)
    want = ref.apply_N(x.to(torch.complex128))
    d = op.apply_N(x).to(torch.complex128) - want
    # three FP32 mode products and their scale beside the transforms: two units of 2^-24
    assert abs(float((want.conj() * d).sum().real / want.norm() ** 2)) <= 1.2e-7 / 2
    op.close()
    ref.close()

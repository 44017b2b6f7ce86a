"""The passes that a complex64 handle runs follow from its grid and basis, not from
the device memory that happens to be free: a handle whose work arrays would take more
than a quarter of it runs what a small one runs, bit for bit; a handle made under
MARIE_GENERIC_FFT, or with a memory cap, keeps the grid's own lengths, and the switch
set after create leaves a padded handle as it is."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _handle(n, max_rhs, **kw):
    from marie_gb300 import VieOperator, phantoms
    rng = np.random.default_rng(4)
    iv = np.zeros((n, n, n, 6), complex)
    for c in (0, 3, 5):
        iv[:4, :4, :4, c] = rng.normal(size=(4, 4, 4)) * 1e-9
    body = phantoms.sphere(n, 5e-3, 0.45 * n * 5e-3, 40.0, 0.5)
    return VieOperator(body.n, 5e-3, 1e8, body.idx_solution(False), body.Mr(1e8), iv, pwl=False, precisions=2, max_rhs=max_rhs, **kw)


@pytest.mark.gpu
def test_path_does_not_depend_on_free_memory(monkeypatch):
    n = 120
    free = torch.cuda.mem_get_info()[0]
    per = 8 * 3 * n * (2 * 128) * (n + 2 * 128)          # work arrays of a right-hand side
    rhs = int(0.3 * free / per)
    op = _handle(n, 1)
    assert op.tiles()["padded"]
    x = torch.randn(op.Nb, dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    y = op.apply(x)
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    assert torch.equal(op.apply(x), y)
    monkeypatch.delenv("MARIE_GENERIC_FFT")
    op.close()
    monkeypatch.setenv("MARIE_WS_RHS", str(rhs))
    big = _handle(n, rhs)
    assert big.tiles()["padded"] and big.tiles()["chunk"] >= rhs
    assert torch.equal(big.apply(x), y)
    big.close()


@pytest.mark.gpu
def test_own_lengths_on_request(monkeypatch):
    monkeypatch.setenv("MARIE_GENERIC_FFT", "1")
    own = _handle(30, 2)
    monkeypatch.delenv("MARIE_GENERIC_FFT")
    capped = _handle(30, 2, mem_cap_bytes=1 << 32)
    pad = _handle(30, 2)
    assert not own.tiles()["padded"] and not capped.tiles()["padded"] and pad.tiles()["padded"]
    x = torch.randn(2 * own.Nb, dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    a, b, c = own.apply(x), capped.apply(x), pad.apply(x)
    assert torch.equal(a, b) and float((a - c).norm() / a.norm()) <= 1e-5
    for o in (own, capped, pad):
        o.close()

"""Tensor-core products (split-BF16x3) over the widths that change their tiles:
bands of 1 to several tiles, and both accumulation orders.

Bound: an operand is hi + lo with |x - hi - lo| <= 2^-18 |x|, and lo lo' (at most
2^-18 of the product) is left out: 3 2^-18 of |a| |b|; the FP32 sums of the three
products, of 2 K real terms each, add at most 6 K 2^-23; sqrt(2) for a complex
result.  A projection followed by D and the back-projection adds the three
relative errors on the product of the magnitudes, D's own sum of pa included.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WIDTHS = [1, 7, 8, 9, 16, 17, 33, 63, 64, 65, 80, 100, 112, 127, 128, 129, 160, 200]


def _rel(K):
    return np.sqrt(2.0) * (3 * 2.0**-18 + 6 * K * 2.0**-23)


def _rand(rng, *shape):
    t = torch.from_numpy(rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).to(torch.complex64)
    return t.to(DEV), t.numpy().astype(complex)


@pytest.mark.parametrize("nb", WIDTHS)
def test_nonlocal(nb):
    rng = np.random.default_rng(nb)
    nk, atoms, pa, G = 2, 5, 4, 203
    P = atoms * pa
    beta, bh = _rand(rng, nk, P, G)
    D, Dh = _rand(rng, atoms, pa, pa)
    C, Ch = _rand(rng, nk, nb, G)
    HC, Hh = _rand(rng, nk, nb, G)
    projT = torch.empty((nk, nb, P), dtype=torch.complex64, device=DEV)
    ops.apply_nonlocal_tc(ops.beta_split(beta), D, C, HC, projT=projT)
    want = np.einsum("kpg,kbg->kbp", bh.conj(), Ch)
    mag = np.einsum("kpg,kbg->kbp", np.abs(bh), np.abs(Ch))
    assert np.all(np.abs(projT.cpu().numpy() - want) <= _rel(G) * mag)
    Dw = np.einsum("arc,kbac->kbar", Dh, want.reshape(nk, nb, atoms, pa)).reshape(nk, nb, P)
    Dm = np.einsum("arc,kbac->kbar", np.abs(Dh), mag.reshape(nk, nb, atoms, pa)).reshape(nk, nb, P)
    out = Hh + np.einsum("kpg,kbp->kbg", bh, Dw)
    om = np.abs(Hh) + np.einsum("kpg,kbp->kbg", np.abs(bh), Dm)
    assert np.all(np.abs(HC.cpu().numpy() - out) <= (_rel(G) + _rel(pa) + _rel(P)) * om)


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("n_out", WIDTHS)
def test_rotation(n_out, accumulate):
    rng = np.random.default_rng(n_out)
    nk, n_in, G = 2, 37, 301
    C, Ch = _rand(rng, nk, n_in, G)
    M, Mh = _rand(rng, nk, n_in, n_out)
    o, oh = _rand(rng, nk, n_out, G)
    got = ops.matmul(C, M, out=o, accumulate=accumulate, tc=True).cpu().numpy()
    want = np.einsum("kij,kig->kjg", Mh, Ch) + (oh if accumulate else 0.0)
    mag = np.einsum("kij,kig->kjg", np.abs(Mh), np.abs(Ch)) + np.abs(oh)
    assert np.all(np.abs(got - want) <= _rel(n_in + 1) * mag)


@pytest.mark.parametrize("nx,ny", [(1, 1), (9, 33), (64, 65), (65, 64), (129, 100), (40, 200)])
def test_overlap(nx, ny):
    rng = np.random.default_rng(nx)
    nk, G = 2, 259
    X, Xh = _rand(rng, nk, nx, G)
    Y, Yh = _rand(rng, nk, ny, G)
    got = ops.dot(X, Y, tc=True).cpu().numpy()
    want = np.einsum("kig,kjg->kij", Xh.conj(), Yh)
    mag = np.einsum("kig,kjg->kij", np.abs(Xh), np.abs(Yh))
    assert np.all(np.abs(got - want) <= _rel(G) * mag)

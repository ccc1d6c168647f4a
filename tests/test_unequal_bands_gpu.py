"""FP64 rotations and back-projections of bands (projectors) of unequal norm, at
sizes that run on the tensor cores: a band's digits do not depend on how large the
others are.

Entries have magnitudes of 0.5 to 1.5 times their band's norm.  The bounds are
those of the small multiply-add kernels (tests/test_small_products_gpu.py): a sum
of n products is off by at most 2 sqrt(2) (n + 2) u sum |a| |b|.
"""
import types

import numpy as np
import pytest
import torch

from qimpy_gb300 import ops, sphere as sp, workloads as wl
from qimpy_gb300.electrons import Wavefunction

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0**-53
SPANS = [0, 8, 16, 40, 300]  # decades between the largest and the smallest band


def _flat(rng, *shape):
    return rng.uniform(0.5, 1.5, shape) * np.exp(2j * np.pi * rng.uniform(size=shape))


def _norms(rng, n, span):
    return rng.permutation(10.0 ** (-span * np.arange(n) / (n - 1)))


def _bound(n, mag):
    return 2.0 * np.sqrt(2.0) * (n + 2) * U * mag


def _gpu(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV)


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("span", SPANS)
def test_identity_rotation(span, accumulate):
    rng = np.random.default_rng(span)
    n = 160
    C = _flat(rng, 1, n, 1200) * _norms(rng, n, span)[:, None]
    out = torch.zeros(C.shape, dtype=torch.complex128, device=DEV)
    got = ops.matmul(_gpu(C), torch.eye(n, dtype=torch.complex128, device=DEV)[None], out=out,
                     accumulate=accumulate).cpu().numpy()
    assert np.all(np.abs(got - C) <= _bound(n + 1, np.abs(C)))


# W takes the norms back (as the matrix that orthonormalises does), takes the inverse
# of other norms on its columns, or leaves the small bands small.
@pytest.mark.parametrize("kind", ["compensated", "columns", "plain"])
@pytest.mark.parametrize("span", SPANS)
@pytest.mark.parametrize("nk,n_in,n_out,G", [(1, 130, 97, 1300), (3, 66, 70, 1027), (1, 352, 64, 777)])
def test_rotation(nk, n_in, n_out, G, span, kind):
    rng = np.random.default_rng(n_in + span)
    s = np.stack([_norms(rng, n_in, min(span, 140)) for _ in range(nk)])
    t = np.stack([_norms(rng, n_out, min(span, 140)) for _ in range(nk)])
    C = _flat(rng, nk, n_in, G) * s[:, :, None]
    M = _flat(rng, nk, n_in, n_out)
    if kind != "plain":
        M = M / s[:, :, None]
    if kind == "columns":
        M = M * t[:, None, :]
    got = ops.matmul(_gpu(C), _gpu(M)).cpu().numpy()
    want = np.einsum("kij,kig->kjg", M, C)
    mag = np.einsum("kij,kig->kjg", np.abs(M), np.abs(C))
    assert np.all(np.abs(got - want) <= _bound(n_in + 1, mag))


def test_zero_and_non_finite_bands_leave_the_others():
    rng = np.random.default_rng(5)
    n, G = 96, 1500
    s = _norms(rng, n, 12)
    C = _flat(rng, 1, n, G) * s[:, None]
    M = _flat(rng, 1, n, 80) / s[:, None]
    C[0, 7] = 0.0
    M[0, 7, :] = 1e300
    C[0, 11, 3] = np.inf
    M[0, 20, 5] = np.nan
    C[0, 30, :50] = 0.0
    got = ops.matmul(_gpu(C), _gpu(M)).cpu().numpy()
    Cf, Mf = np.where(np.isfinite(C), C, 0.0), np.where(np.isfinite(M), M, 0.0)
    want, mag = np.einsum("kij,kig->kjg", Mf, Cf), np.einsum("kij,kig->kjg", np.abs(Mf), np.abs(Cf))
    fine = np.ones(want.shape, bool)
    fine[:, :, 3], fine[:, 5, :] = False, False
    assert np.all((np.abs(got - want) <= _bound(n + 1, mag))[fine])
    assert not np.isfinite(got[~fine]).any()


@pytest.mark.parametrize("span", [0, 8, 12, 16])
def test_orthonormalize(span):
    """Cholesky orthonormalisation deviates by at most 6 (m n + n (n + 1)) u kappa^2
    from orthonormal (Yamamoto, Nakatsukasa, Yanagisawa and Fukaya, ETNA 44, 2015),
    and does not depend on the scale of the rows: kappa is that of the unit rows."""
    rng = np.random.default_rng(span)
    n, G = 96, 1500
    unit = _flat(rng, 1, n, G)
    kappa = np.linalg.cond(unit[0])
    C = unit * _norms(rng, n, span)[:, None]
    basis = types.SimpleNamespace(real=None, tc_subspace=False)
    Q = Wavefunction(basis, coeff=_gpu(C)).orthonormalize().coeff.cpu().numpy()[0]
    assert np.abs(Q.conj() @ Q.T - np.eye(n)).max() <= 6 * (G * n + n * (n + 1)) * U * kappa**2


@pytest.mark.parametrize("span", SPANS[:4])
def test_back_projection(span):
    """H of projectors of unequal scale whose D takes the scale back, without a potential."""
    rng = np.random.default_rng(span)
    Gb = 2.0 * np.pi * np.eye(3) / np.array([12.0, 13.0, 14.0])[:, None]
    shape, atoms, pa, nb = (36, 36, 40), 24, 4, 48
    b = wl.make_basis(Gb, np.zeros((1, 3)), 8.0, shape)
    n = int(b.n[0])
    ds = sp.DeviceSphere(sp.build_tables(b.fft_index, b.n, shape), b.ke, DEV, torch.complex128)
    ds.set_potential(torch.zeros(shape, dtype=torch.float64))
    P = atoms * pa
    s = np.repeat(_norms(rng, atoms, span), pa)
    n_tot = b.ke.shape[1]
    beta, C = np.zeros((1, P, n_tot), complex), np.zeros((1, nb, n_tot), complex)
    beta[:, :, :n] = _flat(rng, 1, P, n) * s[:, None]
    C[:, :, :n] = _flat(rng, 1, nb, n)
    D = _flat(rng, atoms, pa, pa) / (s.reshape(atoms, pa)[:, :, None] * s.reshape(atoms, pa)[:, None, :])
    got, _ = ops.hamiltonian(ds, _gpu(C), _gpu(beta), _gpu(D))

    def term(f):
        proj = np.einsum("kpg,kbg->kbp", f(beta.conj()), f(C)).reshape(1, nb, atoms, pa)
        Dp = np.einsum("arc,kbac->kbar", f(D), proj).reshape(1, nb, P)
        return f(b.ke)[:, None, :] * f(C) + np.einsum("kpg,kbp->kbg", f(beta), Dp)

    assert P * nb * n > 5e6
    err = np.abs(got.cpu().numpy() - term(lambda x: x))
    assert np.all(err <= _bound(n + P + pa + 4, term(np.abs)))

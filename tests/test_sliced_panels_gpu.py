"""FP64 band products by integer slices whose operands are sliced in several panels,
and whose CTAs take several output tiles of several chunks of K each, against
exactly summed products at sampled outputs (tests/test_sliced_products_gpu.py).

The bound adds the sums of the panels (at most 16 here, of which each is rounded
twice) to that of one panel: 2^-48 sum |a| |b| over the real products.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops
from test_sliced_products_gpu import _exact_dot, _rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gpu(x):
    return torch.from_numpy(x).to(DEV)


def _near(got, a, b):
    """got = sum a b of real vectors."""
    want = _exact_dot(a, b)
    ma, mb, sa, sb = np.abs(a).max(), np.abs(b).max(), np.abs(a).sum(), np.abs(b).sum()
    bound = 2.0**-54 * (ma * sb + sa * mb) + 2.0**-58 * len(a) * ma * mb
    return abs(got - want) <= bound + 2.0**-48 * np.abs(a * b).sum()


def _parts(a, b, conj):
    s = -1.0 if conj else 1.0
    re = np.concatenate((a.real, -s * a.imag)), np.concatenate((b.real, b.imag))
    im = np.concatenate((a.real, s * a.imag)), np.concatenate((b.imag, b.real))
    return re, im


def _points(n, m, count=12):
    g = np.random.default_rng(n + m)
    return [(0, 0), (n - 1, m - 1)] + [(int(g.integers(n)), int(g.integers(m))) for _ in range(count)]


# 5 panels; 2 k of 4 panels; 3 output tiles a CTA in one panel of 16 chunks, 6 in 4 panels.
@pytest.mark.parametrize("nk,nx,ny,n", [(1, 352, 176, 37073), (2, 300, 150, 20011), (1, 900, 900, 2000),
                                        (1, 1300, 1300, 6001)])
def test_overlap(nk, nx, ny, n):
    X, Y = _rand((nk, nx, n), 1, 3.0), _rand((nk, ny, n), 2)
    dev = _gpu(X), _gpu(Y)
    got = ops.dot(*dev)
    assert torch.equal(got, ops.dot(*dev))
    got = got.cpu().numpy()
    for k in range(nk):
        for i, j in _points(nx, ny):
            re, im = _parts(X[k, i], Y[k, j], True)
            assert _near(got[k, i, j].real, *re) and _near(got[k, i, j].imag, *im)


def test_weighted_real_overlap():
    nx, ny, n = 300, 200, 37073
    X, Y = _rand((1, nx, n), 3), _rand((1, ny, n), 4)
    w = np.where(np.arange(n) % 3 == 0, 1.0, 2.0)
    got = ops.dot_real(_gpu(X), _gpu(Y), _gpu(w)).cpu().numpy()
    assert np.all(got.imag == 0.0)
    for i, j in _points(nx, ny):
        assert _near(got[0, i, j].real, *_parts(X[0, i], Y[0, j] * w, True)[0])


# 3 panels of 6 chunks, 2 k of 2 panels, 12 output tiles a CTA of 3 chunks.
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("nk,n_in,n_out,n", [(1, 352, 64, 30011), (2, 300, 100, 10007), (1, 150, 640, 11003)])
def test_rotation(nk, n_in, n_out, n, accumulate):
    C, M, O = _rand((nk, n_in, n), 5), _rand((nk, n_in, n_out), 6), _rand((nk, n_out, n), 7)
    got = ops.matmul(_gpu(C), _gpu(M), out=_gpu(O), accumulate=accumulate).cpu().numpy()
    one = np.ones(1) if accumulate else np.zeros(1)
    for k in range(nk):
        for j, g in _points(n_out, n, 40):
            re, im = _parts(M[k, :, j], C[k, :, g], False)
            re = np.concatenate((re[0], one)), np.append(re[1], O[k, j, g].real)
            im = np.concatenate((im[0], one)), np.append(im[1], O[k, j, g].imag)
            assert _near(got[k, j, g].real, *re) and _near(got[k, j, g].imag, *im)


def test_non_finite_entry_in_a_later_panel():
    nx, ny, n = 352, 176, 30000
    X, Y = _rand((1, nx, n), 8), _rand((1, ny, n), 9)
    clean = ops.dot(_gpu(X), _gpu(Y)).cpu().numpy()
    X[0, 5, n - 2], Y[0, 9, 12000] = np.nan, np.inf
    got = ops.dot(_gpu(X), _gpu(Y)).cpu().numpy()
    bad = np.zeros((nx, ny), bool)
    bad[5], bad[:, 9] = True, True
    assert np.array_equal(got[0][~bad], clean[0][~bad])
    assert not np.isfinite(got[0][bad]).any()

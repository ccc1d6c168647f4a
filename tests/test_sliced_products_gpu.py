"""FP64 band products by integer slices on the tensor cores (csrc/ozaki.cu),
against exactly summed products (math.fsum of error-free product terms).

The bound on an output is the one the slicing has by construction: operands
rounded to 2^-55 of their row's largest |value| (2^-54 of it is the quantum),
digit pairs below 2^-59 K max|a| max|b| left out, one rounding of every split's
sum and of the total:
    2^-54 (max|a| sum|b| + sum|a| max|b|) + 2^-58 K max|a| max|b| + 2^-51 |out|
over the real products of an output (complex ones have two real products each).
"""
import math

import numpy as np
import pytest
import torch

from qimpy_gb300 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(shape, seed, decay=0.0):
    g = np.random.default_rng(seed)
    x = g.standard_normal(shape) + 1j * g.standard_normal(shape)
    if decay:
        x = x * np.exp(-decay * np.arange(shape[-1]) / shape[-1])
    return x


def _two_product(a, b):
    """p + e = a b exactly (Dekker / Veltkamp)."""
    p = a * b

    def split(x):
        t = 134217729.0 * x
        hi = t - (t - x)
        return hi, x - hi

    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _exact_dot(a, b):
    """sum a b for real vectors, correctly rounded."""
    p, e = _two_product(a, b)
    return math.fsum(np.concatenate((p, e)).tolist())


def _check(got, a, b, conj):
    """got = sum (conj a) b of complex vectors, within the slicing's bound."""
    s = -1.0 if conj else 1.0
    re = _exact_dot(np.concatenate((a.real, -s * a.imag)), np.concatenate((b.real, b.imag)))
    im = _exact_dot(np.concatenate((a.real, s * a.imag)), np.concatenate((b.imag, b.real)))
    ma = max(np.abs(a.real).max(), np.abs(a.imag).max())
    mb = max(np.abs(b.real).max(), np.abs(b.imag).max())
    sa, sb = np.abs(a.real).sum() + np.abs(a.imag).sum(), np.abs(b.real).sum() + np.abs(b.imag).sum()
    bound = 2.0**-54 * (ma * sb + sa * mb) + 2.0**-58 * 2 * len(a) * ma * mb
    assert abs(got.real - re) <= bound + 2.0**-51 * abs(re)
    assert abs(got.imag - im) <= bound + 2.0**-51 * abs(im)


def _sample(n, m, count=40):
    g = np.random.default_rng(0)
    pts = {(0, 0), (n - 1, m - 1), (0, m - 1), (n - 1, 0)}
    while len(pts) < min(count, n * m):
        pts.add((int(g.integers(n)), int(g.integers(m))))
    return sorted(pts)


@pytest.mark.parametrize("decay", [0.0, 30.0])
@pytest.mark.parametrize("nk,nx,ny,n", [(1, 65, 33, 1409), (2, 64, 32, 3001), (1, 130, 97, 128 * 31), (3, 36, 18, 2305),
                                        (1, 8, 160, 4097), (1, 200, 200, 129)])
def test_overlap(nk, nx, ny, n, decay):
    X, Y = _rand((nk, nx, n), 1, decay), _rand((nk, ny, n), 2)
    got = ops.dot(torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV)).cpu().numpy()
    for k in range(nk):
        for i, j in _sample(nx, ny):
            _check(got[k, i, j], X[k, i], Y[k, j], True)
    again = ops.dot(torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV)).cpu().numpy()
    assert np.array_equal(got, again)


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("nk,n_in,n_out,n", [(1, 65, 33, 1409), (2, 130, 32, 1001), (1, 63, 100, 128 * 9),
                                             (3, 36, 18, 2305), (1, 7, 200, 4097), (1, 353, 64, 129)])
def test_rotation(nk, n_in, n_out, n, accumulate):
    C, M = _rand((nk, n_in, n), 3), _rand((nk, n_in, n_out), 4)
    out = torch.zeros((nk, n_out, n), dtype=torch.complex128, device=DEV)
    got = ops.matmul(torch.from_numpy(C).to(DEV), torch.from_numpy(M).to(DEV), out=out,
                     accumulate=accumulate).cpu().numpy()
    for k in range(nk):
        for j, g in _sample(n_out, n):
            _check(got[k, j, g], M[k, :, j], C[k, :, g], False)


def test_rotation_accumulates():
    C, M, O = _rand((1, 65, 2000), 5), _rand((1, 65, 40), 6), _rand((1, 40, 2000), 7)
    d = [torch.from_numpy(t).to(DEV) for t in (C, M, O)]
    want = ops.matmul(d[0], d[1]) + d[2]
    assert torch.equal(ops.matmul(d[0], d[1], out=d[2].clone(), accumulate=True), want)


@pytest.mark.parametrize("nx,ny,n", [(65, 33, 2817), (8, 100, 64 * 97)])
def test_weighted_real_overlap(nx, ny, n):
    X, Y = _rand((1, nx, n), 8), _rand((1, ny, n), 9)
    w = np.where(np.arange(n) % 3 == 0, 1.0, 2.0)
    got = ops.dot_real(torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV),
                       torch.from_numpy(w).to(DEV)).cpu().numpy()
    assert np.all(got.imag == 0.0)
    for i, j in _sample(nx, ny):
        a, b = X[0, i], Y[0, j] * w
        want = _exact_dot(np.concatenate((a.real, a.imag)), np.concatenate((b.real, b.imag)))
        bound = 2.0**-52 * np.abs(a).max() * np.abs(b).max() * n
        assert abs(got[0, i, j].real - want) <= 2.0**-2 * bound + 2.0**-51 * abs(want)


@pytest.mark.parametrize("value", [0x7F7F7F7F7F7F, -0x808080808080, 0x55AA55AA55AA5])
@pytest.mark.parametrize("n", [128 * 40, 37073])
def test_largest_digit_sums_are_exact(value, n):
    """Equal entries with the largest digits drive the FP32 digit-pair sums to
    their bound; integer inputs make the exact result an integer."""
    nx, ny = 32, 32
    X = np.full((1, nx, n), complex(value, -value))
    Y = np.full((1, ny, n), complex(value, value))
    got = ops.dot(torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV)).cpu().numpy()
    # conj(v - i v)(v + i v) = v^2 (1 + i)(1 + i) = 2 i v^2
    want = float(2 * n * value * value)
    assert np.all(np.abs(got.imag - want) <= 2.0**-52 * want)
    assert np.all(np.abs(got.real) <= 2.0**-52 * want)


@pytest.mark.parametrize("scale", [1e-305, 1e-160, 1e150])
def test_scales(scale):
    """Products are formed from integers, so only the result can leave the range."""
    X, Y = _rand((1, 64, 1200), 10), _rand((1, 64, 1200), 11)
    got = ops.dot(torch.from_numpy(X * scale).to(DEV), torch.from_numpy(Y / scale).to(DEV)).cpu().numpy()
    want = np.einsum("kig,kjg->kij", X.conj(), Y)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()


def test_rows_with_nan_or_infinity():
    X, Y = _rand((1, 66, 1300), 12), _rand((1, 50, 1300), 13)
    X[0, 3, 700] = complex(np.nan, 1.0)
    Y[0, 7, 5] = complex(np.inf, 0.0)
    clean = ops.dot(torch.from_numpy(np.nan_to_num(X, posinf=1.0)).to(DEV),
                    torch.from_numpy(np.nan_to_num(Y, posinf=1.0)).to(DEV)).cpu().numpy()
    got = ops.dot(torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV)).cpu().numpy()
    bad = np.zeros((66, 50), bool)
    bad[3], bad[:, 7] = True, True
    assert np.array_equal(got[0][~bad], clean[0][~bad])
    assert np.all(np.isnan(got[0, 3])) and not np.isfinite(got[0, :, 7]).any()
    M = _rand((1, 66, 50), 14)
    C = X.copy()
    C[0, 3, 700], C[0, 5, 9] = 1.0, complex(0.0, -np.inf)
    M[0, 2, 4] = complex(np.nan, 0.0)
    got = ops.matmul(torch.from_numpy(C).to(DEV), torch.from_numpy(M).to(DEV)).cpu().numpy()
    want = np.einsum("kij,kig->kjg", M[:, :, :4], np.where(np.isfinite(C), C, 0.0))
    fine = np.ones(1300, bool)
    fine[9] = False
    assert np.abs(got[0, :4][:, fine] - want[0][:, fine]).max() <= 1e-13 * np.abs(want).max()
    assert not np.isfinite(got[0, :, 9]).any() and np.isnan(got[0, 4]).all()

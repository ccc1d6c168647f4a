"""Overlaps of a few rows over a long basis: fewer than 3e6 multiply-adds, split
over g as well.  Bounds as in tests/test_small_products_gpu.py."""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops
from test_small_products_gpu import _bound, _dev, _rand

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# One output to many tiles; g a multiple of the parts, one above, and an end that some parts do not reach.
SIZES = [(1, 1, 1, 8192), (1, 1, 1, 300001), (1, 4, 3, 37073), (2, 3, 2, 25601), (1, 9, 5, 20000), (1, 18, 18, 8000),
         (3, 8, 4, 16385), (1, 2, 33, 30011), (30, 2, 2, 9000)]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nk,M,N,K", SIZES)
def test_overlap(nk, M, N, K, dtype):
    rng = np.random.default_rng(K)
    X, Xh = _dev(_rand(rng, nk, M, K), dtype)
    Y, Yh = _dev(_rand(rng, nk, N, K), dtype)
    got = ops.dot(X, Y)
    assert torch.equal(got, ops.dot(X, Y))
    want = np.einsum("kig,kjg->kij", Xh.conj(), Yh)
    mag = np.einsum("kig,kjg->kij", np.abs(Xh), np.abs(Yh))
    assert np.all(np.abs(got.cpu().numpy() - want) <= _bound(K, dtype, mag))


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nk,P,nb,n", [(1, 4, 3, 37073), (2, 5, 2, 25601)])
def test_projection(nk, P, nb, n, dtype):
    """The result has the operands' precision and its own strides."""
    rng = np.random.default_rng(n)
    beta, bh = _dev(_rand(rng, nk, P, n), dtype)
    C, Ch = _dev(_rand(rng, nk, nb, n), dtype)
    got = ops.project(beta, C).cpu().numpy()
    want, mag = np.einsum("kpg,kbg->kbp", bh.conj(), Ch), np.einsum("kpg,kbg->kbp", np.abs(bh), np.abs(Ch))
    assert np.all(np.abs(got - want) <= _bound(n + 1, dtype, mag))


def test_weighted_real_overlap():
    rng = np.random.default_rng(1)
    K = 40001
    X, Xh = _dev(_rand(rng, 1, 5, K), torch.complex128)
    Y, Yh = _dev(_rand(rng, 1, 3, K), torch.complex128)
    w = rng.choice([0.0, 1.0, 2.0], K)
    got = ops.dot_real(X, Y, torch.from_numpy(w).to(DEV)).cpu().numpy()
    mag = np.einsum("kig,kjg->kij", np.abs(Xh), np.abs(Yh) * w)
    assert np.all(got.imag == 0.0)
    assert np.all(np.abs(got - np.einsum("kig,kjg->kij", Xh.conj(), Yh * w).real) <= _bound(K + 1, torch.complex128, mag))


def test_few_rows_fill_the_gpu():
    """4 x 3 over 100000 is 1.2 M multiply-adds of 4 FP64 operations: 20 us of one SM in
    40, so a call that keeps four SMs busy (0.4 ms) is far above this limit."""
    X = torch.randn((1, 4, 100000), dtype=torch.complex128, device=DEV)
    Y = torch.randn((1, 3, 100000), dtype=torch.complex128, device=DEV)
    ops.dot(X, Y)
    times = []
    for _ in range(10):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            ops.dot(X, Y)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) / 10)
    assert min(times) < 0.15

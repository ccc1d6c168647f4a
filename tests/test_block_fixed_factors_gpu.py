"""FP64 local potential with potentials whose fixed-point factors have every kind of
low half: odd multiples of one power of two (a lowest bit that lands on each position
around the middle of 62 bits), values that came from FP32, and values drawn at random.

An FFT of N points is off by at most some 4 log2(N) u of its norm (Higham, Accuracy and
Stability, section 24.1); two of them, a product and the largest of some 1e4 entries
against their norm: 64 log2(N) u of the largest entry.
"""
import numpy as np
import pytest
import torch

from oracle import hpsi as oh
from qimpy_gb300 import ops, sphere as sp

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = [(15, 14, 24), (6, 5, 16), (28, 18, 10), (75, 49, 45)]


def _check(shape, V, seed):
    rng = np.random.default_rng(seed)
    N = int(np.prod(shape))
    n = N // 5
    idx = np.sort(rng.choice(N, n, replace=False))[None]
    ds = sp.DeviceSphere(sp.build_tables(idx, np.array([n]), shape), np.zeros((1, n)), DEV, torch.complex128)
    ds.set_potential(torch.from_numpy(V))
    C = rng.standard_normal((1, 3, n)) + 1j * rng.standard_normal((1, 3, n))
    got = ops.apply_potential(ds, torch.from_numpy(C).to(DEV)).cpu().numpy()
    want = oh.apply_potential(V, idx, np.array([n]), C)
    assert np.abs(got - want).max() <= 64 * np.log2(N) * 2.0**-53 * np.abs(want).max()


@pytest.mark.parametrize("bit", range(20, 40))
@pytest.mark.parametrize("shape", SHAPES)
def test_odd_multiples(shape, bit):
    rng = np.random.default_rng(bit)
    odd = 2.0 * rng.integers(0, 2 ** (bit - 1), shape) + 1.0
    _check(shape, odd * 2.0**-bit * rng.choice([-1.0, 1.0], shape), bit)


@pytest.mark.parametrize("decades", [0, 4])
@pytest.mark.parametrize("shape", SHAPES)
def test_values_from_fp32(shape, decades):
    rng = np.random.default_rng(decades)
    V = rng.standard_normal(shape) * 10.0 ** rng.uniform(-decades, 0.0, shape)
    _check(shape, V.astype(np.float32).astype(np.float64), 1)


@pytest.mark.parametrize("seed", range(6))
def test_random_values(seed):
    shape = SHAPES[3]
    _check(shape, np.random.default_rng(seed).standard_normal(shape), seed)

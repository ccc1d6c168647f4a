"""Axes of one codelet size, transformed in one pass or (the default from 8 on)
in two: the local potential and the density of both plans against each other.

Bounds.  FP64: 24 2^-52 of the 2-norm for each plan against exact transforms
(11 passes and the product with V at 2^-52 each, and as much again), so 48 2^-52
between two.  FP32: a codelet of at most 16 points adds to each of its outputs a
rounding error of at most 8 2^-24 of the block's norm; 12 passes and the two
plans: 2 * 12 * 8 2^-24.  The density is a sum of |psi|^2 after the inverse
transforms alone; its relative error is twice psi's.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops, sphere as sp, workloads as wl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BOUND = {torch.complex128: 48 * 2.0**-52, torch.complex64: 192 * 2.0**-24}


def test_default_rule():
    assert [sp.factor_axis(N) for N in (1, 2, 5, 7)] == [(1, 1), (2, 1), (5, 1), (7, 1)]
    assert [sp.factor_axis(N) for N in (8, 9, 10, 12, 14, 15, 16)] == [
        (4, 2), (3, 3), (5, 2), (4, 3), (7, 2), (5, 3), (4, 4)]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 9, 9), (10, 10, 10), (12, 12, 12), (14, 14, 14), (15, 15, 15),
                                   (16, 16, 16), (7, 8, 16), (15, 4, 36), (48, 9, 5), (2, 16, 10)])
def test_split_matches_one_pass(shape, dtype):
    R = np.diag([0.31 * s for s in shape])
    b = wl.make_basis(2.0 * np.pi * np.linalg.inv(R.T), np.array([[0.0, 0.0, 0.0], [0.3, -0.2, 0.4]]),
                      0.5 * (np.pi / 0.31 / 2.0) ** 2, shape)
    rng = np.random.default_rng(5)
    V = torch.from_numpy(rng.standard_normal(shape))
    C = (rng.standard_normal((2, 3, b.n_tot)) + 1j * rng.standard_normal((2, 3, b.n_tot))) / (1.0 + b.ke[:, None])
    for k in range(2):
        C[k, :, b.n[k]:] = 0.0
    C = torch.from_numpy(C).to(DEV, dtype)
    pre = torch.from_numpy(rng.random((2, 3)) + 0.1).to(DEV)
    out = []
    for fac in (None, tuple((N, 1) if N <= 16 else sp.factor_axis(N) for N in shape)):
        ds = sp.DeviceSphere(sp.build_tables(b.fft_index, b.n, shape, fac), b.ke, DEV, dtype)
        ds.set_potential(V)
        out.append((ops.apply_potential(ds, C), ops.collect_density(ds, C, pre)))
    (h, n), (h1, n1) = out
    err = (h - h1).abs().to(torch.float64).norm(dim=-1) / h1.abs().to(torch.float64).norm(dim=-1)
    assert float(err.max()) <= BOUND[dtype]
    assert float((n - n1).norm() / n1.norm()) <= 2 * BOUND[dtype]

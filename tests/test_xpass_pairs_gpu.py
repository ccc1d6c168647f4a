"""FP32 local potential, whose x-pass takes pairs of columns 32 apart: last tiles
of 1 to 32 and of 33 to 63 columns, planes of fewer than 32, axes of one codelet,
every radix in either place, and axes long enough for the wide CTAs.

Bound: a codelet of at most 16 points adds to each output a rounding error of at
most 8 2^-24 of its block's norm; 12 passes (V's product and numpy's rounding of
the inputs included): 96 2^-24 of the 2-norm.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops, sphere as sp, workloads as wl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BOUND = 96 * 2.0**-24

FACTORS = [(f, g) for f in (2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16) for g in (2, 9)]
SHAPES = [((12, 5, 5), None), ((20, 5, 14), None), ((24, 9, 7), None), ((18, 8, 12), None), ((16, 15, 14), None),
          ((6, 9, 10), None), ((15, 10, 10), ((15, 1), (5, 2), (5, 2))), ((16, 10, 10), ((1, 16), (5, 2), (5, 2))),
          ((135, 12, 12), None), ((144, 9, 14), None), ((225, 10, 12), None), ((256, 8, 9), None)]


def _check(shape, fac, nb=3):
    R = np.diag([0.31 * s for s in shape])
    b = wl.make_basis(2.0 * np.pi * np.linalg.inv(R.T), np.array([[0.0, 0.0, 0.0], [0.1, -0.05, 0.2]]),
                      0.5 * (np.pi / 0.31 / 2.0) ** 2, shape)
    ds = sp.DeviceSphere(sp.build_tables(b.fft_index, b.n, shape, fac), b.ke, DEV, torch.complex64)
    rng = np.random.default_rng(sum(shape))
    V = rng.standard_normal(shape).astype(np.float32)
    ds.set_potential(torch.from_numpy(V.astype(np.float64)))
    C = ((rng.standard_normal((2, nb, b.n_tot)) + 1j * rng.standard_normal((2, nb, b.n_tot)))
         / (1.0 + b.ke[:, None])).astype(np.complex64)
    for k in range(2):
        C[k, :, b.n[k]:] = 0.0
    C[:, 1] = 0.0
    got = ops.apply_potential(ds, torch.from_numpy(C).to(DEV)).cpu().numpy()
    assert np.all(got[:, 1] == 0.0)
    for k in range(2):
        idx = b.fft_index[k, : b.n[k]]
        for i in range(nb):
            grid = np.zeros(int(np.prod(shape)), complex)
            grid[idx] = C[k, i, : b.n[k]]
            want = np.fft.fftn(np.fft.ifftn(grid.reshape(shape), norm="forward") * V, norm="forward").reshape(-1)[idx]
            assert np.linalg.norm(got[k, i, : b.n[k]] - want) <= BOUND * np.linalg.norm(want)


@pytest.mark.parametrize("shape,fac", SHAPES)
def test_tiles(shape, fac):
    _check(shape, fac)


@pytest.mark.parametrize("f,g", FACTORS)
def test_radices(f, g):
    _check((f * g, 6, 9), ((f, g), (6, 1), (3, 3)), nb=2)
    _check((f * g, 6, 9), ((g, f), (6, 1), (3, 3)), nb=2)

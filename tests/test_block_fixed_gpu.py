"""FP64 local potential through the block fixed-point codelets (csrc/block_fixed.cuh).

Every codelet radix as the first and the second factor of an axis, axes of one
codelet, odd sizes, x-pass column splits, values from 1e-250 to 1e250 and
non-finite inputs, against numpy FFTs.  A codelet rounds each output once
(2^-53 of it) and its integers to below 2^-54 of the block's largest, so a pass
adds at most 2^-52 of the 2-norm; there are 11 passes and the multiplication by
V, and numpy's transforms are taken to be as far off: 24 2^-52.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops, sphere as sp, workloads as wl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BOUND = 24 * 2.0**-52


def _setup(shape, fac=None, ecut=None, nb=3, seed=1):
    R = np.diag([0.31 * s for s in shape])
    Gb = 2.0 * np.pi * np.linalg.inv(R.T)
    # the sphere takes half of each axis, as the density grid rule leaves it
    ecut = ecut or 0.5 * (np.pi / 0.31 / 2.0) ** 2
    b = wl.make_basis(Gb, np.array([[0.0, 0.0, 0.0], [0.3, -0.2, 0.4]]), ecut, shape)
    ds = sp.DeviceSphere(sp.build_tables(b.fft_index, b.n, shape, fac), b.ke, DEV, torch.complex128)
    g = np.random.default_rng(seed)
    V = g.standard_normal(shape)
    C = (g.standard_normal((2, nb, b.n_tot)) + 1j * g.standard_normal((2, nb, b.n_tot))) / (1.0 + b.ke[:, None])
    for k in range(2):
        C[k, :, b.n[k]:] = 0.0
    ds.set_potential(torch.from_numpy(V))
    return b, ds, V, C


def _want(b, V, C, shape):
    out = np.zeros_like(C)
    for k in range(C.shape[0]):
        idx = b.fft_index[k, : b.n[k]]
        for i in range(C.shape[1]):
            grid = np.zeros(int(np.prod(shape)), complex)
            grid[idx] = C[k, i, : b.n[k]]
            psi = np.fft.ifftn(grid.reshape(shape), norm="forward") * V
            out[k, i, : b.n[k]] = np.fft.fftn(psi, norm="forward").reshape(-1)[idx]
    return out


def _check(b, ds, V, C, shape, scale=1.0):
    got = ops.apply_potential(ds, torch.from_numpy(C * scale).to(DEV)).cpu().numpy() / scale
    want = _want(b, V, C, shape)
    for k in range(C.shape[0]):
        for i in range(C.shape[1]):
            assert np.linalg.norm(got[k, i] - want[k, i]) <= BOUND * np.linalg.norm(want[k, i])


RADIX_AXES = [(4, (2, 2)), (6, (3, 2)), (10, (2, 5)), (12, (4, 3)), (15, (3, 5)), (18, (3, 6)), (21, (7, 3)),
              (24, (4, 6)), (27, (9, 3)), (28, (14, 2)), (30, (2, 15)), (32, (16, 2)), (36, (3, 12)), (40, (10, 4)),
              (42, (3, 14)), (45, (15, 3)), (48, (3, 16)), (56, (7, 8)), (60, (6, 10)), (63, (7, 9)), (96, (12, 8))]


@pytest.mark.parametrize("N,f", RADIX_AXES)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_every_radix_on_every_axis(N, f, axis):
    shape, fac = [15, 15, 15], [(15, 1)] * 3
    shape[axis], fac[axis] = N, f
    _check(*_setup(tuple(shape), tuple(fac)), tuple(shape))


@pytest.mark.parametrize("shape", [(16, 14, 12), (9, 10, 7), (8, 5, 6), (20, 84, 90), (100, 18, 108), (112, 30, 112)])
def test_shapes_and_column_splits(shape):
    _check(*_setup(shape, nb=2), shape)


def test_axis_of_one_codelet_as_second_factor():
    _check(*_setup((14, 15, 16), ((1, 14), (1, 15), (1, 16))), (14, 15, 16))


@pytest.mark.parametrize("scale", [1e-250, 1e-60, 1e150, 1e250])
def test_scales(scale):
    shape = (20, 24, 28)
    _check(*_setup(shape), shape, scale)


def test_zero_and_single_coefficient_bands():
    """A zero band stays exactly zero; one coefficient is a plane wave, whose
    product with V is V's own coefficients shifted."""
    shape = (20, 24, 28)
    b, ds, V, C = _setup(shape)
    C[:, 0] = 0.0
    C[:, 1] = 0.0
    C[:, 1, 5] = 1.0 - 2.0j
    got = ops.apply_potential(ds, torch.from_numpy(C).to(DEV)).cpu().numpy()
    assert np.all(got[:, 0] == 0.0)
    want = _want(b, V, C, shape)
    for k in range(2):
        assert np.linalg.norm(got[k, 1] - want[k, 1]) <= BOUND * np.linalg.norm(want[k, 1])


def test_large_potential_range():
    """V from 1e-12 to 1e12 over the cell."""
    shape = (20, 24, 28)
    b, ds, V, C = _setup(shape)
    V = V * 10.0 ** np.linspace(-12, 12, shape[0])[:, None, None]
    ds.set_potential(torch.from_numpy(V))
    _check(b, ds, V, C, shape)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_bands_stay_apart(value):
    shape = (20, 24, 28)
    b, ds, V, C = _setup(shape)
    clean = ops.apply_potential(ds, torch.from_numpy(C).to(DEV)).cpu().numpy()
    bad = C.copy()
    bad[0, 1, 7] = complex(value, 0.0)
    got = ops.apply_potential(ds, torch.from_numpy(bad).to(DEV)).cpu().numpy()
    assert not np.isfinite(got[0, 1, : b.n[0]]).any()
    keep = np.ones((2, 3), bool)
    keep[0, 1] = False
    assert np.array_equal(got[keep], clean[keep])
    Vbad = V.copy()
    Vbad[3, 4, 5] = value
    ds.set_potential(torch.from_numpy(Vbad))
    got = ops.apply_potential(ds, torch.from_numpy(C).to(DEV)).cpu().numpy()
    for k in range(2):
        assert not np.isfinite(got[k, :, : b.n[k]]).any()

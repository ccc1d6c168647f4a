"""The FP64 local potential near the ends of the range of doubles: a band scaled by
a power of two comes back scaled by it, while every value of the transforms (the
largest is bounded below) is under 2^1018; smaller ones are kept to 2^-1022."""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops, sphere as sp, workloads as wl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = [(15, 20, 25), (16, 18, 28), (6, 5, 24)]


def _sphere(shape, V):
    Gb = 2.0 * np.pi * np.eye(3) / (0.45 * np.array(shape))[:, None]
    b = wl.make_basis(Gb, np.zeros((1, 3)), 5.0, shape)
    ds = sp.DeviceSphere(sp.build_tables(b.fft_index, b.n, shape), b.ke, DEV, torch.complex128)
    ds.set_potential(torch.from_numpy(V))
    return b, ds


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    V = rng.uniform(-1.0, 1.0, shape)
    b, ds = _sphere(shape, V)
    C = rng.standard_normal((1, 3, b.ke.shape[1])) + 1j * rng.standard_normal((1, 3, b.ke.shape[1]))
    C[:, :, int(b.n[0]):] = 0.0
    return V, b, ds, torch.from_numpy(C).to(DEV)


def _largest(V, b, C):
    """Bound on any value of the transforms, inside their passes too: the sums of magnitudes."""
    n = int(b.n[0])
    return np.abs(C.cpu().numpy()[0, :, :n]).sum(axis=1).max() * np.abs(V).max() * V.size


@pytest.mark.parametrize("shape", SHAPES)
def test_large(shape):
    V, b, ds, C = _case(shape, 1)
    ref = ops.apply_potential(ds, C, add_ke=True)
    m = 1018 - int(np.ceil(np.log2(_largest(V, b, C))))
    assert m > 960
    got = ops.apply_potential(ds, C * 2.0**m, add_ke=True)
    assert torch.equal(got * 2.0**-m, ref)


@pytest.mark.parametrize("shape", SHAPES)
def test_large_values_meet_in_one_block(shape):
    """Blocks whose largest value is above 2^1016: one plane wave, whose amplitude is all there is."""
    V = np.ones(shape)
    b, ds = _sphere(shape, V)
    C = torch.zeros((1, 1, b.ke.shape[1]), dtype=torch.complex128, device=DEV)
    C[0, 0, int(b.n[0]) // 2] = 1.0
    ref = ops.apply_potential(ds, C)
    m = 1017 - int(np.ceil(np.log2(V.size)))
    got = ops.apply_potential(ds, C * 2.0**m)
    assert torch.equal(got * 2.0**-m, ref)


def test_potential_of_the_lowest_value():
    """A mask of the most negative double: finite where the exact result is."""
    shape = SHAPES[0]
    rng = np.random.default_rng(2)
    mask = rng.random(shape) < 0.1
    b, ds = _sphere(shape, np.where(mask, np.finfo(float).min, 0.0))
    _, ds1 = _sphere(shape, np.where(mask, -1.0, 0.0))
    C = torch.from_numpy(rng.standard_normal((1, 2, b.ke.shape[1])) * 2.0**-30 + 0j).to(DEV)
    C[:, :, int(b.n[0]):] = 0.0
    got, one = ops.apply_potential(ds, C), ops.apply_potential(ds1, C)
    want = one * 2.0**30 * (np.finfo(float).max * 2.0**-30)
    assert bool(torch.isfinite(torch.view_as_real(got)).all())
    assert float((got - want).abs().max()) <= 1e-13 * float(want.abs().max())


@pytest.mark.parametrize("down", [900, 940, 960, 980])
@pytest.mark.parametrize("shape", SHAPES)
def test_small(shape, down):
    """Numbers are kept to 2^-1022, so a band of 2^-down to 2^(down - 1022) of its largest."""
    V, b, ds, C = _case(shape, 3)
    ref = ops.apply_potential(ds, C)
    got = ops.apply_potential(ds, C * 2.0**-down) * 2.0**down
    scale = float(ref.abs().max())
    # Each of the six passes' two codelets (and the product) rounds to 2^-1022, and the
    # forward ones add up to N of these before the division by N.
    bound = 13 * np.sqrt(2.0) * V.size * 2.0 ** (down - 1022) + 1e-14 * scale
    assert float((got - ref).abs().max()) <= bound


def test_small_potential():
    shape = SHAPES[0]
    V, b, ds, C = _case(shape, 4)
    ref = ops.apply_potential(ds, C)
    _, tiny = _sphere(shape, V * 2.0**-500)
    got = ops.apply_potential(tiny, C * 2.0**-460) * 2.0**960
    assert float((got - ref).abs().max()) <= 13 * np.sqrt(2.0) * V.size * 2.0**-62 + 1e-14 * float(ref.abs().max())

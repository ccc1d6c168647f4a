"""FP64 overlaps of rows whose large entries do not meet.

The sliced form is accurate relative to the largest entries of the rows within
each range of K that it sums by itself,
    2^-54 (max|a| sum|b| + sum|a| max|b|) + 2^-59 K max|a| max|b|
(each real product of a complex one, plus the rounding of the result).  Grades over
the basis as a whole are met by the ranges; where they repeat within every range, the
result loses, relative to sum |a| |b|, what the entries that meet are below the
largest.  The multiply-add form, which qgb_dot takes with a workspace of
qgb_dot_workspace_bytes, keeps to 2 sqrt(2) (K + 2) 2^-53 sum |a| |b|.  The errors
relative to sum |a| |b| are recorded with the test.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import _lib, ops
from test_sliced_products_gpu import _exact_dot

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _plain_dot(X, Y):
    """qgb_dot with the workspace of the multiply-add form."""
    lib = _lib.lib()
    nk, nx, n = X.shape
    ny = Y.shape[1]
    out = torch.empty((nk, nx, ny), dtype=torch.complex128, device=DEV)
    ws = torch.empty(max(1, lib.qgb_dot_workspace_bytes(_lib.QGB_F64, nk, nx, ny, n)), dtype=torch.uint8, device=DEV)
    _lib.check(lib.qgb_dot(_lib.QGB_F64, X.data_ptr(), nx, Y.data_ptr(), ny, nk, n, out.data_ptr(), ws.data_ptr(),
                           ws.numel(), torch.cuda.current_stream().cuda_stream), "dot")
    return out


@pytest.mark.parametrize("decay", [0, 5, 10, 20, 30])
@pytest.mark.parametrize("period", [4096, 128])
def test_opposite_grades(period, decay, record_property):
    rng = np.random.default_rng(decay)
    m, n = 48, 4096
    X, Y = (rng.standard_normal((1, m, n)) + 1j * rng.standard_normal((1, m, n)) for _ in range(2))
    grade = np.exp(-decay * (np.arange(n) % period) / period)
    X, Y = X * grade, Y * grade[::-1]
    dev = torch.from_numpy(X).to(DEV), torch.from_numpy(Y).to(DEV)
    sliced, plain = ops.dot(*dev).cpu().numpy()[0], _plain_dot(*dev).cpu().numpy()[0]
    assert not np.array_equal(sliced, plain)  # two forms
    worst = {"sliced": 0.0, "plain": 0.0}
    for i, j in zip(rng.integers(0, m, 12), rng.integers(0, m, 12)):
        a, b = X[0, i], Y[0, j]
        re = _exact_dot(np.concatenate((a.real, a.imag)), np.concatenate((b.real, b.imag)))
        im = _exact_dot(np.concatenate((a.real, -a.imag)), np.concatenate((b.imag, b.real)))
        ma, mb = (max(np.abs(x.real).max(), np.abs(x.imag).max()) for x in (a, b))
        sa, sb = (np.abs(x.real).sum() + np.abs(x.imag).sum() for x in (a, b))
        bound = 2.0**-54 * (ma * sb + sa * mb) + 2.0**-59 * 2 * n * ma * mb
        mag = (np.abs(a) * np.abs(b)).sum()
        for name, got in (("sliced", sliced[i, j]), ("plain", plain[i, j])):
            err = abs(got - complex(re, im))
            worst[name] = max(worst[name], err / mag)
            if name == "sliced":
                assert abs(got.real - re) <= bound + 2.0**-51 * abs(re)
                assert abs(got.imag - im) <= bound + 2.0**-51 * abs(im)
            else:
                assert err <= 2.0 * np.sqrt(2.0) * (n + 2) * 2.0**-53 * mag
    for name, w in worst.items():
        record_property(f"{name}_error_over_sum", w)
    print(f"period {period}, decay {decay}: error over sum |a||b|: sliced {worst['sliced']:.1e}, multiply-adds {worst['plain']:.1e}")

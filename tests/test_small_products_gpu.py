"""Small band products (fewer than 3e6 multiply-adds): overlaps in tiles of 4 x 4,
2 x 4 and 2 x 2, rotations of 4, 2 and 1 columns a thread and CTAs of 64 and 32
threads, and the back-projection that applies D itself.

Bounds: a sum of n products of O(1) complex numbers in precision u is off by at
most sqrt(2) (n + 2) u sum |a| |b| in the worst case; with the reference in FP64
(twice the same for FP64).  D adds a sum of pa before it: n + pa + 2.
"""
import numpy as np
import pytest
import torch

from qimpy_gb300 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = {torch.complex128: 2.0**-53, torch.complex64: 2.0**-24}


def _rand(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _dev(x, dtype):
    t = torch.from_numpy(x).to(DEV, dtype)
    return t, t.cpu().numpy().astype(complex)


def _bound(n, dtype, mag):
    return 2.0 * np.sqrt(2.0) * (n + 2) * U[dtype] * mag


# nk, M, N, K: outputs 1, odd, one tile each way, enough CTAs for each tile size;
# K of 1, below, at and above the 256 threads.
GRAMS = [(1, 1, 1, 1), (1, 2, 2, 255), (2, 3, 5, 256), (1, 5, 3, 257), (3, 17, 19, 31), (8, 8, 18, 1150),
         (2, 33, 31, 700), (1, 63, 65, 500), (19, 4, 8, 300), (19, 5, 9, 300), (38, 8, 4, 77)]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nk,M,N,K", GRAMS)
def test_overlap(nk, M, N, K, dtype):
    rng = np.random.default_rng(M * 100 + N)
    X, Xh = _dev(_rand(rng, nk, M, K), dtype)
    Y, Yh = _dev(_rand(rng, nk, N, K), dtype)
    got = ops.dot(X, Y).cpu().numpy()
    want = np.einsum("kig,kjg->kij", Xh.conj(), Yh)
    mag = np.einsum("kig,kjg->kij", np.abs(Xh), np.abs(Yh))
    assert np.all(np.abs(got - want) <= _bound(K, dtype, mag))


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 7, 300), (40, 40, 900)])
def test_weighted_real_overlap(M, N, K, dtype):
    rng = np.random.default_rng(K)
    X, Xh = _dev(_rand(rng, 1, M, K), dtype)
    Y, Yh = _dev(_rand(rng, 1, N, K), dtype)
    w = rng.choice([0.0, 1.0, 2.0], K)
    got = ops.dot_real(X, Y, torch.from_numpy(w).to(DEV)).cpu().numpy()
    want = np.einsum("kig,kjg->kij", Xh.conj(), Yh * w).real
    mag = np.einsum("kig,kjg->kij", np.abs(Xh), np.abs(Yh) * w)
    assert np.all(np.abs(got - want) <= _bound(K + 1, dtype, mag))


# nk, n_in, n_out, G: G below, at and above the CTAs' 32 and 64.
ROTATIONS = [(1, 1, 1, 1), (1, 3, 2, 31), (2, 12, 6, 300), (1, 7, 5, 64), (1, 9, 3, 65), (8, 8, 18, 1150),
             (1, 40, 33, 2000), (3, 5, 41, 1027)]


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nk,n_in,n_out,G", ROTATIONS)
def test_rotation(nk, n_in, n_out, G, dtype, accumulate):
    rng = np.random.default_rng(G)
    X, Xh = _dev(_rand(rng, nk, n_in, G), dtype)
    M, Mh = _dev(_rand(rng, nk, n_in, n_out), dtype)
    o, oh = _dev(_rand(rng, nk, n_out, G), dtype)
    got = ops.matmul(X, M, out=o, accumulate=accumulate).cpu().numpy()
    want = np.einsum("kij,kig->kjg", Mh, Xh) + (oh if accumulate else 0.0)
    mag = np.einsum("kij,kig->kjg", np.abs(Mh), np.abs(Xh)) + np.abs(oh)
    assert np.all(np.abs(got - want) <= _bound(n_in + 1, dtype, mag))


# nk, atoms, pa, nb, G: blocks of 1, 4, 8 (D applied in the rotation) and 9 (its
# own launch), 512 and 520 projectors, columns that 4, 2 and 1 leave over.
NONLOCAL = [(1, 1, 1, 1, 1), (2, 3, 4, 6, 300), (8, 2, 4, 18, 1150), (2, 2, 8, 5, 65), (2, 2, 9, 5, 65),
            (1, 128, 4, 7, 700), (1, 130, 4, 7, 700), (1, 3, 5, 23, 1000)]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("nk,atoms,pa,nb,G", NONLOCAL)
def test_back_projection(nk, atoms, pa, nb, G, dtype):
    rng = np.random.default_rng(atoms * 10 + pa)
    P = atoms * pa
    beta, bh = _dev(_rand(rng, nk, P, G), dtype)
    D, Dh = _dev(_rand(rng, atoms, pa, pa), dtype)
    proj, ph = _dev(_rand(rng, nk, nb, P), dtype)
    out, oh = _dev(_rand(rng, nk, nb, G), dtype)
    got = ops.apply_nonlocal(beta, D, proj, out).cpu().numpy()
    pb = ph.reshape(nk, nb, atoms, pa)
    Dp = np.einsum("arc,kbac->kbar", Dh, pb).reshape(nk, nb, P)
    Dm = np.einsum("arc,kbac->kbar", np.abs(Dh), np.abs(pb)).reshape(nk, nb, P)
    want = oh + np.einsum("kpg,kbp->kbg", bh, Dp)
    mag = np.abs(oh) + np.einsum("kpg,kbp->kbg", np.abs(bh), Dm)
    assert np.all(np.abs(got - want) <= _bound(P + pa + 1, dtype, mag))


def test_short_workspace_is_refused():
    """The overlap's workspace is asked for on every route, also where the small kernel has no use for it."""
    from qimpy_gb300 import _lib

    lib = _lib.lib()
    X = torch.ones((1, 8, 4000), dtype=torch.complex128, device=DEV)
    out = torch.empty((1, 8, 8), dtype=torch.complex128, device=DEV)
    need = lib.qgb_dot_workspace_bytes(_lib.QGB_F64, 1, 8, 8, 4000)
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    st = torch.cuda.current_stream().cuda_stream
    args = (_lib.QGB_F64, X.data_ptr(), 8, X.data_ptr(), 8, 1, 4000, out.data_ptr())
    assert lib.qgb_dot(*args, None, 0, st) != 0
    assert lib.qgb_dot(*args, ws.data_ptr(), need - 1, st) != 0
    assert lib.qgb_dot(*args, ws.data_ptr(), need, st) == 0
    assert torch.equal(out, torch.full_like(out, 4000.0))

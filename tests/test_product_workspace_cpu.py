"""Workspaces of the FP64 band products stay in proportion to their operands and
results, at any size (host arithmetic of the built library; no GPU)."""
import os
import types

import numpy as np
import pytest
import torch

from qimpy_gb300 import _lib, ops

pytestmark = pytest.mark.skipif(not os.path.exists(_lib.LIB_PATH), reason="library not built")

PANEL = 128 << 20  # digits of one panel
WAVE = 152 * 128 * 64 * 8  # partial sums of one wave of CTAs
SIZES = [(1, 65, 33, 1409), (8, 36, 18, 2305), (1, 352, 176, 37073), (1, 2000, 1000, 150000), (4, 1600, 800, 20000),
         (1, 2000, 2000, 200000), (1, 4000, 4000, 300000), (64, 500, 250, 40000), (1, 4, 3, 2000000),
         (512, 40, 40, 5000)]


@pytest.mark.parametrize("nk,M,N,K", SIZES)
def test_overlap(nk, M, N, K):
    lib = _lib.lib()
    n = lib.qgb_dot_fast_workspace_bytes(_lib.QGB_F64, nk, M, N, K)
    plain = lib.qgb_dot_workspace_bytes(_lib.QGB_F64, nk, M, N, K)
    assert n >= plain
    # Digits of 4 chunks of 128 K (28 B a value); partial sums of 128 MB or twice the
    # result; a scale per row and chunk.
    digits = max(PANEL, 4 * 128 * 28 * nk * (M + N))
    scales = 4 * nk * (M + N) * (K // 64 + 2)
    assert n <= max(plain, digits + max(PANEL, WAVE, 32 * nk * M * N) + scales + 4096)


@pytest.mark.parametrize("nk,M,N,K", SIZES)
def test_rotation(nk, M, N, K):
    n = _lib.lib().qgb_matmul_workspace_bytes(_lib.QGB_F64, nk, M, N, K)
    # Digits of 128 g at least, and of the matrix (both of its real forms, 56 B an element).
    rows = max(PANEL, nk * 128 * 28 * (M + 4))
    assert n <= rows + 56 * nk * (M + 4) * (N + 32) + 4 * nk * (M + N + 32 + K + 128) + 4096


def test_projection_and_back_projection():
    """What H.psi asks for beside D proj and the planes."""
    lib = _lib.lib()
    for nk, P, nb, n in ((1, 256, 32, 37073), (1, 2000, 1000, 150000)):
        both = max(lib.qgb_dot_fast_workspace_bytes(_lib.QGB_F64, nk, P, nb, n),
                   lib.qgb_matmul_workspace_bytes(_lib.QGB_F64, nk, P, nb, n))
        assert both < 3 * PANEL


@pytest.mark.parametrize("nk,M,N,K", SIZES + [(1, 1, 1, 1), (2, 12, 6, 300), (8, 36, 18, 1150), (1, 24, 12, 900),
                                              (4, 400, 200, 20000), (1, 256, 32, 37073), (1, 16, 3, 100000)])
def test_estimate_covers_what_the_calls_ask_for(nk, M, N, K):
    lib = _lib.lib()
    asked = max(lib.qgb_dot_fast_workspace_bytes(_lib.QGB_F64, nk, M, N, K),
                lib.qgb_matmul_workspace_bytes(_lib.QGB_F64, nk, M, N, K))
    assert asked <= ops.fp64_product_bytes(nk, M, N, K)


def test_served_requests_count_their_products():
    from qimpy_gb300 import batch as bt, serve as sv

    spec = bt.make_batch_specs(count=1, seed=3)[0]
    for dtype in (torch.complex64, torch.complex128):
        fake = types.SimpleNamespace(dtype=dtype, bands_extra=lambda nb, n: nb // 10 + 1)
        need = sv.EigenServer.estimate_bytes(fake, spec, 64)
        n = int((2.0 * spec.ke_cutoff) ** 1.5 * spec.side**3 / (6 * np.pi**2) * 1.1)
        nbt, elem = 71, 8 if dtype == torch.complex64 else 16
        held = 12 * len(spec.k) * nbt * n * elem + len(spec.k) * nbt * (spec.grid // 2 + 2) * spec.grid**2 * elem
        assert need >= held + _lib.lib().qgb_dot_fast_workspace_bytes(_lib.QGB_F64, len(spec.k), 2 * nbt, nbt, n)

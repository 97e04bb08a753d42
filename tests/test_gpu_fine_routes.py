"""Blocks that the integer-pipe product (csrc/hz_fine_fixed.cu) cannot serve or need not work on,
timed against the native kernel that hz_apply_noalloc runs on the same operator and block:
stretched meshes, whose coefficients lie too far apart, and columns of zeros."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NRHS = 16


def operator(hz, cells, h):
    M = hz.getRegularMesh([v for c, s in zip(cells, h) for v in (0.0, c * s)], list(cells))
    n = int(np.prod([c + 1 for c in cells]))
    m = 0.2 + 0.2 * np.random.default_rng(0).random(n)
    w = 0.2 * np.pi / (min(h) * np.sqrt(m.max()))
    return hz.GetHelmholtzOperator(hz.HelmholtzParam(M, 0.05 * w * np.ones(n), m, w, True, True)), n


def native(hz, A, X):
    handle = next(iter(A._devices.values())).handle
    Y = X.new_empty(X.shape)
    hz._lib.check(hz._lib.load().hz_apply_noalloc(handle, hz._lib.HZ_OP_H, int(A.adj), X.data_ptr(), Y.data_ptr(),
                                                  X.shape[1], X.shape[0]), handle)
    return Y


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("cells,h,zero", [((96, 90, 80), (1, 1, 0.25), False), ((96, 90, 80), (1, 0.3, 0.3), False),
                                          ((1500, 1200), (1, 0.25), False), ((96, 90, 80), (1, 1, 1), True),
                                          ((1500, 1200), (1, 1), True)])
def test_no_slower_than_the_native_kernel(hz, cells, h, zero, adjoint):
    import torch
    H, n = operator(hz, cells, [0.01 * v for v in h])
    A = H.adjoint() if adjoint else H
    gen = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((NRHS, n), dtype=torch.complex128, device="cuda", generator=gen)
    if zero:
        X.zero_()
        X[::3, n // 2] = 1.0
    got, ref = (A @ X.t()).t(), native(hz, A, X)
    assert (got - ref).abs().max() <= 1e-14 * ref.abs().max()

    def once(f):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        f()
        torch.cuda.synchronize()
        return time.perf_counter() - t0

    for _ in range(3):
        once(lambda: A @ X.t()), once(lambda: native(hz, A, X))
    pairs = [(once(lambda: A @ X.t()), once(lambda: native(hz, A, X))) for _ in range(25)]
    mine, theirs = (np.median(v) for v in zip(*pairs))
    assert mine <= 1.15 * theirs, (mine, theirs)

"""Device memory of an operator handle: diag(H), diag(SH) and 1 / diag(SH) in complex FP64 (48
bytes per node); the fixed-point words of H or SH (16 each) come with the first block that needs them."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_words_come_with_their_first_block(hz):
    import torch
    L, lib = hz._lib, hz._lib.load()

    def handle(cells):
        M = hz.getRegularMesh([v for c in cells for v in (0.0, 0.01 * c)], list(cells))
        n = int(np.prod([c + 1 for c in cells]))
        p, keep = hz.api._problem(hz.HelmholtzParam(M, np.full(n, 0.1), np.full(n, 0.3), 20.0, True, True))
        o, h = L.hz_options(), C.c_void_p()
        lib.hz_default_options(C.byref(o))
        L.check(lib.hz_create(C.byref(p), C.byref(o), C.byref(h)))
        return h, n, keep

    def apply(h, n, op, X, Y):
        L.check(lib.hz_apply(h, op, 0, X.data_ptr(), Y.data_ptr(), n, 1, L.HZ_MEM_DEVICE), h)

    # a small handle first: the kernels' code is loaded with their first use
    cells = (160, 128, 128)
    n = int(np.prod([c + 1 for c in cells]))
    X = torch.ones(n, dtype=torch.complex128, device="cuda")
    Y = torch.empty_like(X)
    warm, k, keep0 = handle((64, 64, 64))
    for op in (L.HZ_OP_H, L.HZ_OP_SH):
        apply(warm, k, op, X, Y)
    torch.cuda.synchronize()
    used = [torch.cuda.mem_get_info()[0]]
    h, n, keep = handle(cells)
    used.append(torch.cuda.mem_get_info()[0])
    for op in (L.HZ_OP_H, L.HZ_OP_SH):
        apply(h, n, op, X, Y)
        used.append(torch.cuda.mem_get_info()[0])
    per_node = -np.diff(np.array(used, dtype=float)) / n
    lib.hz_destroy(h)
    lib.hz_destroy(warm)
    slack = 4.0  # allocations round up to 2 MB: 0.8 bytes per node each
    assert abs(per_node[0] - 48) <= slack, per_node
    assert abs(per_node[1] - 16) <= slack and abs(per_node[2] - 16) <= slack, per_node

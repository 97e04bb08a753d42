"""The check of the coarsest level's inverse (csrc/hz_solver.cu, invert_coarsest): undamped
operators near a resonance, where the explicit inverse's backward error is 1e-13 and more and
the band LU's stays at rounding level, are solved by the LU; damped ones by the inverse."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import helmholtz_oracle as O
import problems as PB

pytestmark = pytest.mark.gpu


def launches(hz, S):
    """Launch counts of the solver's kernels by name."""
    lib, h = hz._lib.load(), S._handle
    name, n, timed, ms, by = C.create_string_buffer(64), C.c_int64(), C.c_int64(), C.c_double(), C.c_double()
    out = {}
    for k in range(lib.hz_kernel_times(h, -1, None, 0, None, None, None, None)):
        lib.hz_kernel_times(h, k, name, 64, C.byref(n), C.byref(timed), C.byref(ms), C.byref(by))
        out[name.value.decode()] = (n.value, by.value)
    return out


def solver(hz, prm, levels=1, precision="fp64", outer="fp64", shift=0.0):
    MG = hz.getMGparam(complex, int, levels, 1, 3, 1e-9 if levels == 1 else 1e-6, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0,
                       precision=precision, outerArithmetic=outer)
    MG.cudaGraph = False  # a graph's bytes are charged to the graph
    return hz.getShiftedLaplacianMultigridSolver(prm, MG, shift, "GMRES", 5)


@pytest.mark.parametrize("cells,off", [((33, 64), 0.1), ((24, 24), 0.01), ((60, 30), 0.001), ((16, 16, 16), 0.01)])
def test_near_resonance_takes_the_band_lu(hz, cells, off):
    M = hz.getRegularMesh([v for c in cells for v in (0.0, float(c))], list(cells))
    n = int(np.prod([c + 1 for c in cells]))
    lam = sum(2 - 2 * np.cos(np.pi * (c // 4) / c) for c in cells)  # an eigenvalue of the Neumann Laplacian
    w = np.sqrt(lam * (1 + off))
    S = solver(hz, hz.HelmholtzParam(M, np.zeros(n), np.ones(n), w, True, False))
    B = PB.rhs(n, 2, seed=1)
    X, S = hz.solveLinearSystem(None, B, S)
    assert launches(hz, S).get("band_solve", (0, 0))[0] > 0
    assert list(S.last_iters) == [1, 1]
    assert (S.last_relres <= 1e-9).all()


@pytest.mark.parametrize("cells", [(33, 64), (40, 6), (10, 9, 12), (16, 16, 16)])
def test_damped_operators_take_the_inverse(hz, cells):
    P = PB.layered(cells, seed=3, pad=2)
    S = solver(hz, PB.hz_param(hz, P))
    X, S = hz.solveLinearSystem(None, PB.rhs(P["m"].size, 2, seed=1), S)
    t = launches(hz, S)
    assert t["coarse_product"][0] > 1 and "band_solve" not in t


@pytest.mark.parametrize("precision,outer,digits", [("fp64", "fp64", 8), ("mixed", "fp64", 8), ("mixed", "emulated", 6)])
def test_digits_of_the_inverse(hz, precision, outer, digits):
    """The mixed form's coarsest level is FP64 (8 digits of 8 bits; FP32 is what its cycle's vectors
    are held in); the emulated form's holds the 48 bits of its double-float data.  Bytes charged to a
    product: 4 per digit and entry of the inverse, and the columns."""
    P = PB.layered((64, 32), seed=4, pad=4)
    S = solver(hz, PB.hz_param(hz, P), levels=3, precision=precision, outer=outer, shift=0.5)
    hz.solveLinearSystem(None, PB.rhs(P["m"].size, 3, seed=1), S)
    n, by = launches(hz, S)["coarse_product"]
    N = 17 * 9
    assert by / n >= 4 * digits * N * N
    assert by / n < 4 * (digits + 1) * N * N

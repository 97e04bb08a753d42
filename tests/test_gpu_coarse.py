"""The coarsest level's solve as a product with its inverse in digit form
(csrc/hz_coarse.cu).  With one level and no shift the preconditioner is H^-1, so
the first FGMRES iteration leaves only the error of that product: the inverse's
residual is checked to 1e-10 at setup and the digits carry 64 bits, so a relative
residual above 1e-9 after one iteration is a wrong product."""
from __future__ import annotations

import numpy as np
import pytest

import helmholtz_oracle as O
from problems import hz_param, layered, rhs

pytestmark = pytest.mark.gpu

# node counts around the 16-row and 8-column steps, slab axes x, y and z, narrow
# grids whose slabs hold several planes; the last is above the dense limit (band LU)
GRIDS = [(1, 1), (2, 4), (3, 4), (15, 16), (16, 15), (40, 6), (5, 60), (33, 64), (1, 1, 2), (3, 4, 5), (9, 4, 4),
         (4, 11, 6), (10, 9, 12), (128, 64)]


@pytest.mark.parametrize("cells", GRIDS)
@pytest.mark.parametrize("adjoint", [0, 1])
def test_single_level_is_the_inverse(hz, cells, adjoint):
    P = layered(cells, seed=3, pad=1)
    n = P["m"].size
    H = P["H"].conj().T.tocsr() if adjoint else P["H"]
    for nrhs in (1, 4, 5, 9):
        B = rhs(n, nrhs, seed=nrhs)
        B[:, 0] = 0.0
        B[n // 2, 0] = 1e-100  # a point source far below the other columns' scale
        MG = hz.getMGparam(complex, int, 1, 1, 1, 1e-9, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0)
        S = hz.getShiftedLaplacianMultigridSolver(hz_param(hz, P), MG, 0.0, "GMRES", 10)
        X, S = hz.solveLinearSystem(None, B, S, adjoint)
        assert list(S.last_iters) == [1] * nrhs
        X = X.reshape(n, nrhs)
        Xref = O.direct_solve(H, B).reshape(n, nrhs)
        err = np.linalg.norm(X - Xref, axis=0) / np.linalg.norm(Xref, axis=0)
        assert err.max() <= 1e-7


@pytest.mark.parametrize("cells,levels", [((16, 8), 2), ((36, 20), 3), ((8, 12, 4), 2)])
@pytest.mark.parametrize("outer", ["fp64", "emulated"])
def test_fp32_columns(hz, cells, levels, outer):
    """The 48-bit image under the FP32 cycle: the iterations of the FP64 cycle."""
    P = layered(cells, seed=4, pad=2)
    B = rhs(P["m"].size, 5, seed=7)
    iters = {}
    for prec in ("fp64", "mixed"):
        MG = hz.getMGparam(complex, int, levels, 1, 60, 1e-6, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0,
                           precision=prec, outerArithmetic=outer if prec == "mixed" else "fp64")
        S = hz.getShiftedLaplacianMultigridSolver(hz_param(hz, P), MG, 0.5, "GMRES", 10)
        X, S = hz.solveLinearSystem(None, B, S)
        assert (S.last_relres <= 1e-6).all()
        iters[prec] = S.last_iters
    assert np.abs(iters["fp64"] - iters["mixed"]).max() <= 1
    Xref = O.direct_solve(P["H"], B)
    assert np.linalg.norm(X - Xref) <= 1e-4 * np.linalg.norm(Xref)


@pytest.mark.parametrize("cells", [(1, 1), (3, 4), (33, 9), (64, 32), (3, 4, 5), (10, 9, 12), (16, 16, 16)])
def test_bicgstab_keeps_the_band_substitution(hz, cells):
    """The band LU under BiCGSTAB (one cluster per column, or the whole GPU on the
    larger grids): one level and no shift leave its rounding error after one iteration."""
    P = layered(cells, seed=5, pad=1)
    n = P["m"].size
    Xs = []
    for nrhs in (3, 1):
        B = rhs(n, 3, seed=2)[:, :nrhs]
        MG = hz.getMGparam(complex, int, 1, 1, 3, 1e-9, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0)
        S = hz.getShiftedLaplacianMultigridSolver(hz_param(hz, P), MG, 0.0, "BiCGSTAB", 0)
        X, S = hz.solveLinearSystem(None, B, S)
        assert list(S.last_iters) == [1] * nrhs
        Xref = O.direct_solve(P["H"], B)
        Xs.append(X.reshape(n, nrhs)[:, 0])
        assert np.linalg.norm(X.reshape(Xref.shape) - Xref) <= 1e-7 * np.linalg.norm(Xref)
    np.testing.assert_array_equal(*Xs)  # a column's arithmetic does not depend on the block's width

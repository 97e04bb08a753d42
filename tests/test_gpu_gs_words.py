"""FGMRES with its basis in fixed-point words, one reference per 128 nodes (csrc/hz_krylov.cu):
node counts around that group, restarts above one launch's 16 vectors, zero groups (point
sources) and values whose products leave the words' range and take the native steps.

A solve to 1e-10 ends with a relative residual below it, measured in native FP64; the solution's
error is at most that times the condition number, below 1e4 on these grids: 1e-6.  Iteration
counts are those of the native steps to within one where rounding decides the last."""
from __future__ import annotations

import numpy as np
import pytest

import helmholtz_oracle as O
from problems import hz_param, layered, rhs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,levels", [((1, 1), 1), ((6, 16), 1), ((7, 15), 1), ((2, 42), 1), ((24, 16), 2),
                                          ((64, 64), 3), ((8, 8, 8), 2)])
@pytest.mark.parametrize("restart", [5, 20])
def test_solves_around_a_group(hz, cells, levels, restart):
    P = layered(cells, seed=6, pad=1)
    n = P["m"].size
    B = rhs(n, 3, seed=4)
    B[:, 1] = 0.0
    B[n // 2, 1] = 1.0 + 2.0j
    Xref = O.direct_solve(P["H"], B)
    iters = []
    for scale in (1.0, 2.0**-490):  # the products of two values below 2^-474 are out of range
        MG = hz.getMGparam(complex, int, levels, 1, 200, 1e-10, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0)
        S = hz.getShiftedLaplacianMultigridSolver(hz_param(hz, P), MG, 0.5, "GMRES", restart)
        X, S = hz.solveLinearSystem(None, B * scale, S)
        assert (S.last_relres <= 1e-10).all()
        iters.append(np.asarray(S.last_iters))
        assert np.linalg.norm(X / scale - Xref) <= 1e-6 * np.linalg.norm(Xref)
    assert np.abs(iters[0] - iters[1]).max() <= 1


@pytest.mark.parametrize("restart", [1, 10, 11, 20])
def test_emulated_passes(hz, restart):
    """The double-float form: the first update with the second pass's dots up to 10 vectors,
    separate launches above.  Iterations as in the FP64 form to within one; the residual bound
    1e-6 times the condition number (below 1e2 on this grid) bounds the error."""
    P = layered((24, 16), seed=6, pad=2)
    B = rhs(P["m"].size, 3, seed=4)
    Xref = O.direct_solve(P["H"], B)
    iters = []
    for outer in ("fp64", "emulated"):
        MG = hz.getMGparam(complex, int, 2, 1, 400, 1e-6, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0, precision="mixed",
                           outerArithmetic=outer)
        S = hz.getShiftedLaplacianMultigridSolver(hz_param(hz, P), MG, 0.5, "GMRES", restart)
        X, S = hz.solveLinearSystem(None, B, S)
        assert (S.last_relres <= 1e-6).all()
        iters.append(np.asarray(S.last_iters))
        assert np.linalg.norm(X - Xref) <= 1e-4 * np.linalg.norm(Xref)
    assert np.abs(iters[0] - iters[1]).max() <= 1

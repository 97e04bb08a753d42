"""Cycles that amplify (over-relaxed sweeps) under the FP32 K-cycle and its GMRES smoothing: the
stored basis vector's scale leaves the range in which FP32 values can be squared within one
restart.  FGMRES with any finite preconditioner leaves no residual above the right-hand
side's, so the solves end without convergence, finite and below 1."""
from __future__ import annotations

import numpy as np
import pytest

import problems as PB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relax,relax_from,w,restart", [("Jac", 0, 3.0, 30), ("Jac", 0, 10.0, 10), ("Jac", 0, 30.0, 10),
                                                        ("Jac", 0, 100.0, 10), ("Jac-GMRES", 1, 10.0, 20),
                                                        ("Jac-GMRES", 1, 30.0, 15)])
def test_amplifying_cycles_stay_finite(hz, relax, relax_from, w, restart):
    P = PB.layered((64, 64), seed=5, pad=8)
    B = PB.rhs(P["m"].size, 2, seed=2)
    MG = hz.getMGparam(complex, int, 4, 1, 3, 1e-6, relax, w, 1, 1, "K", "Julia", 0.5, 0.0, precision="mixed",
                       relaxFrom=relax_from)
    S = hz.getShiftedLaplacianMultigridSolver(PB.hz_param(hz, P), MG, 0.5, "GMRES", restart)
    X, S = hz.solveLinearSystem(None, B, S)
    assert np.isfinite(X).all()
    assert (S.last_relres < 1.0).all()
    assert list(S.last_iters) == [3 * restart] * 2

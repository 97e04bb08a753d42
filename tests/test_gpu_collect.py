"""Training pairs collected again from one solver with more columns: the workspace of
the 3D targets' two-step corrections has to follow the block's width."""
from __future__ import annotations

import numpy as np
import pytest

import problems as PB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relax", ["Jac", "Jac-GMRES"])
@pytest.mark.parametrize("cycle", ["V", "K"])
def test_collect_with_more_columns(hz, cycle, relax):
    P = PB.layered((16, 16, 16), seed=6, pad=3, ellipsoid=True)
    n = P["m"].size

    def solver():
        MG = hz.getMGparam(complex, int, 3, 1, 20, 1e-6, relax, 0.8, 1, 1, cycle, "Julia", 0.3, 0.0)
        return hz.getShiftedLaplacianMultigridSolver(PB.hz_param(hz, P), MG, 0.3, "GMRES", 10)

    def collect(S, nrhs):
        return hz.learned.collect_pairs(S, PB.rhs(n, nrhs, seed=nrhs), level=1, sweeps=4, max_pairs=40)

    S = solver()
    collect(S, 2)
    got, ref = collect(S, 5), collect(solver(), 5)
    for k in ("x", "t"):
        np.testing.assert_array_equal(got[k].cpu().numpy(), ref[k].cpu().numpy())
    np.testing.assert_array_equal(got["plain_err"], ref["plain_err"])
    assert got["target_relres"] == ref["target_relres"]

"""The operator product's integer-pipe route for large blocks (csrc/hz_fine_fixed.cu)
against the assembled sparse operators, node by node.

Bound: the device's diagonal is within 6 u of the oracle's (u = 2^-53), a native sum of
16 terms within 8 u of sum |a||x|.  In the integer sum a value is off by 2^-56 of a
reference at most 2^5 above the node's largest value (4 u of it), a coefficient by 2^-58 of
one at most 2^4 above it (1 u); of the products of two references up to five low
parts of 2^-58 are dropped (5 2^-58 2^9 over the four neighbours' coefficients or more: 20 u),
and the result is rounded (1 u).  Per component of a complex value less than 48 u times the
row's |a| times the largest component around the node."""
from __future__ import annotations

import numpy as np
import pytest

import scipy.sparse as sp

import problems as PB

pytestmark = pytest.mark.gpu
TOL = 48 * 2.0**-53

# tile edges 16 x 16 and 8 planes: below, at and above; the smallest grids; unequal spacings
GRIDS = [((1, 40), None), ((15, 15), None), ((16, 15), None), ((33, 17), [1.0, 0.7]), ((128, 96), None),
         ((1, 1, 2), None), ((15, 16, 7), None), ((17, 15, 8), [1.0, 0.9, 0.45]), ((33, 2, 9), None),
         ((9, 20, 30), [1.0, 1.1, 0.8]), ((4, 5, 6), [40.0, 1.0, 1.0])]


def columns(n, nrhs, rng):
    """Noise, noise that decays over the grid by 2^-200, an isolated point, zero, values
    near the limits of FP64, NaN and Inf; the rest noise."""
    X = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    X[:, 1] *= 2.0 ** -(200.0 * np.arange(n) / n)
    X[:, 2] = 0.0
    X[n // 2, 2] = 3.0 - 1e-30j
    X[:, 3] = 0.0
    X[:, 4] *= 1e-300
    X[:, 5] *= 1e290
    X[n // 3, 6] = complex(np.nan, 0.0)
    X[n // 3, 7] = complex(0.0, np.inf)
    X[:, 8] *= 2.0 ** rng.integers(-12, 1, n)
    return X


@pytest.mark.parametrize("order", [2, 1])
@pytest.mark.parametrize("cells,lengths", GRIDS, ids=lambda v: "x".join(map(str, v)) if v else "")
def test_large_blocks_match_oracle(hz, O, cells, lengths, order):
    P = PB.layered(cells, seed=2, pad=1, neumann=order == 2, lengths=lengths)
    n = P["m"].size
    nrhs = -(-(1 << 18) // n) + 3
    X = columns(n, nrhs, np.random.default_rng(n))
    Ho = PB.operator_from_parts(P, order)
    H = hz.GetHelmholtzOperator(PB.hz_param(hz, P), order)
    shift = hz.GetHelmholtzShiftOP(P["m"], P["w"], 0.5)
    S = sp.diags(0.5j * P["w"] ** 2 * P["m"])
    for A, Ao in ((H, Ho), (H + shift, Ho + S)):
        for op, oo in ((A, Ao.tocsr()), (A.H, Ao.conj().T.tocsr())):
            got = op @ X
            with np.errstate(all="ignore"):
                ref = oo @ X
            fin = np.isfinite(ref)
            np.testing.assert_array_equal(np.isfinite(got), fin)
            # the largest component among a row's values
            mag = np.where(np.isfinite(X), np.maximum(abs(X.real), abs(X.imag)), 0.0)
            row = np.asarray(abs(oo).sum(axis=1)).ravel()
            largest = np.zeros_like(mag)
            for r in range(n):
                largest[r] = mag[oo.indices[oo.indptr[r]:oo.indptr[r + 1]]].max(axis=0)
            bound = TOL * row[:, None] * largest + 1e-307
            with np.errstate(all="ignore"):
                d = got - ref
                bad = fin & ((abs(d.real) > bound) | (abs(d.imag) > bound))
            assert not bad.any(), (np.argwhere(bad)[:5], np.nanmax(np.where(fin, abs(d) / bound, 0)))



@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("cells", [(64, 32), (16, 12, 10)])
def test_cycle_on_large_blocks(hz, O, cells, adjoint):
    """The FP64 cycle's finest level: a block above the threshold against its first columns
    alone.  Both stop at a relative residual of 1e-10, so they differ by twice that times the
    condition number (below 1e3 here); rounding may move the last iteration by one."""
    P = PB.layered(cells, seed=3, pad=2)
    n = P["m"].size
    nrhs = -(-(1 << 17) // n)
    B = PB.rhs(n, nrhs, seed=1)

    def solve(C):
        MG = hz.getMGparam(complex, int, 2 if len(cells) == 3 else 3, 1, 200, 1e-10, "Jac", 0.8, 1, 1, "V", "Julia", 0.5,
                           0.0)
        S = hz.getShiftedLaplacianMultigridSolver(PB.hz_param(hz, P), MG, 0.5, "GMRES", 10)
        X, S = hz.solveLinearSystem(None, C, S, adjoint)
        assert (S.last_relres <= 1e-10).all()
        return X, np.asarray(S.last_iters)

    X, it = solve(B)
    Y, jt = solve(B[:, :3].copy())
    assert np.abs(it[:3] - jt).max() <= 1
    assert np.linalg.norm(X[:, :3] - Y) <= 2e-7 * np.linalg.norm(Y)

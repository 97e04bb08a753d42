"""The reference exponents of the operator's coefficients (csrc/hz_krylov.cu, k_fine_setup):
one node of 861 with a coefficient above all others, at the ends and in the middle of
warps, of blocks and of the last, partial warp.  Bound as in test_gpu_fine_fixed.py."""
from __future__ import annotations

import numpy as np
import pytest

import problems as PB

pytestmark = pytest.mark.gpu
TOL = 48 * 2.0**-53


@pytest.mark.parametrize("at", [0, 31, 32, 255, 256, 300, 831, 832, 850, 860])
def test_largest_coefficient_anywhere(hz, O, at):
    M = O.getRegularMesh([0.0, 40.0, 0.0, 20.0], [40, 20])  # unit spacing: the neighbours' coefficients are 1
    n = 861
    m = np.full(n, 1.5)
    m[at] = 50.0  # |diagonal| 8.5, one exponent above the others'
    P = dict(M=M, m=m, w=0.5, gamma=np.full(n, 0.005), neumann=True, sommerfeld=False)
    Ho = PB.operator_from_parts(P, 2)
    H = hz.GetHelmholtzOperator(PB.hz_param(hz, P))
    X = PB.rhs(n, 160, seed=at)  # 2^17 node-columns
    for A, Ao in ((H, Ho), (H.H, Ho.conj().T.tocsr())):
        d = A @ X - Ao @ X
        row = np.asarray(abs(Ao).sum(axis=1)).ravel()
        bound = TOL * row[:, None] * np.maximum(abs(X.real), abs(X.imag)).max(axis=0)
        assert (np.maximum(abs(d.real), abs(d.imag)) <= bound).all()

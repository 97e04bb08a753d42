"""The autotuner leaves the fine stencil's launch shape alone where the finest level runs on
the integer pipe, whose kernel does not know it: what it timed there was noise, which the
native kernel then used once columns had converged."""
from __future__ import annotations

import ctypes as C

import pytest

import problems as PB

pytestmark = pytest.mark.gpu


def test_integer_pipe_blocks_are_not_tuned(hz):
    P = PB.layered((128, 64), seed=7, pad=8)
    n = P["m"].size
    chosen = []
    for nrhs in range(16, 48):  # 2^17 node-columns and more
        MG = hz.getMGparam(complex, int, 3, 1, 1, 1e-1, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0)
        S = hz.getShiftedLaplacianMultigridSolver(PB.hz_param(hz, P), MG, 0.5, "GMRES", 2)
        hz.solveLinearSystem(None, PB.rhs(n, nrhs, seed=3), S)
        f, r = C.c_int32(), C.c_int32()
        assert hz._lib.load().hz_tune_info(S._handle, C.byref(f), C.byref(r)) == 0
        chosen.append(f.value)
    assert not any(chosen), chosen

"""Handles of two threads on one device whose kernels take unequal shared memory: every
call succeeds and returns what it returns alone."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import problems as PB

pytestmark = pytest.mark.gpu


def together(jobs, rounds):
    """Each job `rounds` times in a thread of its own; the results, or the first error."""
    out, errors, start = [[] for _ in jobs], [], threading.Barrier(len(jobs))

    def work(k):
        try:
            start.wait()
            for _ in range(rounds):
                out[k].append(jobs[k]())
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]
    return out


def test_band_solves(hz):
    """BiCGSTAB's coarsest levels of 45 and 1,105 nodes, launched one by one."""
    def job(cells, levels):
        P = PB.layered(cells, seed=3, pad=4)
        B = PB.rhs(P["m"].size, 2, seed=1)
        MG = hz.getMGparam(complex, int, levels, 1, 60, 1e-8, "Jac", 0.8, 1, 1, "V", "Julia", 0.5, 0.0)
        MG.cudaGraph = False
        S = hz.getShiftedLaplacianMultigridSolver(PB.hz_param(hz, P), MG, 0.5, "BiCGSTAB", 0)
        return lambda: np.array(hz.solveLinearSystem(None, B, S)[0])

    jobs = [job((32, 16), 3), job((64, 32), 2), job((128, 64), 2)]
    alone = [f() for f in jobs]
    for ref, got in zip(alone, together(jobs, 6)):
        for X in got:
            np.testing.assert_array_equal(X, ref)


def test_weight_gradients(hz):
    """Row lengths of 9 and 137 nodes; the FP32 sums of a gradient depend on the order of blocks:
    8,000 terms or fewer per weight, 2^-24 of their magnitudes each."""
    def job(grid, batch):
        net = hz.learned.CoarseNet(seed=4)
        rng = np.random.default_rng(5)
        x = rng.standard_normal((batch, *grid[::-1], 4)).astype(np.float32)
        t = rng.standard_normal((batch, *grid[::-1], 2)).astype(np.float32)
        return lambda: np.array(net.gradient(x, t)[1])

    jobs = [job((9, 9), 3), job((137, 17), 3)]
    alone = [f() for f in jobs]
    for ref, got in zip(alone, together(jobs, 200)):
        for g in got:
            assert np.linalg.norm(g - ref) <= 1e-3 * np.linalg.norm(ref)

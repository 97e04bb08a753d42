"""The networks' weight gradients (csrc/hz_wgrad.cu) and loss against the oracles
on grids around the kernel's steps: rows of 16- and 8-node steps, rows split into
segments (more than 144 nodes), single-row chunks, one sample and many."""
from __future__ import annotations

import numpy as np
import pytest

import coarse_net as CN
import coarse_net3d as CN3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,batch", [((9, 9), 1), ((17, 25), 3), ((25, 17), 40), ((33, 65), 2), ((153, 9), 2),
                                        ((9, 153), 1), ((289, 17), 1), ((9, 9), 5), ((17, 25, 1), 1), ((5, 5, 5), 1),
                                        ((13, 9, 17), 2), ((9, 5, 13), 9), ((149, 5, 5), 1), ((5, 5, 149), 1)])
@pytest.mark.parametrize("path", ["auto", "mma"])
def test_weight_gradient(hz, grid, batch, path):
    grid = tuple(n for n in grid if n > 1)
    dim = len(grid)
    oracle = CN3 if dim == 3 else CN
    net = (hz.learned.CoarseNet3D if dim == 3 else hz.learned.CoarseNet)(seed=4)
    net.set_conv_path(path)
    rng = np.random.default_rng(5)
    x = rng.standard_normal((batch, *grid[::-1], 4)).astype(np.float32)
    t = rng.standard_normal((batch, *grid[::-1], 2)).astype(np.float32)
    loss, grad = net.gradient(x, t)
    w = net.get_weights()
    y, cache = oracle.forward(w, x.astype(np.float64), emulate=True)
    lo, go = oracle.backward(cache, t.astype(np.float64))
    assert abs(loss - lo) <= 1e-3 * lo
    # per layer, relative L2: the bound of the networks' gradient tests (a rounding of
    # an activation to BF16 can flip with the order of an FP32 sum)
    for l, (a, b) in enumerate(zip(oracle.split(grad), oracle.split(go))):
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), l

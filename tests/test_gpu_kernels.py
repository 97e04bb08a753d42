"""Single launches against their definitions (kernel_checks.cu): the integer-pipe operator in
all its modes and inputs at the seams of its tiles, the band solve's two schedules bit for
bit, and the weight gradient on its own BF16 operands."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent
PKG = HERE.parent / "helmholtz.jl_gb300"


@pytest.fixture(scope="module")
def check(hz, tmp_path_factory):
    exe = tmp_path_factory.mktemp("checks") / "kernel_checks"
    r = subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                        "--expt-relaxed-constexpr", f"-I{PKG / 'csrc'}", f"-I{HERE.parent / 'include'}",
                        str(HERE / "kernel_checks.cu"), "-o", str(exe), f"-L{PKG}", "-lhelmgpu", "-Xlinker",
                        f"-rpath={PKG}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

    def run(*args):
        r = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True)
        assert r.returncode == 0, (args, r.stdout, r.stderr)

    return run


# tiles (choose_tile): 2D 15 x 68, 22 x 40, 23 x 44, 50 x 20; 3D 9 x 20, 14 x 16, 11 x 17, 15 x 14,
# planes by fours: two tiles or more along every axis, with remainders and without
@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("order", [2, 1])
@pytest.mark.parametrize("nodes,h", [((71, 203, 1), (1, 1, 1)), ((131, 77, 1), (1, 0.7, 1)), ((67, 131, 1), (1, 1, 1)),
                                     ((200, 333, 1), (0.01, 0.01, 1)), ((45, 39, 5), (1, 1, 1)),
                                     ((53, 47, 6), (1, 0.9, 0.8)), ((33, 33, 33), (0.01, 0.01, 0.01)),
                                     ((30, 70, 7), (1, 1, 0.8))])
def test_fine_operator(check, nodes, h, order, adjoint):
    check("fine", *nodes, order, adjoint, *h)


# below, at and above a warp's 32 entries and a cluster's 128 warps; windows of 2 x 17, 66, 131, 307
@pytest.mark.parametrize("rows,width,columns", [(4, 1, 1), (31, 17, 3), (289, 18, 1), (861, 42, 5), (2145, 66, 2),
                                                (1430, 131, 3), (2601, 307, 2)])
def test_band_schedules(check, rows, width, columns):
    check("band", rows, width, columns)


@pytest.mark.parametrize("grid,batch,channels", [((9, 9, 1), 1, (16, 8)), ((17, 25, 1), 3, (16, 16)),
                                                 ((33, 65, 1), 2, (128, 64)), ((153, 9, 1), 2, (64, 64)),
                                                 ((289, 17, 1), 1, (32, 32)), ((129, 33, 1), 1, (96, 32)),
                                                 ((5, 5, 5), 1, (16, 8)), ((13, 9, 17), 2, (48, 16)),
                                                 ((149, 5, 5), 1, (32, 16)), ((9, 5, 13), 3, (16, 32))])
def test_weight_gradient(check, grid, batch, channels):
    check("wgrad", *grid, batch, *channels)

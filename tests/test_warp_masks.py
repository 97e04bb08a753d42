"""Warp-synchronous code names its lanes: __activemask() is whatever subset of a warp
happens to run together there, so no kernel may take it for the set of lanes that a
reduction, a shuffle or a vote needs."""
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "helmholtz.jl_gb300" / "csrc"


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh")))
def test_no_activemask(src):
    assert "__activemask" not in (CSRC / src).read_text()

"""Sums run in the order in which they always ran: products, recurrences, eigen-pairs and Green's functions equal stored
values to the last bit (tests/golden/make_solver_values.py says why that matters, and what magnifies a last bit)."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))


@pytest.mark.parametrize("group", ["products", "pairs", "greens_functions", "solves"])
def test_values_to_the_last_bit(group):
    from edlib_gb300 import build
    build.build()
    import make_solver_values
    stored = np.load(os.path.join(HERE, "golden", "solver_values.npz"))
    off = []
    for name, value in make_solver_values.GROUPS[group]():
        x = stored[name]
        if x.shape != value.shape or not np.array_equal(x, value):
            off.append((name, "shape" if x.shape != value.shape else float(np.abs(x - value).max() / np.abs(x).max())))
    assert not off, off

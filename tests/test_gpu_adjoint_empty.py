"""Gradients of no parameter set at all: empty results, by every method, and the
arguments checked as ever.  In a process of its own: a division by the number of
sets ends it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import numpy as np
import ket_b200 as kb
from ket_b200.autograd import adjoint_expval
for n in (3, 11, 12, 16):
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.0)
    index = np.arange(n, dtype=np.int32)
    for precision in ("c64", "c128"):
        for method in ("auto", "per_gate", "tiled", "tiled_jit"):
            if method.startswith("tiled") and n < 12:
                continue
            v, g = adjoint_expval(c, index, np.zeros((0, n)), [(1.0, "Z" * n)], precision, method=method)
            assert v.shape == (0,) and g.shape == (0, n)
        try:
            adjoint_expval(c, index + 1, np.zeros((0, n)), [(1.0, "Z" * n)], precision)
        except Exception as e:
            assert "out of range" in str(e)
        else:
            raise AssertionError("an index beyond the parameters was taken")
"""


def test_no_sets():
    subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, check=True, timeout=300)

"""Block tables built on the device, at the edges of the gate staging.

Tolerances: an entry carries at most 4 roundings per gate (<= 129 gates, FP64);
complex128 1e-13, complex64 the suite's 1e-5 max-abs per amplitude.
"""
import numpy as np
import pytest

from test_gpu_parity import _block_circuit

pytestmark = pytest.mark.gpu

TOL = {"c128": 1e-13, "c64": 1e-5}


@pytest.mark.parametrize("count", [2, 31, 32, 33, 64, 65, 129])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("precision,tc", [("c128", True), ("c64", True), ("c64", False)])
def test_gate_counts(oracle, count, k, precision, tc):
    import ket_b200 as kb
    n = 13
    qs = list(range(3, 3 + k))
    ops = _block_circuit(n, qs, seed=count + k, depth=(count + 2) // 3)[:count]
    psi = np.random.default_rng(count).standard_normal((1 << n, 2)) @ np.array([1, 1j])
    psi /= np.linalg.norm(psi)
    st = kb.DeviceState(n, precision)
    st.from_numpy(psi)
    st.apply(ops, kb.make_options(precision, "greedy", k, tc))
    want = oracle.apply(n, psi, ops, fuse=0)
    assert np.abs(st.to_numpy() - want).max() < TOL[precision]


@pytest.mark.parametrize("n", [7, 11, 12, 13])
@pytest.mark.parametrize("precision", ["c128", "c64"])
def test_diagonal_tables(oracle, n, precision):
    """Diagonal runs with fewer, as many and more qubits than the table's bits."""
    import ket_b200 as kb
    g = np.random.default_rng(n)
    c = kb.Circuit(n)
    for i in range(n):
        c.rz(i, float(g.uniform(0, 6.2)))
        for j in range(i + 1, n):
            c.cp(i, j, float(g.uniform(0, 6.2)))
    psi = g.standard_normal((1 << n, 2)) @ np.array([1, 1j])
    psi /= np.linalg.norm(psi)
    st = kb.DeviceState(n, precision)
    st.from_numpy(psi)
    st.apply(c, kb.make_options(precision))
    assert np.abs(st.to_numpy() - oracle.apply(n, psi, c.to_ops(), fuse=0)).max() < TOL[precision]

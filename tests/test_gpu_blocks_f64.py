"""complex128 dense blocks on the FP64 matrix instructions against the oracle.

Tolerance: an output is a sum of 2^(k+1) products of a unit-norm state with
matrix entries that carry at most 4 roundings per gate (91 gates), so its
error is below (2^(k+1) + 4 * 91) * 2^-53 < 6e-14 for k <= 6; 1e-13 is used.
"""
import pytest

from test_gpu_parity import _block_circuit

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _targets(kind, n, k):
    if kind == "low":
        return list(range(k))
    if kind == "high":
        return list(range(n - k, n))
    if kind == "from1":  # qubit 0 a group bit, qubit 1 a target
        return list(range(1, k + 1))
    return sorted({0, 2, n - 1, n - 2, n // 2, n // 2 + 1})[:k] if kind == "mixed" else None


# n = k + 3: one column block; 13: fewer tiles than SMs; 19: the tile shrinks
# to 2^8 amplitudes; 21: the first size with full tiles
@pytest.mark.parametrize("kind", ["low", "high", "from1", "mixed"])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("size", ["least", 13, 19, 21])
def test_block_positions(oracle, size, k, kind):
    import numpy as np

    import ket_b200 as kb
    n = max(k, 3) + 3 if size == "least" else size
    qs = _targets(kind, n, k)
    if len(qs) != k:
        pytest.skip("the positions coincide at this size")
    ops = _block_circuit(n, qs, seed=17 * k + n, depth=30)
    rng = np.random.default_rng(n + k)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    plan = kb.Plan(n, ops, kb.make_options("c128", "greedy", k))
    assert [plan.pass_info(i)["kind"] for i in range(plan.stats()["n_passes"])] == [2]
    st = kb.DeviceState(n, "c128")
    st.from_numpy(psi)
    plan.execute(st)
    want = oracle.apply(n, psi, ops, fuse=0)
    assert np.abs(st.to_numpy() - want).max() < TOL

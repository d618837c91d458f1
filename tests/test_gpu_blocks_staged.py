"""Tensor-core blocks whose output goes through shared memory (qubit 0 a target,
or lanes spread thin), and those that fetch tiles without a tensor copy: the
highest target among a thread's bits and among its chunks, one tile to
several per slot.

Tolerance: an output is a row of a unitary (norm 1) times 2^k amplitudes, each
product good to 2^-21 of its largest, so it is off by less than
2^-21 2^(k/2) max|psi| a block; two blocks and the norm pass: 2^-15 max|psi|.
"""
import numpy as np
import pytest

from test_gpu_parity import _block_circuit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,first,second", [
    (13, [0, 1, 2, 3, 4, 5], [0, 3, 6, 8, 10, 12]),
    (14, [0, 5, 7, 11, 12, 13], [1, 2, 3, 4, 8, 9]),
    (22, [0, 1, 2, 3, 4, 5], [0, 6, 13, 15, 17, 21]),
    (22, [1, 4, 7, 16, 19, 21], [6, 9, 12, 14, 17, 19]),
    (12, [0, 1, 2, 3, 4], [0, 2, 5, 9, 11]),
    (21, [1, 3, 4, 8, 11], [0, 3, 4, 13, 20]),
    (20, [8, 10, 12, 14, 16], [2, 9, 11, 14, 18]),
    (11, [0, 1, 2, 3], [1, 2, 9, 10]),
    (20, [0, 4, 9, 19], [1, 5, 11, 13]),
])
def test_block_pairs(oracle, n, first, second):
    import ket_b200 as kb
    k = len(first)
    ops = np.concatenate([_block_circuit(n, qs, seed=n + qs[-1], depth=8) for qs in (first, second)])
    opt = kb.make_options("c64", "greedy", k, True)
    plan = kb.Plan(n, ops, opt)
    blocks = [i for i in range(plan.stats()["n_passes"]) if plan.pass_info(i)["tensor"]]
    assert [list(plan.pass_qubits(i)) for i in blocks] == [first, second]
    psi = np.random.default_rng(n).standard_normal((1 << n, 2)) @ np.array([1, 1j])
    psi /= np.linalg.norm(psi)
    st = kb.DeviceState(n, "c64")
    st.from_numpy(psi)
    plan.execute(st)
    want = oracle.apply(n, psi, ops, fuse=0)
    assert np.abs(st.to_numpy() - want).max() < 2.0 ** -15 * np.abs(psi).max()

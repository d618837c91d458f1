"""Runs from |0...0> touch only the amplitudes that can be nonzero; they must
give what a run over the whole state gives.

Tolerances: those of the parity tests (complex128 1e-12, complex64 1e-5 max-abs
per amplitude).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"c128": 1e-12, "c64": 1e-5}


def _circuit(n, qubits, seed, gates=40):
    """Gates of every kind on growing prefixes of `qubits`."""
    import ket_b200 as kb
    g = np.random.default_rng(seed)
    c = kb.Circuit(n)
    c.cx(qubits[0], qubits[-1])  # control still zero
    c.swap(qubits[0], qubits[1])
    c.cz(qubits[0], qubits[2])
    for i in range(gates):
        top = 3 + (len(qubits) - 3) * i // gates
        a, b, t = (int(q) for q in g.permutation(qubits[:top + 1])[:3])
        th = float(g.uniform(0, 2 * math.pi))
        name = ["u", "cx", "swap", "ccx", "cswap", "rz", "cp", "t", "h", "cry"][int(g.integers(0, 10))]
        args = {"u": (a, th, 1.1, 0.3), "cx": (a, b), "swap": (a, b), "ccx": (a, b, t), "cswap": (a, b, t),
                "rz": (a, th), "cp": (a, b, th), "t": (a,), "h": (a,), "cry": (a, b, th)}[name]
        getattr(c, name)(*args)
    return c


MODES = [("c128", "greedy", 0, True), ("c128", "none", 0, True), ("c128", "greedy", 3, True),
         ("c128", "greedy", 6, True), ("c64", "greedy", 0, True), ("c64", "greedy", 4, True),
         ("c64", "greedy", 0, False), ("c64", "none", 0, True), ("c64", "reference", 0, True)]


@pytest.mark.parametrize("n,order", [(4, "up"), (9, "down"), (13, "up"), (14, "mixed"), (18, "down"), (19, "mixed")])
def test_growing_circuits(oracle, n, order):
    import ket_b200 as kb
    qs = list(range(n))
    if order == "down":
        qs = qs[::-1]
    elif order == "mixed":
        qs = [int(q) for q in np.random.default_rng(n).permutation(n)]
    first, second = _circuit(n, qs[: max(4, n // 2)], n), _circuit(n, qs, n + 1)
    ops = np.concatenate([first.to_ops(), second.to_ops()])
    want = oracle.run(n, ops, fuse=0)
    for precision, fusion, k, tc in MODES:
        opt = kb.make_options(precision, fusion, k, tc)
        st = kb.DeviceState(n, precision)
        st.apply(first, opt)  # leaves qubits inactive for the second
        st.apply(second, opt)
        assert np.abs(st.to_numpy() - want).max() < TOL[precision], (precision, fusion, k, tc)


@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_writes_through_an_earlier_view(oracle, precision):
    """A tensor view taken before a reset still writes the state."""
    import torch

    import ket_b200 as kb
    n = 14
    c = _circuit(n, [5, 6, 7, 8, 9], 3)
    psi = np.random.default_rng(1).standard_normal(1 << n) + 0j
    psi /= np.linalg.norm(psi)
    st = kb.DeviceState(n, precision)
    view = st.torch_view()
    plan = kb.Plan(n, c.to_ops(), kb.make_options(precision))
    for _ in range(2):
        st.reset()
        plan.execute(st)  # |0...0>
        assert np.abs(st.to_numpy() - oracle.run(n, c.to_ops(), fuse=0)).max() < TOL[precision]
        st.reset()
        view.copy_(torch.from_numpy(psi))
        torch.cuda.synchronize()
        plan.execute(st)
        assert np.abs(st.to_numpy() - oracle.apply(n, psi, c.to_ops(), fuse=0)).max() < TOL[precision]


def test_non_finite_parameters_reach_every_amplitude():
    import ket_b200 as kb
    n = 13
    c = kb.Circuit(n)
    c.rx(0, math.inf)
    for q in range(1, 4):
        c.h(q)
    got = {}
    for start in ("ground", "uploaded"):
        st = kb.DeviceState(n, "c128")
        if start == "uploaded":
            e0 = np.zeros(1 << n, dtype=np.complex128)
            e0[0] = 1
            st.from_numpy(e0)
        st.apply(c, kb.make_options("c128"))
        got[start] = np.isnan(st.to_numpy())
    assert np.array_equal(got["ground"], got["uploaded"]) and got["ground"].all()

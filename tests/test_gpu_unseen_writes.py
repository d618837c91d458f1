"""Amplitudes written without a call of the library, after a reset: through a
tensor view taken earlier, or before a replay of a captured plan.  A complex64
plan with tensor-core blocks restores the norm it finds, not that of |0...0>.

Tolerances: 1e-5 max-abs per amplitude of a state of norm 1 (the parity tests'),
so 2e-5 for one of norm 4 (amplitudes twice as large); the norm itself to 1e-6
of its value (FP32 rounding of the rescaled amplitudes, 2^-24 each).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(n):
    g = np.random.default_rng(n)
    psi = g.standard_normal(1 << n) + 1j * g.standard_normal(1 << n)
    return 2.0 * psi / np.linalg.norm(psi)


# 14 qubits: below the size of the check for |0...0>; 20: at it
@pytest.mark.parametrize("n", [14, 20])
def test_norm_of_a_state_written_through_an_earlier_view(oracle, n):
    import torch

    import ket_b200 as kb
    from ket_b200.workloads import random_brickwork
    c = random_brickwork(n, 4, seed=n)
    plan = kb.Plan(n, c.to_ops(), kb.make_options("c64"))
    psi = _start(n)
    want = oracle.apply(n, psi.copy(), c.to_ops(), fuse=0)
    st = kb.DeviceState(n, "c64")
    view = st.torch_view()
    for _ in range(2):
        st.reset()
        plan.execute(st)
        assert abs(st.norm() - 1.0) < 1e-6
        st.reset()
        view.copy_(torch.from_numpy(psi))
        torch.cuda.synchronize()
        plan.execute(st)
        assert abs(st.norm() / 4.0 - 1.0) < 1e-6
        assert np.abs(st.to_numpy() - want).max() < 2e-5


@pytest.mark.parametrize("n", [14, 20])
def test_norm_of_a_state_that_a_replay_finds(oracle, n):
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    from ket_b200.workloads import random_brickwork
    c = random_brickwork(n, 4, seed=n)
    plan = kb.Plan(n, c.to_ops(), kb.make_options("c64"))
    psi = _start(n)
    st = kb.DeviceState(n, "c64")
    plan.execute(st)  # builds the plan's tables
    st.reset()
    stream = torch.cuda.ExternalStream(_lib.lib.ketgpu_state_stream(st.handle))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        plan.execute(st, sync=False)
    for start in (None, psi):
        st.reset()
        scale = 1.0
        if start is not None:
            st.from_numpy(start)
            scale = 4.0
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        assert abs(st.norm() / scale - 1.0) < 1e-6
        e0 = np.zeros(1 << n, dtype=np.complex128)
        e0[0] = 1
        want = oracle.apply(n, e0 if start is None else start.copy(), c.to_ops(), fuse=0)
        assert np.abs(st.to_numpy() - want).max() < 2e-5


@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_execute_waits_for_nothing(precision):
    """After a reset a plan on a state whose address was handed out is enqueued
    behind what the stream still does."""
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    from ket_b200.workloads import random_brickwork
    n = 21
    plan = kb.Plan(n, random_brickwork(n, 4, seed=1).to_ops(), kb.make_options(precision))
    st = kb.DeviceState(n, precision)
    plan.execute(st)  # builds the plan's tables
    want = st.to_numpy()
    st.torch_view()
    stream = torch.cuda.ExternalStream(_lib.lib.ketgpu_state_stream(st.handle))
    st.reset()
    plan.execute(st)
    st.reset()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(10**9)  # about half a second
        slept = torch.cuda.Event()
        slept.record(stream)
    plan.execute(st, sync=False)
    assert not slept.query()
    assert np.array_equal(st.to_numpy(), want)


MODES = [("c128", "greedy", 0, True), ("c128", "none", 0, True), ("c64", "greedy", 0, True),
         ("c64", "greedy", 4, True), ("c64", "greedy", 0, False), ("c64", "none", 0, True),
         ("c64", "reference", 0, True)]


@pytest.mark.parametrize("n", [19, 20, 21])
def test_every_kind_of_pass_after_unseen_writes(oracle, n):
    """Passes of every kind on a state that is |0...0> after a reset, and on one
    that was written since: each takes its part of the state on the device."""
    import torch

    import ket_b200 as kb
    g = np.random.default_rng(n)
    c = kb.Circuit(n)
    c.cx(0, n - 1)  # the control is zero
    c.cz(0, 2)
    c.swap(1, 3)
    for i in range(40):
        top = 3 + (n - 3) * i // 40
        a, b, t = (int(q) for q in g.permutation(top + 1)[:3])
        th = float(g.uniform(0, 6.28))
        name = ["u", "cx", "swap", "ccx", "cswap", "rz", "cp", "t", "h", "cry"][int(g.integers(0, 10))]
        args = {"u": (a, th, 1.1, 0.3), "cx": (a, b), "swap": (a, b), "ccx": (a, b, t), "cswap": (a, b, t),
                "rz": (a, th), "cp": (a, b, th), "t": (a,), "h": (a,), "cry": (a, b, th)}[name]
        getattr(c, name)(*args)
    for i in range(n):  # a run of diagonal gates
        c.cp(i, (i + 5) % n, 0.1 * i)
    psi = _start(n)
    clean = oracle.run(n, c.to_ops(), fuse=0)
    written = oracle.apply(n, psi.copy(), c.to_ops(), fuse=0)
    for precision, fusion, k, tc in MODES:
        plan = kb.Plan(n, c.to_ops(), kb.make_options(precision, fusion, k, tc))
        st = kb.DeviceState(n, precision)
        view = st.torch_view()
        tol = 2e-5 if precision == "c64" else 2e-12
        for start, want in ((None, clean), (psi, written), (None, clean)):
            st.reset()
            if start is not None:
                view.copy_(torch.from_numpy(start))
                torch.cuda.synchronize()
            plan.execute(st)
            assert np.abs(st.to_numpy() - want).max() < tol, (precision, fusion, k, tc, start is None)
        plan.close()
        st.close()

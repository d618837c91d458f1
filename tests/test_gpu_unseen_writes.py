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

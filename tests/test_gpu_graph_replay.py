"""A plan captured into a CUDA graph: its replays write the state without a
call of the library, and what runs afterwards must see all of it.

Tolerances: those of the parity tests (complex128 1e-12, complex64 1e-5 max-abs
per amplitude).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"c128": 1e-12, "c64": 1e-5}


# 14 qubits: everything below the size of the check for |0...0>; 20: above it
@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n", [14, 20])
def test_runs_after_a_replay(oracle, n, precision):
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    from ket_b200.workloads import random_brickwork
    opt = kb.make_options(precision)
    first = random_brickwork(n, 4, seed=n)
    second = kb.Circuit(n)  # stays on a few qubits
    for q in range(3):
        second.ry(q, 0.3 + q)
        second.cx(q, q + 1)
    second.cz(n - 2, n - 1)
    st = kb.DeviceState(n, precision)
    plan = kb.Plan(n, first.to_ops(), opt)
    plan.execute(st)  # builds the plan's tables
    stream = torch.cuda.ExternalStream(_lib.lib.ketgpu_state_stream(st.handle))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        plan.execute(st, sync=False)
    once = oracle.run(n, first.to_ops(), fuse=0)
    want = oracle.apply(n, once.copy(), second.to_ops(), fuse=0)
    for _ in range(2):
        st.reset()
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        assert np.abs(st.to_numpy() - once).max() < TOL[precision]
        st.apply(second, opt)
        assert np.abs(st.to_numpy() - want).max() < TOL[precision]

"""Draws after the replays of a captured plan are of the state that they left.

x on every qubit takes |0...0> to |1...1> and back: every draw is exact.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n", [4, 14, 20])  # 4: no tree
def test_draws_after_a_replay(n, precision):
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    c = kb.Circuit(n)
    for q in range(n):
        c.x(q)
    st = kb.DeviceState(n, precision)
    plan = kb.Plan(n, c.to_ops(), kb.make_options(precision))
    plan.execute(st)  # builds the plan's tables
    stream = torch.cuda.ExternalStream(_lib.lib.ketgpu_state_stream(st.handle))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        plan.execute(st, sync=False)
    u = np.array([0.0, 0.5, 0.999])
    st.reset()
    for replays in range(4):
        want = (1 << n) - 1 if replays % 2 else 0
        assert (st.sample(u) == want).all()
        assert (st.sample_seeded(3, 3000) == want).all()
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()

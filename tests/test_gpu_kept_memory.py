"""What the library keeps between calls is given back before an allocation
fails: with the device nearly full, each kind of call that needs more than is
left takes the room of idle memory.  Results are those of the same call on an
empty device, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEFT = 32 << 20  # bytes left on the device


@pytest.fixture
def full():
    """Fills the device up to LEFT bytes; gives all of it back at the end."""
    import torch

    from ket_b200 import _lib
    held = []

    def fill():
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        held.append(torch.empty(max(free - LEFT, 1), dtype=torch.uint8, device="cuda"))
        assert torch.cuda.mem_get_info()[0] <= LEFT

    yield fill
    held.clear()
    torch.cuda.empty_cache()
    _lib.check(_lib.lib.ketgpu_release_cache())


def _keep_workspace():
    """An adjoint call whose 2.4 GB of states are kept."""
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    c = kb.Circuit(24)
    for q in range(24):
        c.ry(q, 0.0)
    adjoint_expval(c, np.arange(24, dtype=np.int32), np.full((6, 24), 0.3), [(1.0, "Z" * 24)], "c64")


def _keep_idle_states():
    import ket_b200 as kb
    states = [kb.DeviceState(22, "c128") for _ in range(4)]
    for s in states:
        s.close()


def _sampling_tree():
    import ket_b200 as kb
    st = kb.DeviceState(28, "c64")
    c = kb.Circuit(28)
    for q in range(28):
        c.ry(q, 0.1 * (q + 1))
    st.apply(c, kb.make_options("c64"))
    u = np.linspace(0.001, 0.999, 1000)
    return st, lambda: st.sample(u)  # a tree of 69 MB


def _scratch():
    import ket_b200 as kb
    n, terms = 27, 60000  # 60,000 x 296 partial sums: 142 MB
    st = kb.DeviceState(n, "c64")
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.1 * (q + 1))
    st.apply(c, kb.make_options("c64"))
    obs = [(1.0 / terms, format(t * 1777 % (1 << n), f"0{n}b").replace("0", "I").replace("1", "Z"))
           for t in range(terms)]
    return st, lambda: st.expval(obs)


def _tables():
    import ket_b200 as kb
    from ket_b200.workloads import random_brickwork
    ops = random_brickwork(14, 4000, seed=1).to_ops()
    opt = kb.make_options("c128", "greedy", 6)
    st = kb.DeviceState(14, "c128")

    def run():
        plan = kb.Plan(14, ops, opt)  # its tables are made at its first execution
        kinds = [plan.pass_info(i) for i in range(int(plan.stats()["n_passes"]))]
        assert sum(16 * 4 ** p["k"] for p in kinds if p["kind"] == 2) > 128 << 20
        st.reset()
        plan.execute(st)
        plan.close()
        return st.to_numpy()
    return st, run


def _workspace():
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    n = 20
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.0)
    theta = np.linspace(-1, 1, 2 * n).reshape(2, n)  # 50 MB of states

    def run():
        v, g = adjoint_expval(c, np.arange(n, dtype=np.int32), theta, [(1.0, "Z" * n)], "c64")
        return np.concatenate([v, g.ravel()])
    return None, run


@pytest.mark.parametrize("keep,make", [(_keep_workspace, _sampling_tree), (_keep_workspace, _scratch),
                                       (_keep_workspace, _tables), (_keep_idle_states, _workspace)])
def test_idle_memory_is_given_back(full, keep, make):
    from ket_b200 import _lib
    st, call = make()
    want = call()
    if st is not None and make is _sampling_tree:
        st.close()  # the tree lives with the state
        _lib.check(_lib.lib.ketgpu_release_cache())
        st, call = make()
    _lib.check(_lib.lib.ketgpu_release_cache())
    keep()
    full()
    assert np.array_equal(call(), want)
    if st is not None:
        st.close()

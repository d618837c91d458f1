"""Draws whose uniforms are made on the device: the outcomes of the host's
std::mt19937 stream, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2048: the first count with device uniforms; 2156 and 2157: the last word of
# a 454-word step and the first of the next; 1: far below
@pytest.mark.parametrize("count", [1, 2047, 2048, 2156, 2157, 30000, 1000001])
@pytest.mark.parametrize("seed", [0, 42, 4294967295])
@pytest.mark.parametrize("n,precision", [(3, "c64"), (11, "c128"), (17, "c64")])
def test_same_outcomes(n, precision, count, seed):
    import ket_b200 as kb
    rng = np.random.default_rng(n)
    psi = rng.standard_normal((1 << n, 2)) @ np.array([1, 1j])
    st = kb.DeviceState(n, precision)
    st.from_numpy(psi / np.linalg.norm(psi))
    assert np.array_equal(st.sample_seeded(seed, count), st.sample(kb.uniforms(seed, count)))
    # after a change of the state that the stream has not finished yet
    c = kb.Circuit(n)
    c.x(n - 1)
    plan = kb.Plan(n, c.to_ops(), kb.make_options(precision, "none"))
    plan.execute(st, sync=False)
    got = st.sample_seeded(seed, count)
    assert np.array_equal(got, st.sample(kb.uniforms(seed, count)))

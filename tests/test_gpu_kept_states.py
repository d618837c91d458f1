"""A destroyed state's memory is used again only when nothing reads it any more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_work_of_other_streams_on_a_destroyed_state(precision):
    """A copy of the amplitudes, enqueued on a stream of the caller's own
    before the state is destroyed, is of that state and not of the next."""
    import torch

    import ket_b200 as kb
    n = 16
    other = torch.cuda.Stream()
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.2 + q)
    for _ in range(2):
        st = kb.DeviceState(n, precision)
        st.apply(c, kb.make_options(precision))
        want = st.to_numpy_raw()
        with torch.cuda.stream(other):
            torch.cuda._sleep(2 * 10**8)  # about a tenth of a second
            copy = st.torch_view().clone()
        st.close()
        following = kb.DeviceState(n, precision)  # |0...0>
        assert following.to_numpy()[0] == 1
        torch.cuda.synchronize()
        assert np.array_equal(copy.cpu().numpy(), want)
        following.close()

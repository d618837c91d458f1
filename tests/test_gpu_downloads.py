"""Downloads of every size class, and states made from kept memory: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 4 MB: the first staged size; 64 MB: the staging buffers, above them the ring
@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n", [3, 17, 18, 19, 22, 23, 24])
def test_amplitudes_arrive(n, precision):
    import torch

    import ket_b200 as kb
    st = kb.DeviceState(n, precision)
    v = torch.view_as_real(st.torch_view())
    v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape))  # exact in FP32 up to 2^24, rounded beyond
    torch.cuda.synchronize()
    want = torch.view_as_complex(v).cpu().numpy()
    dim = 1 << n
    assert np.array_equal(st.to_numpy_raw(), want)
    assert np.array_equal(st.to_numpy(), want.astype(np.complex128))
    for first, count in ((0, 0), (1, dim - 1), (dim // 3, dim // 2), (dim - 1, 1)):
        assert np.array_equal(st.to_numpy(first, count), want[first:first + count].astype(np.complex128))
        assert np.array_equal(st.to_numpy_raw(first, count), want[first:first + count])


def test_reused_states_start_clean():
    import ket_b200 as kb
    c = kb.Circuit(12)
    for q in range(12):
        c.h(q)
    for _ in range(20):  # more than are kept
        states = [kb.run_device(c, p) for p in ("c64", "c128")]
        for s in states:
            s.sample(np.array([0.5]))
            s.close()
        for p in ("c64", "c128"):
            s = kb.DeviceState(12, p)
            a = s.to_numpy()
            assert a[0] == 1 and not a[1:].any()
            assert list(s.sample(np.array([0.0, 0.999]))) == [0, 0]
            s.close()

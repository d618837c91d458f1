"""Downloads through staging buffers of other shapes (environment, read once a
process): ranges around what the buffers hold, exact."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import numpy as np, torch
import ket_b200 as kb
n = 21
for precision, amp in (("c64", 8), ("c128", 16)):
    st = kb.DeviceState(n, precision)
    v = torch.view_as_real(st.torch_view())
    v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape))
    torch.cuda.synchronize()
    want = torch.view_as_complex(v).cpu().numpy()
    for mb in (2, 3, 4, 5):
        for count in (mb * 2**20 // amp + d for d in (-1, 0, 1)):
            for first in (0, 3):
                w = want[first:first + count]
                assert np.array_equal(st.to_numpy(first, count), w.astype(np.complex128)), (precision, mb, count)
                assert np.array_equal(st.to_numpy_raw(first, count), w), (precision, mb, count)
    assert np.array_equal(st.to_numpy(), want.astype(np.complex128))
"""


@pytest.mark.parametrize("ring", [2, 3, 4])
def test_ranges_around_the_buffers(ring):
    env = dict(os.environ, KETGPU_DOWN_CHUNK_MB="1", KETGPU_DOWN_RING=str(ring))
    subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, check=True, timeout=300)

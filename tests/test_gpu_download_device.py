"""complex128 amplitudes into a buffer on the device: the copy there as it is,
whatever its size.  In a process of its own: written to by the host, such a
buffer ends it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import numpy as np, torch
import ket_b200 as kb
from ket_b200 import _lib
for n in (16, 18, 21, 23):  # 1 MB, 4 MB (the first staged size), 32 MB, 128 MB
    st = kb.DeviceState(n, "c128")
    v = torch.view_as_real(st.torch_view())
    v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape))
    out = torch.zeros_like(v)
    torch.cuda.synchronize()
    _lib.check(_lib.lib.ketgpu_state_download(st.handle, 0, 1 << n, out.data_ptr()))
    assert torch.equal(out, v)
    out.zero_()
    torch.cuda.synchronize()
    _lib.check(_lib.lib.ketgpu_state_download_raw(st.handle, 0, 1 << n, out.data_ptr()))
    assert torch.equal(out, v)
st = kb.DeviceState(12, "c64")
count = 1 << 20  # 8 MB of draws
draws = torch.ones(count, dtype=torch.int64, device="cuda")
torch.cuda.synchronize()
_lib.check(_lib.lib.ketgpu_sample_seeded(st.handle, 1, count, draws.data_ptr()))
assert not draws.any()
"""


def test_device_buffers():
    subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, check=True, timeout=300)

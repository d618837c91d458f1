"""Downloads and their helper threads: none to be had, a stream with other work
ahead, several downloads at once, page-locked buffers."""
import os
import subprocess
import sys
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int left_to_start = 1 << 30;
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* p) {
  static int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  if (!real) real = dlsym(RTLD_NEXT, "pthread_create");
  if (__sync_fetch_and_sub(&left_to_start, 1) <= 0) return EAGAIN;
  return real(t, a, f, p);
}
"""

CHILD = """
import ctypes, sys
import numpy as np, torch
import ket_b200 as kb
left = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "left_to_start")
for n, precision in ((19, "c64"), (19, "c128"), (22, "c128"), (23, "c64"), (23, "c128")):
    st = kb.DeviceState(n, precision)
    v = torch.view_as_real(st.torch_view())
    v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape))
    want = torch.view_as_complex(v).cpu().numpy()
    first = st.to_numpy()
    for threads in (0, 1, 3):
        left.value = threads
        got = st.to_numpy()
        raw = st.to_numpy_raw()
        left.value = 1 << 30
        assert np.array_equal(first, want.astype(np.complex128)) and np.array_equal(got, first)
        assert np.array_equal(raw, want)
"""


def test_without_threads_to_start(tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(tmp_path / "shim.c"), "-o", so, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=so)
    subprocess.run([sys.executable, "-c", CHILD, so], cwd=ROOT, env=env, check=True, timeout=300)


@pytest.mark.parametrize("n", [21, 23])  # 32 MB: all pieces at once; 128 MB: the ring
def test_helpers_do_not_spin_behind_other_work(n):
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    st = kb.DeviceState(n, "c128")
    st.to_numpy()
    stream = torch.cuda.ExternalStream(_lib.lib.ketgpu_state_stream(st.handle))
    with torch.cuda.stream(stream):
        torch.cuda._sleep(10**9)  # about half a second
    cpu, wall = time.process_time(), time.perf_counter()
    st.to_numpy()
    cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
    assert wall > 0.3
    # the calling thread's wait and the copy itself; a single helper that spun
    # beside it would double the first
    assert cpu < 1.5 * wall


def test_downloads_at_once():
    import torch

    import ket_b200 as kb
    states, want = [], []
    for i, (n, precision) in enumerate([(21, "c128"), (21, "c64"), (22, "c128"), (23, "c64")]):
        st = kb.DeviceState(n, precision)
        v = torch.view_as_real(st.torch_view())
        v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape) + i)
        states.append(st)
        want.append(torch.view_as_complex(v).cpu().numpy())
    bad = []

    def read(i):
        for _ in range(5):
            if not np.array_equal(states[i].to_numpy_raw(), want[i]):
                bad.append(i)
            if not np.array_equal(states[i].to_numpy(), want[i].astype(np.complex128)):
                bad.append(i)

    threads = [threading.Thread(target=read, args=(i,)) for i in range(len(states))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("n", [17, 21, 23])
def test_page_locked_buffers(n):
    import torch

    import ket_b200 as kb
    from ket_b200 import _lib
    st = kb.DeviceState(n, "c128")
    v = torch.view_as_real(st.torch_view())
    v.copy_(torch.arange(v.numel(), device="cuda").reshape(v.shape))
    torch.cuda.synchronize()
    out = torch.zeros((1 << n, 2), dtype=torch.float64).pin_memory()
    _lib.check(_lib.lib.ketgpu_state_download(st.handle, 0, 1 << n, out.data_ptr()))
    assert torch.equal(out, v.cpu())

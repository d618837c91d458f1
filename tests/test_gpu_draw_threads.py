"""Several threads that draw from one state at once, its tree and second stream
not made yet: every draw as by one thread alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n", [8, 16])
def test_draws_at_once(n, precision):
    import ket_b200 as kb
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.3 + q)
    opt = kb.make_options(precision)
    alone = kb.DeviceState(n, precision)
    alone.apply(c, opt)
    want = [alone.sample_seeded(seed, 5000) for seed in range(4)]
    bad = []
    for _ in range(20):
        st = kb.DeviceState(n, precision)
        st.apply(c, opt)
        gate = threading.Barrier(len(want))

        def work(seed):
            try:
                gate.wait()
                for _ in range(3):
                    if not np.array_equal(st.sample_seeded(seed, 5000), want[seed]):
                        bad.append((seed, "other draws"))
            except Exception as e:  # reported below, on the main thread
                bad.append((seed, repr(e)))

        threads = [threading.Thread(target=work, args=(seed,)) for seed in range(len(want))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
    alone.close()

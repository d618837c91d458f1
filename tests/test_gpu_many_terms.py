"""Pauli sums of very many terms: time in proportion, values unchanged."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_terms_of_one_flip():
    """Terms that differ in their Z's alone: four times the terms take about
    four times as long (10 times when each searched through the groups of all
    before it)."""
    import ket_b200 as kb
    n = 20
    st = kb.DeviceState(n, "c128")
    c = kb.Circuit(n)
    for q in range(n):
        c.ry(q, 0.2 + q)
    st.apply(c, kb.make_options("c128"))

    def seconds(terms):
        s = np.random.default_rng(terms).integers(0, 1 << (n - 1), terms)
        obs = [(1.0, "X" + format(int(v), f"0{n - 1}b").replace("0", "I").replace("1", "Z")) for v in s]
        t0 = time.perf_counter()
        st.expval(obs)
        return time.perf_counter() - t0

    seconds(1000)
    small = min(seconds(40000) for _ in range(2))
    assert seconds(160000) < 6.5 * small
    # a product state: <Z> = cos, <X> = sin of its angles; FP64 sums of 2^20
    # products, far inside 1e-12
    a = [0.2 + q for q in range(n)]
    for p, want in (("X" + "I" * (n - 2) + "Z", np.sin(a[n - 1]) * np.cos(a[0])),
                    ("X" + "Z" + "I" * (n - 2), np.sin(a[n - 1]) * np.cos(a[n - 2]))):
        got = st.expval([(1.0, "X" + "I" * (n - 1))] * 5 + [(0.0, p)] * 3 + [(1.0, p)])
        assert abs(got - 5 * np.sin(a[n - 1]) - want) < 1e-12

"""Gradients of several sizes at once, a thread each: every call gives what it
gives alone, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_sizes_at_once(precision):
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval

    def problem(n):
        c = kb.Circuit(n)
        for q in range(n):
            c.ry(q, 0.0)
        for q in range(n - 1):
            c.cx(q, q + 1)
        index = np.array(list(range(n)) + [-1] * (n - 1), dtype=np.int32)
        theta = np.linspace(-1.0, 1.0, 2 * n).reshape(2, n)
        return c, index, theta, [(0.5, "Z" * n), (0.25, "X" * n)], precision

    # shared memory for the states of 11 qubits, of 10, and next to none
    problems = [problem(n) for n in (11, 10, 3, 2)]
    want = [adjoint_expval(*p) for p in problems]
    bad = []

    def work(i):
        try:
            for _ in range(400):
                values, grads = adjoint_expval(*problems[i])
                if not (np.array_equal(values, want[i][0]) and np.array_equal(grads, want[i][1])):
                    bad.append((i, "another result"))
        except Exception as e:  # reported below, on the main thread
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(problems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad

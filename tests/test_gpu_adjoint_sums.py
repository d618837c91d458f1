"""Gate matrices and gradient sums made on the device: every parameterised
gate, parameters shared by several gates and used by none, batches.

Tolerances: those of the adjoint tests (complex128 1e-9, complex64 1e-5
against the FP64 adjoint).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"c128": 1e-9, "c64": 1e-5}


@pytest.mark.parametrize("n", [3, 11, 12, 13])  # per gate; the first sizes of the tiled sweeps
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_shared_parameters(oracle, n, batch, precision):
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    c, index = kb.Circuit(n), []
    g = np.random.default_rng(n)

    def add(name, qs, par, *fixed):
        getattr(c, name)(*qs, *([0.0] if par >= 0 else []), *fixed)
        index.append(par)

    for q in range(n):
        add("h", (q,), -1)
    for layer in range(2):
        for q in range(n):
            a, b = q, (q + 1) % n
            name, par = [("rx", 0), ("ry", 1), ("rz", 2), ("crx", 0), ("cry", 3), ("crz", 2), ("cp", 4)][(q + 3 * layer) % 7]
            add(name, (a,) if len(name) == 2 and name != "cp" else (a, b), par)
            if q % 3 == 0:
                add("t", (b,), -1)
            if q % 4 == 1:
                add("cx", (b, a), -1)
        c.barrier()
        index.append(-1)
    nparams = 6  # parameter 5 belongs to no gate
    theta = g.uniform(-3, 3, (batch, nparams))
    terms = [(float(g.standard_normal()), "".join(g.choice(list("IXYZ"), n))) for _ in range(5)]
    index = np.array(index, dtype=np.int32)
    values, grads = adjoint_expval(c, index, theta, terms, precision)
    for row in range(batch):
        v, gr = oracle.adjoint(n, c.to_ops(), index, theta[row], terms)
        assert abs(values[row] - v) < TOL[precision]
        assert np.abs(grads[row] - gr).max() < TOL[precision]
    assert not grads[:, 5].any()

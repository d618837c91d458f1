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


@pytest.mark.parametrize("order", ["up", "down", "few"])
@pytest.mark.parametrize("n,precision", [(13, "c64"), (13, "c128"), (16, "c64")])  # 16: blocks compiled at run time
@pytest.mark.parametrize("ckpt", [1, 2, 0])
def test_qubits_that_join_late_or_never(oracle, order, n, precision, ckpt):
    """Blocks before all qubits have been acted on run on part of the tiles;
    the Hamiltonian reaches every qubit."""
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    qs = list(range(n))
    if order == "down":
        qs = qs[::-1]
    elif order == "few":
        qs = [2, 3, 9]
    c, index, k = kb.Circuit(n), [], 0
    for layer in range(4):
        use = qs[: max(2, (layer + 1) * len(qs) // 4)]
        for q in use:
            for name in ("ry", "rz", "rx"):
                getattr(c, name)(q, 0.0)
                index.append(k)
                k += 1
            c.rz(q, 0.3 + layer)
            index.append(-1)
        for a, b in zip(use[:-1], use[1:]):
            c.cx(a, b)
            index.append(-1)
        c.crz(use[0], use[-1], 0.0)
        index.append(k)
        k += 1
        c.barrier()
        index.append(-1)
    index = np.array(index, dtype=np.int32)
    g = np.random.default_rng(n)
    theta = g.uniform(-3, 3, (2, k))
    terms = [(float(g.standard_normal()), "".join(g.choice(list("IXYZ"), n))) for _ in range(6)]
    values, grads = adjoint_expval(c, index, theta, terms, precision, checkpoint_every=ckpt)
    for row in range(2):
        v, gr = oracle.adjoint(n, c.to_ops(), index, theta[row], terms)
        assert abs(values[row] - v) < TOL[precision]
        assert np.abs(grads[row] - gr).max() < TOL[precision]


@pytest.mark.parametrize("terms", [1, 31, 32, 33, 70, 300, 1101])  # 1101: beyond the shared-memory form
@pytest.mark.parametrize("n", [1, 2, 3, 9, 13])
@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_hamiltonians_of_every_length(oracle, n, terms, precision):
    """lambda = H psi: term counts around the 32-term masks, states of less
    than a CTA's word count, strings with and without Y and X on qubit 0."""
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    c, index = kb.Circuit(n), []
    for q in range(n):
        c.ry(q, 0.0)
        c.rx(q, 0.0)
        index += [2 * q, 2 * q + 1]
    for q in range(n - 1):
        c.cx(q, q + 1)
        index.append(-1)
    index = np.array(index, dtype=np.int32)
    g = np.random.default_rng(terms + n)
    theta = g.uniform(-3, 3, (1, 2 * n))
    ham = [(float(g.standard_normal()) / terms, "".join(g.choice(list("IXYZ"), n))) for _ in range(terms)]
    values, grads = adjoint_expval(c, index, theta, ham, precision)
    v, gr = oracle.adjoint(n, c.to_ops(), index, theta[0], ham)
    assert abs(values[0] - v) < TOL[precision]
    assert np.abs(grads[0] - gr).max() < TOL[precision]

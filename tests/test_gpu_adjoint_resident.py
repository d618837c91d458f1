"""Adjoint gradients over every gate kind: states that one CTA holds (more gates
than are staged at a time, gradient rows beyond one sum, checkpoints, a
Hamiltonian on both sides of the size that the CTA sums itself), and the
complex128 tiled sweeps (every gate body, one tile and several).

Tolerance: each gate rounds an amplitude a few times, forwards and backwards,
in the state's precision, so a value or gradient is off by less than
8 G eps sum|c| (G gates).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"c64": 2.0 ** -24, "c128": 2.0 ** -53}


def check(oracle, n, layers, terms, precision, **options):
    import ket_b200 as kb
    from ket_b200.autograd import adjoint_expval
    g = np.random.default_rng(100 * n + layers)
    c, index, gates = kb.Circuit(n), [], 0

    def add(name, qs, *ps, par=-1):
        nonlocal gates
        getattr(c, name)(*qs, *([0.0] if par >= 0 else ps))
        index.append(par)
        gates += 1

    k = 0
    for _ in range(layers):
        for q in range(n):
            for name in ("ry", "rz", "rx"):
                add(name, (q,), par=k)
                k += 1
            add("u", (q,), *g.uniform(-3, 3, 3))
        for q in range(n - 1):
            a, b = (q, q + 1) if q % 2 else (q + 1, q)
            for name in ("crx", "cry", "crz", "cp"):
                if g.integers(2):
                    add(name, (a, b), par=k)
                    k += 1
            add(str(g.choice(["cx", "cz", "swap"])), (a, b))
        if n > 2:
            qs = tuple(int(x) for x in g.permutation(n)[:3])
            add("ccx", qs)
            add("cswap", qs[::-1])
            add("t", (qs[0],))
        c.barrier()
        index.append(-1)
    theta = g.uniform(-3, 3, (2, k))
    ham = [(float(g.standard_normal()) / terms, "".join(g.choice(list("IXYZ"), n))) for _ in range(terms)]
    index = np.array(index, dtype=np.int32)
    values, grads = adjoint_expval(c, index, theta, ham, precision, **options)
    tol = 8 * gates * EPS[precision] * sum(abs(x) for x, _ in ham)
    for row in range(2):
        v, gr = oracle.adjoint(n, c.to_ops(), index, theta[row], ham)
        assert abs(values[row] - v) < tol
        assert np.abs(grads[row] - gr).max() < tol


@pytest.mark.parametrize("n,layers,terms", [(1, 9, 2), (2, 12, 5), (3, 5, 7), (6, 4, 33), (10, 2, 9), (11, 2, 128),
                                            (11, 1, 129), (5, 3, 1100)])
@pytest.mark.parametrize("checkpoint", [0, 1, 2])
@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_one_cta(oracle, n, layers, terms, checkpoint, precision):
    check(oracle, n, layers, terms, precision, checkpoint_every=checkpoint)


@pytest.mark.parametrize("n", [11, 12, 14])
@pytest.mark.parametrize("checkpoint", [0, 1])
def test_tiled_c128(oracle, n, checkpoint):
    check(oracle, n, 3, 6, "c128", checkpoint_every=checkpoint, method="tiled")

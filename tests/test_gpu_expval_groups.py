"""Pauli terms in groups of independent flips, and diagonal terms, against numpy.

Tolerance 1e-12 (the suite's bar for FP64 expectations of a unit-norm state);
the sums are FP64 over at most 2^22 products whose moduli add up to at most 1.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _reference(psi, pauli):
    n = len(pauli)
    flip = sum(1 << i for i in range(n) if pauli[n - 1 - i] in "XY")
    sign = sum(1 << i for i in range(n) if pauli[n - 1 - i] in "YZ")
    x = np.arange(len(psi))
    par = x & sign
    for s in (16, 8, 4, 2, 1):
        par ^= par >> s
    return float((1j ** (pauli.count("Y") % 4) * np.vdot(psi[x ^ flip], psi * (1 - 2 * (par & 1)))).real)


def _terms(n, rng, kind):
    if kind == "random":
        return ["".join(rng.choice(list("IXYZ"), n)) for _ in range(12)]
    if kind == "diagonal":  # more than one CTA row of diagonal terms where that many exist
        return ["".join(rng.choice(list("IZ"), n)) for _ in range(1100 if n <= 6 else 40)]
    if kind == "shared":  # one flip, many sign masks: more terms than a group takes of a flip
        f = rng.choice(list("IX"), n)
        f[0] = "X"
        return ["".join(rng.choice(["X", "Y"] if c == "X" else ["I", "Z"]) for c in f) for _ in range(7)]
    # dependent flips: the third of each triple is the product of the others
    out = []
    for _ in range(4):
        a, b = rng.integers(1, 1 << n, 2)
        out += ["".join("X" if (v >> (n - 1 - i)) & 1 else "Z" for i in range(n)) for v in (a, b, a ^ b)]
    return out


# 1..5: fewer qubits than flips a group; 12 and 13: one and two diagonal
# chunks; 19..22: groups of 2..5 flips
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 12, 13, 19, 20, 21, 22])
@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_terms_match_numpy(n, precision):
    import ctypes as ct

    import ket_b200 as kb
    from ket_b200 import _lib
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    st = kb.DeviceState(n, precision)
    st.from_numpy(psi)
    psi = st.to_numpy()  # as held (rounded to complex64)
    for kind in ("random", "diagonal", "shared", "dependent"):
        terms = _terms(n, rng, kind)
        arr, keep = _lib.c_strings(terms)
        got = np.zeros(len(terms))
        _lib.check(_lib.lib.ketgpu_expval_terms(st.handle, ct.cast(arr, ct.c_void_p), len(terms), got.ctypes.data))
        cache = {}
        for p, v in zip(terms, got):
            if p not in cache:
                cache[p] = _reference(psi, p)
            assert abs(v - cache[p]) < TOL, (kind, p)

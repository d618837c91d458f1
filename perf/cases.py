"""The work that users of this library have it do, as cases that can be timed.

A case names a kind of call, its sizes and its options.  ``prepare`` makes
what a program has in hand before the call (a circuit, a plan and a state,
parameters), ``run`` makes one pass through the public entry points, ``work``
counts the bytes and operations that no implementation can do without, and
``exact`` computes the same outputs with plain torch in 64 bits.

Kinds
  run      ket_b200.run(circuit): a host circuit in, 2^n host amplitudes out
  energy   ket_b200.expval(circuit, hamiltonian): one step of a search over
           circuits, nothing kept between calls
  shots    ket_b200.sample_shots(circuit, shots)
  plan     DeviceState.reset + Plan.execute: a compiled circuit run again
  apply    DeviceState.reset + DeviceState.apply: a new circuit on a kept
           state (planned inside the call)
  expval   DeviceState.expval of a Pauli sum
  sample   a one-gate change of the state, then DeviceState.sample_seeded
  adjoint  values and gradients of a variational circuit through torch
"""
import math
import random

import numpy as np
import torch

import ket_b200 as kb
from ket_b200.autograd import adjoint_expval_torch

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a small circuit run interactively, ket's own default precision:
        # launches and host work
        {"name": "run_c128_10q", "kind": "run", "n": 10, "depth": 10, "circuit": "brickwork"},
        # the largest size at which reading all amplitudes back is usual
        {"name": "run_c128_21q", "kind": "run", "n": 21, "depth": 20, "circuit": "mixed"},
        # the inner step of a search over circuits: evolve, then the energy
        # of a spin chain
        {"name": "energy_c128_14q", "kind": "energy", "n": 14, "depth": 8, "circuit": "brickwork", "obs": "chain"},
        # 20 qubits, depth 20, complex128: the reference configuration
        {"name": "plan_c128_20q", "kind": "plan", "n": 20, "depth": 20, "circuit": "brickwork", "precision": "c128"},
        # complex128 at a size far beyond L2
        {"name": "plan_c128_27q", "kind": "plan", "n": 27, "depth": 20, "circuit": "brickwork", "precision": "c128"},
        # a new complex64 circuit over the full gate mix, planned in the call
        {"name": "apply_c64_24q", "kind": "apply", "n": 24, "depth": 30, "circuit": "mixed", "precision": "c64"},
        # the benchmark's circuit: 30 qubits, depth 40, complex64
        {"name": "plan_c64_30q", "kind": "plan", "n": 30, "depth": 40, "circuit": "brickwork", "precision": "c64"},
        # QFT pattern + GHZ ladder + Rz: long runs of diagonal gates
        {"name": "plan_c64_29q_qft", "kind": "plan", "n": 29, "depth": 1, "circuit": "qft", "precision": "c64"},
        # 64 random Pauli strings on a large complex64 state
        {"name": "expval_c64_27q", "kind": "expval", "n": 27, "terms": 64, "obs": "random", "precision": "c64"},
        # 10^6 shots from a state that has just changed
        {"name": "sample_c64_28q", "kind": "sample", "n": 28, "shots": 1000000, "precision": "c64"},
        # the gradient benchmark: 8 layers, 384 parameters, 64 terms, 64 sets
        {"name": "adjoint_c64_24q", "kind": "adjoint", "n": 24, "layers": 8, "terms": 64, "batch": 64,
         "precision": "c64"},
        # a small variational model trained in double precision
        {"name": "adjoint_c128_14q", "kind": "adjoint", "n": 14, "layers": 4, "terms": 32, "batch": 8,
         "precision": "c128"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "energy", "shots", "plan", "plan", "plan", "apply", "expval", "expval", "sample",
                       "adjoint", "adjoint"])
    circuit = rng.choice(["brickwork", "mixed", "qft"])
    precision = rng.choice(["c64", "c128"])
    big = 28 if precision == "c64" else 26
    depth = 1 if circuit == "qft" else _log_int(rng, 3, 30)
    if kind == "run":
        return {"kind": kind, "n": rng.randint(4, 21), "depth": depth, "circuit": circuit}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(4, 20), "depth": depth, "circuit": circuit,
                "obs": rng.choice(["chain", "random"])}
    if kind == "shots":
        return {"kind": kind, "n": rng.randint(4, 18), "depth": depth, "circuit": circuit,
                "shots": _log_int(rng, 1, 20000)}
    if kind == "plan":
        return {"kind": kind, "n": rng.randint(8, big), "depth": depth, "circuit": circuit, "precision": precision}
    if kind == "apply":
        return {"kind": kind, "n": rng.randint(8, big - 2), "depth": depth, "circuit": circuit,
                "precision": precision}
    if kind == "expval":
        return {"kind": kind, "n": rng.randint(6, big), "terms": _log_int(rng, 1, 128),
                "obs": rng.choice(["chain", "random"]), "precision": precision}
    if kind == "sample":
        return {"kind": kind, "n": rng.randint(6, big), "shots": _log_int(rng, 1, 1000000), "precision": precision}
    return {"kind": kind, "n": rng.randint(6, 22 if precision == "c64" else 20), "layers": rng.randint(1, 8),
            "terms": _log_int(rng, 1, 64), "batch": _log_int(rng, 1, 32), "precision": precision}


# ---- circuits, as plain (name, qubits, params) lists ------------------------
_MIX = ["h", "s", "t", "rx", "ry", "rz", "u", "cx", "cz", "cp", "crz", "swap", "ccx", "cswap"]
_ARITY = {"cx": 2, "cz": 2, "cp": 2, "crz": 2, "swap": 2, "ccx": 3, "cswap": 3}
_PARAMS = {"rx": 1, "ry": 1, "rz": 1, "u": 3, "cp": 1, "crz": 1}


def _gates(case, seed):
    rng = random.Random(seed)
    n, out = case["n"], []
    if case["circuit"] == "brickwork":
        for layer in range(case["depth"]):
            for q in range(n):
                out.append(("u", (q,), tuple(rng.uniform(0.0, TWO_PI) for _ in range(3))))
            for a in range(layer % 2, n - 1, 2):
                out.append(("cx", (a, a + 1), ()))
    elif case["circuit"] == "mixed":
        for _ in range(case["depth"]):
            free = list(range(n))
            rng.shuffle(free)
            while free:
                name = rng.choice(_MIX)
                a = _ARITY.get(name, 1)
                if a > len(free):
                    continue
                qs = tuple(free.pop() for _ in range(a))
                out.append((name, qs, tuple(rng.uniform(0.0, TWO_PI) for _ in range(_PARAMS.get(name, 0)))))
    else:
        for q in range(n):
            out.append(("h", (q,), ()))
        for i in range(n):
            for j in range(i + 1, n):
                out.append(("cp", (i, j), (math.pi / (2 ** (j - i)),)))
        out.append(("h", (0,), ()))
        for i in range(n - 1):
            out.append(("cx", (i, i + 1), ()))
        for q in range(n):
            out.append(("rz", (q,), (rng.uniform(0.0, TWO_PI),)))
        # the transform's own last rotations, seeded, so that the amplitudes
        # (and not their phases alone) depend on the inputs
        for q in range(n):
            out.append(("ry", (q,), (rng.uniform(0.0, TWO_PI),)))
    return out


def _circuit(n, gates):
    c = kb.Circuit(n)
    for name, qs, ps in gates:
        getattr(c, name)(*qs, *ps)
    return c


def _hamiltonian(case, seed):
    n = case["n"]
    rng = random.Random(seed * 2 + 1)
    if case.get("obs", "random") == "chain":  # a Heisenberg chain in a field
        out, most = [], case.get("terms", 4 * n)
        for q in range(n):
            for p in ("XX", "YY", "ZZ"):
                if q + 1 < n:
                    out.append((rng.gauss(0.0, 1.0), "I" * (n - q - 2) + p + "I" * q))
            out.append((rng.gauss(0.0, 1.0), "I" * (n - q - 1) + "Z" + "I" * q))
        return out[:most]
    return [(rng.gauss(0.0, 1.0), "".join(rng.choice("IXYZ") for _ in range(n))) for _ in range(case["terms"] if "terms" in case else 16)]


def _random_state(n, precision, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if precision == "c64" else torch.float64
    v = torch.randn((1 << n, 2), generator=g, device="cuda", dtype=dt)
    v /= math.sqrt(2.0 * (1 << n))
    return torch.view_as_complex(v)


def _device_state(n, precision, seed):
    st = kb.DeviceState(n, precision)
    st.torch_view().copy_(_random_state(n, precision, seed))
    torch.cuda.synchronize()
    return st


def _ansatz(case):
    """Ry then Rz on every qubit, then a CX ring, per layer."""
    n, out = case["n"], []
    for _ in range(case["layers"]):
        out += [("ry", (q,)) for q in range(n)]
        out += [("rz", (q,)) for q in range(n)]
        out += [("cx", (q, (q + 1) % n)) for q in range(n)]
        out.append(("barrier", ()))
    return out


def _theta(case, seed):
    g = torch.Generator().manual_seed(seed)
    t = (torch.rand((case["batch"], 2 * case["n"] * case["layers"]), generator=g, dtype=torch.float64) * 2 - 1) * math.pi
    return t.to(torch.float32) if case["precision"] == "c64" else t


def _view(state):
    """The amplitudes without a copy; the tensor keeps their owner alive."""
    amps = state.torch_view()
    amps.owner = state
    return amps


# ---- the passes -------------------------------------------------------------
def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"kind": kind, "case": case}
    if kind in ("run", "energy", "shots", "apply"):
        s["circuit"] = _circuit(n, _gates(case, seed))
        if kind == "energy":
            s["obs"] = _hamiltonian(case, seed)
        if kind == "shots":
            s["circuit"].measure_all()
            s["seed"] = seed & 0xFFFF
        if kind == "apply":
            s["state"] = kb.DeviceState(n, case["precision"])
            s["options"] = kb.make_options(precision=case["precision"])
    elif kind == "plan":
        opt = kb.make_options(precision=case["precision"])
        s["plan"] = kb.Plan(n, _circuit(n, _gates(case, seed)).to_ops(), opt)
        s["state"] = kb.DeviceState(n, case["precision"])
    elif kind == "expval":
        s["state"] = _device_state(n, case["precision"], seed)
        s["obs"] = _hamiltonian(case, seed)
    elif kind == "sample":
        s["state"] = _device_state(n, case["precision"], seed)
        c = kb.Circuit(n)
        c.x(seed % n)
        s["plan"] = kb.Plan(n, c.to_ops(), kb.make_options(precision=case["precision"], fusion="none"))
        s["seed"] = seed & 0xFFFF
    else:
        c, index, k = kb.Circuit(n), [], 0
        for name, qs in _ansatz(case):
            if name in ("ry", "rz"):
                getattr(c, name)(*qs, 0.0)
                index.append(k)
                k += 1
            else:
                getattr(c, name)(*qs)
                index.append(-1)
        s["circuit"], s["index"] = c, np.array(index, dtype=np.int32)
        s["obs"] = _hamiltonian(case, seed)
        s["theta"] = _theta(case, seed).cuda().requires_grad_(True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "run":
        return kb.run(s["circuit"]).to_numpy()
    if kind == "energy":
        return kb.expval(s["circuit"], s["obs"])
    if kind == "shots":
        return kb.sample_shots(s["circuit"], s["case"]["shots"], s["seed"])
    if kind == "plan":
        s["state"].reset()
        s["plan"].execute(s["state"])
        return _view(s["state"])
    if kind == "apply":
        s["state"].reset()
        s["state"].apply(s["circuit"], s["options"])
        return _view(s["state"])
    if kind == "expval":
        return s["state"].expval(s["obs"])
    if kind == "sample":
        s["plan"].execute(s["state"], sync=False)
        return s["state"].sample_seeded(s["seed"], s["case"]["shots"])
    values = adjoint_expval_torch(s["theta"], s["circuit"], s["index"], s["obs"], s["case"]["precision"], 2)
    (grad,) = torch.autograd.grad(values.sum(), s["theta"])
    return {"values": values, "grad": grad}


# ---- what a pass cannot do without ------------------------------------------
def _gate_flops(name, dim):
    if name in ("s", "t"):
        return 3.0 * dim
    if name in ("cz", "cp", "crz"):
        return 1.5 * dim
    if name == "rz":
        return 6.0 * dim
    if name in ("cx", "swap", "ccx", "cswap", "barrier"):
        return 0.0
    return 14.0 * dim


def work(case):
    kind, n = case["kind"], case["n"]
    dim = float(1 << n)
    amp = 8.0 if case.get("precision", "c128") == "c64" else 16.0
    terms = len(_hamiltonian(case, 1)) if kind in ("energy", "expval", "adjoint") else 0
    if kind in ("run", "energy", "shots", "plan", "apply"):
        flops = sum(_gate_flops(g[0], dim) for g in _gates(case, 1))
        bytes_ = amp * dim  # the state written once
        if kind == "energy":
            flops += 8.0 * dim * terms
        if kind == "shots":
            flops += 4.0 * dim
            bytes_ += 4.0 * n * case["shots"]
        return {"bytes": bytes_, "flops": flops}
    if kind == "expval":
        return {"bytes": amp * dim, "flops": 8.0 * dim * terms}
    if kind == "sample":  # the changed state read and written, then read
        return {"bytes": 3.0 * amp * dim + 8.0 * case["shots"], "flops": 4.0 * dim}
    gates = [g[0] for g in _ansatz(case)]
    fwd = sum(_gate_flops(g, dim) for g in gates)
    inner = 8.0 * dim * 2 * n * case["layers"]
    return {"bytes": 4.0 * amp * dim * case["batch"],
            "flops": case["batch"] * (3.0 * fwd + inner + 8.0 * dim * terms)}


# ---- the same outputs from plain torch in 64 bits ---------------------------
def _matrix(name, p):
    r = math.sqrt(0.5)
    if name in ("h",):
        return (r, r, r, -r)
    if name in ("x", "cx", "ccx"):
        return (0, 1, 1, 0)
    if name == "s":
        return (1, 0, 0, 1j)
    if name == "t":
        return (1, 0, 0, complex(r, r))
    if name == "cz":
        return (1, 0, 0, -1)
    if name == "cp":
        return (1, 0, 0, complex(math.cos(p[0]), math.sin(p[0])))
    c, s = math.cos(p[0] / 2), math.sin(p[0] / 2)
    if name == "rx":
        return (c, -1j * s, -1j * s, c)
    if name == "ry":
        return (c, -s, s, c)
    if name in ("rz", "crz"):
        return (complex(c, -s), 0, 0, complex(c, s))
    e = lambda a: complex(math.cos(a), math.sin(a))  # noqa: E731
    return (c, -e(p[2]) * s, e(p[1]) * s, e(p[1] + p[2]) * c)


def _pair(psi, n, fixed):
    """The view of the amplitudes whose bit q is fixed[q], for each q of `fixed`."""
    shape, index, top = [], [], n
    for q in sorted(fixed, reverse=True):
        shape += [1 << (top - q - 1), 2]
        index += [slice(None), fixed[q]]
        top = q
    return psi.view(shape + [1 << top])[tuple(index)]


def _apply(psi, n, name, qs, ps):
    if name in ("swap", "cswap"):
        ctl = {qs[0]: 1} if name == "cswap" else {}
        x, y = qs[-2:]
        a, b = _pair(psi, n, {**ctl, x: 1, y: 0}), _pair(psi, n, {**ctl, x: 0, y: 1})
        m = (0, 1, 1, 0)
    else:
        ctl, t = {q: 1 for q in qs[:-1]}, qs[-1]
        a, b = _pair(psi, n, {**ctl, t: 0}), _pair(psi, n, {**ctl, t: 1})
        m = _matrix(name, ps)
    if m[1] == 0 and m[2] == 0:
        if m[0] != 1:
            a.mul_(m[0])
        b.mul_(m[3])
        return
    if m == (0, 1, 1, 0):
        old = a.clone()
        a.copy_(b)
        b.copy_(old)
        return
    na = a * m[0]
    na.add_(b, alpha=m[1])
    b.mul_(m[3]).add_(a, alpha=m[2])
    a.copy_(na)


def _evolve(n, gates):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    for name, qs, ps in gates:
        _apply(psi, n, name, qs, ps)
    return psi


def _masks(pauli):
    n = len(pauli)
    flip = sum(1 << i for i in range(n) if pauli[n - 1 - i] in "XY")
    sign = sum(1 << i for i in range(n) if pauli[n - 1 - i] in "YZ")
    return flip, sign, pauli.count("Y") % 4


def _pauli_on(psi, index, pauli):
    """P psi for one Pauli string: out[x ^ flip] = i^q (-1)^|x & sign| psi[x]."""
    flip, sign, q = _masks(pauli)
    src = index ^ flip
    par = src & sign
    for sh in (32, 16, 8, 4, 2, 1):
        par ^= par >> sh
    out = psi[src]
    del src
    return out.mul_((1 - 2 * (par & 1)).to(torch.float64)).mul_(1j ** q)


def _energy(psi, obs):
    index = torch.arange(psi.numel(), device="cuda")
    return sum(c * float(torch.vdot(psi, _pauli_on(psi, index, p)).real) for c, p in obs)


def _exact_adjoint(case, seed):
    n, ops, obs = case["n"], _ansatz(case), _hamiltonian(case, seed)
    theta = _theta(case, seed).double()
    index = torch.arange(1 << n, device="cuda")
    values, grads = torch.zeros(case["batch"], dtype=torch.float64), torch.zeros_like(theta)
    for row in range(case["batch"]):
        angles, k, gates = theta[row].tolist(), 0, []
        for name, qs in ops:
            if name in ("ry", "rz"):
                gates.append((name, qs, (angles[k],)))
                k += 1
            elif name == "cx":
                gates.append((name, qs, ()))
        psi = _evolve(n, gates)
        lam = torch.zeros_like(psi)
        for c, p in obs:
            lam.add_(_pauli_on(psi, index, p), alpha=c)
        values[row] = float(torch.vdot(psi, lam).real)
        got = []
        for name, qs, ps in reversed(gates):
            if ps:  # d/dt exp(-i t P / 2): the imaginary part of <lam|P psi>
                q = qs[0]
                a, b = _pair(psi, n, {q: 0}), _pair(psi, n, {q: 1})
                la, lb = _pair(lam, n, {q: 0}), _pair(lam, n, {q: 1})
                d = (la.conj() * a - lb.conj() * b) if name == "rz" else (lb.conj() * a - la.conj() * b) * 1j
                got.append(d.sum().imag)
                back = (name, qs, (-ps[0],))
            else:
                back = (name, qs, ps)
            _apply(psi, n, *back)
            _apply(lam, n, *back)
        grads[row] = torch.stack(got[::-1]).cpu()
    return {"values": values, "grad": grads}


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("run", "plan", "apply", "energy"):
        gates = _gates(case, seed)
        if len(gates) * (1 << n) > 4e11:  # a minute of plain torch
            return None
        psi = _evolve(n, gates)
        if kind == "energy":
            return _energy(psi, _hamiltonian(case, seed))
        return psi.cpu().numpy() if kind == "run" else psi
    if kind == "expval":
        return _energy(_random_state(n, case["precision"], seed).to(torch.complex128), _hamiltonian(case, seed))
    if kind == "adjoint":
        gates = 3 * len(_ansatz(case)) + 4 * case["terms"]
        if case["batch"] * gates * ((1 << n) + (1 << 17)) > 3e10:
            return None
        return _exact_adjoint(case, seed)
    return None  # draws are whole numbers

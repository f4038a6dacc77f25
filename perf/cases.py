"""What is measured of this engine: the calls its users make, over their real range.

A case is one of seven kinds of call:

  run      a circuit on a register through ``CudaStateVectorBackend.run_into`` (complex128 or
           complex64, tiled or fused), then what a program reads from it: shots, and either the
           whole state ("read": "state") or, from a large register, what fits the question: the
           distribution of its low qubits and a few Pauli expectations ("read": "statistics")
  steps    a program that drives the register gate by gate and measures on the way
           (``State.apply_1q`` / ``apply_2q`` / ``apply_controlled_1q`` / ``measure_qubit``)
  energy   the terms of a transverse-field Ising Hamiltonian on a state at hand
  batch    many small Trotter circuits in one call (``batch.run_batch``)
  serve    a mixed burst of requests through the request loop (``serve.Server``)
  density  a noisy circuit on a density matrix (``DensityMatrixBackend``)

Circuits are made here from the seed alone as lists of (kind, qubits, matrix) so that ``exact``
can evaluate the same lists in plain torch in 64 bits.  Numbers read from a complex64 register are
kept in single precision, as a program that chose complex64 keeps them.
"""
import math

import numpy as np
import torch

from everett_gb300 import CudaStateVectorBackend, Circuit, Gate1, Gate2, PauliString, State
from everett_gb300 import batch, density, serve, workloads
from everett_gb300.rng import Rng

LOW = 20  # the qubits whose distribution a program reads from a large register


def listed():
    return [
        # the smallest call: a 10-qubit circuit whose amplitudes are looked at, as in a notebook or
        # the inner step of a variational loop -- latency and launches count
        {"name": "run small c128", "kind": "run", "circuit": "layers", "n": 10, "depth": 10,
         "dtype": "complex128", "mode": "tiled", "shots": 0, "read": "state"},
        # an ordinary odd-sized register in the default mode, amplitudes and shots
        {"name": "run 17q c128", "kind": "run", "circuit": "layers", "n": 17, "depth": 20,
         "dtype": "complex128", "mode": "tiled", "shots": 1000, "read": "state"},
        # the reference's own sampling workload: 20 qubits, depth 20, 10000 shots
        {"name": "run 20q c128", "kind": "run", "circuit": "layers", "n": 20, "depth": 20,
         "dtype": "complex128", "mode": "tiled", "shots": 10000, "read": "state"},
        # the same circuit family on a register far beyond the caches: the default mode's bulk
        # work, with the state back on the host as the reference's run leaves it
        {"name": "run 26q c128", "kind": "run", "circuit": "layers", "n": 26, "depth": 10,
         "dtype": "complex128", "mode": "tiled", "shots": 1000, "read": "state"},
        # double precision on the tensor cores
        {"name": "fused 26q c128", "kind": "run", "circuit": "layers", "n": 26, "depth": 20,
         "dtype": "complex128", "mode": "fused", "shots": 1000, "read": "statistics"},
        # Haar-random layers in single precision on the tensor cores, the largest register listed
        {"name": "fused 28q c64", "kind": "run", "circuit": "haar", "n": 28, "depth": 16,
         "dtype": "complex64", "mode": "fused", "shots": 0, "read": "statistics"},
        # a Fourier transform of a basis state: long ladders of controlled phases, odd size
        {"name": "qft 25q c64", "kind": "run", "circuit": "qft", "n": 25, "depth": 1,
         "dtype": "complex64", "mode": "tiled", "shots": 0, "read": "statistics"},
        # a program that applies its own gates one by one and measures mid-way
        {"name": "steps 26q c128", "kind": "steps", "n": 26, "dtype": "complex128",
         "read": "statistics"},
        # energy of a spin chain on a state at hand: bonds (Z Z) and fields (X)
        {"name": "energy 26q c64", "kind": "energy", "n": 26, "dtype": "complex64"},
        # parameter sweep: many Trotter circuits of uneven size in one launch
        {"name": "batch 512 c64", "kind": "batch", "count": 512, "nmin": 8, "nmax": 18,
         "smin": 10, "smax": 30, "shots": 16, "dtype": "complex64"},
        # a burst of mixed requests on the serving loop
        {"name": "serve 48", "kind": "serve", "count": 48, "nmin": 10, "nmax": 18, "shots": 1000},
        # noise study: depolarizing noise after every gate
        {"name": "density 11q", "kind": "density", "n": 11, "depth": 3, "p": 0.001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "steps", "energy", "batch", "serve", "density"])
    if kind == "run":
        dtype, mode = rng.choice([("complex128", "tiled"), ("complex128", "tiled"),
                                  ("complex128", "fused"), ("complex64", "fused"),
                                  ("complex64", "tiled")])
        family = rng.choice(["layers", "haar", "qft"])
        top = 25 if (dtype, mode) == ("complex128", "tiled") else 26
        n = rng.randint(13 if mode == "fused" else 5, top)
        depth = 1 if family == "qft" else rng.randint(4, 10 if n > 24 else 20)
        # shots of a complex64 run hang on its last bits: its statistics are read instead
        shots = 0 if dtype == "complex64" else rng.choice([0, _log_int(rng, 50, 10000)])
        return {"kind": "run", "circuit": family, "n": n, "depth": depth, "dtype": dtype,
                "mode": mode, "shots": shots, "read": "state" if n <= 22 else "statistics"}
    if kind == "steps":
        n = rng.randint(8, 26)
        return {"kind": "steps", "n": n, "dtype": rng.choice(["complex128", "complex64"]),
                "read": "state" if n <= 22 else "statistics"}
    if kind == "energy":
        return {"kind": "energy", "n": rng.randint(8, 26),
                "dtype": rng.choice(["complex128", "complex64"])}
    if kind == "batch":
        nmin = rng.randint(4, 9)
        return {"kind": "batch", "count": _log_int(rng, 8, 400), "nmin": nmin,
                "nmax": rng.randint(nmin + 2, 17), "smin": 5, "smax": rng.randint(8, 30),
                "shots": 16, "dtype": rng.choice(["complex64", "complex64", "complex128"])}
    if kind == "serve":
        nmin = rng.randint(8, 12)
        return {"kind": "serve", "count": rng.randint(4, 40), "nmin": nmin,
                "nmax": rng.randint(nmin + 1, 18), "shots": _log_int(rng, 50, 1000)}
    return {"kind": "density", "n": rng.randint(3, 10), "depth": rng.randint(1, 3),
            "p": rng.choice([0.0005, 0.001, 0.01])}


# ---- circuits as plain lists ------------------------------------------------------------------

def _rz(t):
    return np.array([[np.exp(-0.5j * t), 0], [0, np.exp(0.5j * t)]])


def _ry(t):
    c, s = math.cos(t / 2), math.sin(t / 2)
    return np.array([[c, -s], [s, c]], dtype=complex)


_H = np.array([[1, 1], [1, -1]], dtype=complex) * 0.7071067811865476
_X = np.array([[0, 1], [1, 0]], dtype=complex)


def _haar(rng):
    z = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))
    q, r = np.linalg.qr(z)
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _gates(family, n, depth, rng):
    """[(kind, qubits, argument)]: rz/ry (angle), u (2x2), x/h, cphase (angle), cx, cz, swap."""
    ops = []
    if family == "qft":
        ops += [("x", (q,), None) for q in range(n) if rng.random() < 0.5]
        for j in range(n - 1, -1, -1):
            ops.append(("h", (j,), None))
            ops += [("cphase", (k, j), math.tau / float(1 << (j - k + 1)))
                    for k in range(j - 1, -1, -1)]
        ops += [("swap", (i, n - 1 - i), None) for i in range(n // 2)]
        return ops
    for layer in range(depth):
        for q in range(n):
            if family == "haar":
                ops.append(("u", (q,), _haar(rng)))
            else:
                a, b, c = rng.uniform(0, math.tau, 3)
                ops += [("rz", (q,), a), ("ry", (q,), b), ("rz", (q,), c)]
        two = "cz" if family == "haar" else "cx"
        ops += [(two, (i, i + 1), None) for i in range(layer % 2, n - 1, 2)]
    return ops


def _circuit(n, ops):
    c = Circuit(n)
    for kind, q, arg in ops:
        if kind in ("rz", "ry"):
            getattr(c, kind)(q[0], float(arg))
        elif kind == "u":
            c.gate1(Gate1.from_matrix(arg), q[0])
        elif kind in ("x", "h"):
            getattr(c, kind)(q[0])
        elif kind == "cphase":
            c.controlled([q[0]], Gate1.phase(arg), q[1])
        else:
            {"cx": c.cnot, "cz": c.cz, "swap": c.swap}[kind](*q)
    return c


def _strings(n, rng, count=4):
    """A few two-body Pauli strings, as a program checks correlations with, and the identity
    (the squared norm) beside them."""
    out = ["I" * n]
    for _ in range(count):
        t = ["I"] * n
        for q in rng.choice(n, size=min(2, n), replace=False):
            t[int(q)] = "XYZ"[int(rng.integers(3))]
        out.append("".join(t))
    return out


def _chain(n):
    """The terms of a transverse-field Ising chain: Z Z on every bond, X on every site."""
    return ([("I" * i + "ZZ" + "I" * (n - i - 2)) for i in range(n - 1)]
            + [("I" * i + "X" + "I" * (n - i - 1)) for i in range(n)])


def _steps(n, rng):
    """A gate-by-gate program: a layer of H and rotations, entanglers near and far, a controlled
    phase, an Rzz, and three measurements with their uniforms."""
    ops = [("h", (q,), None) for q in range(0, n, 2)]
    ops += [("u", (q,), _haar(rng)) for q in range(1, n, 4)]
    for q in range(0, n, 5):
        ops += [("rz", (q,), rng.uniform(0, math.tau)), ("ry", (q,), rng.uniform(0, math.tau))]
    ops += [("cx", (q, (q + n // 2) % n), None) for q in range(0, n, 6)]
    ops += [("cz", (q, (q + 1) % n), None) for q in range(1, n, 7)]
    ops += [("cphase", (q, n - 1 - q), rng.uniform(0, math.tau)) for q in range(0, n // 2, 3)]
    ops += [("rzz", (q, q + 2), rng.uniform(0, math.tau)) for q in range(0, n - 2, 6)]
    for q in rng.choice(n, size=min(3, n), replace=False):
        ops.append(("measure", (int(q),), float(rng.random())))
        ops.append(("u", ((int(q) + 1) % n,), _haar(rng)))
    return ops


# ---- what a program has in hand, and the call ---------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    if kind == "run":
        n = case["n"]
        circuit = _circuit(n, _gates(case["circuit"], n, case["depth"], rng))
        circuit.validate()
        paulis = [PauliString.parse(t) for t in _strings(n, rng)]
        return {"case": case, "circuit": circuit, "state": State.zero(n, case["dtype"]),
                "paulis": paulis, "seed": seed}
    if kind == "steps":
        n = case["n"]
        made = []
        for what, q, arg in _steps(n, rng):
            g = {"rz": Gate1.rz, "ry": Gate1.ry, "u": Gate1.from_matrix, "cphase": Gate1.phase,
                 "rzz": Gate2.rzz}.get(what)
            named = {"h": Gate1.h, "cx": Gate2.cnot, "cz": Gate2.cz}.get(what)
            made.append((what, q, g(arg) if g else named() if named else arg))
        paulis = [PauliString.parse(t) for t in _strings(n, rng)]
        return {"case": case, "ops": made, "state": State.zero(n, case["dtype"]),
                "paulis": paulis}
    if kind == "energy":
        n = case["n"]
        state = State.zero(n, case["dtype"])
        CudaStateVectorBackend.run_into(state, _circuit(n, _gates("layers", n, 2, rng)))
        return {"case": case, "state": state, "paulis": [PauliString.parse(t) for t in _chain(n)]}
    if kind == "batch":
        draws = Rng.seed_from_u64(seed)
        circuits = [workloads.tfim_raw(draws, case["nmin"], case["nmax"], case["smin"], case["smax"])
                    for _ in range(case["count"])]
        return {"case": case, "circuits": circuits, "seeds": list(range(seed, seed + len(circuits)))}
    if kind == "serve":
        draws = Rng.seed_from_u64(seed)
        requests = [workloads.serve_request(draws, case["nmin"], case["nmax"])[1]
                    for _ in range(case["count"])]
        return {"case": case, "server": serve.Server(),
                "requests": [(c, seed + i, case["shots"]) for i, c in enumerate(requests)]}
    n = case["n"]
    circuit = _circuit(n, _gates("layers", n, case["depth"], rng))
    circuit.validate()
    return {"case": case, "circuit": circuit, "seed": seed,
            "noise": density.NoiseModel.uniform_depolarizing(case["p"])}


def _read(state, case, paulis, out):
    """What a program takes from a register after its circuit."""
    single = case["dtype"] == "complex64"
    if case["read"] == "state":
        amps = state.amplitudes()
        out["amplitudes"] = amps.astype(np.complex64) if single else amps
    else:
        marginal = state.marginal_low(LOW)
        values = state.pauli_expectation(paulis)
        out["marginal"] = marginal.astype(np.float32) if single else marginal
        out["paulis"] = values.astype(np.float32) if single else values
    return out


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "run":
        reg, out = state["state"], {}
        CudaStateVectorBackend.run_into(reg, state["circuit"], mode=case["mode"])
        if case["shots"]:
            out["shots"] = reg.sample(case["shots"], seed=state["seed"])
        return _read(reg, case, state["paulis"], out)
    if kind == "steps":
        reg, bits = state["state"], []
        reg.set_zero()
        for what, q, arg in state["ops"]:
            if what == "measure":
                bits.append(reg.measure_qubit(q[0], arg))
            elif what == "cphase":
                reg.apply_controlled_1q([q[0]], q[1], arg)
            elif len(q) == 2:
                reg.apply_2q(q[0], q[1], arg)
            else:
                reg.apply_1q(q[0], arg)
        return _read(reg, case, state["paulis"], {"bits": bits})
    if kind == "energy":
        values = state["state"].pauli_expectation(state["paulis"])
        return {"terms": values.astype(np.float32) if case["dtype"] == "complex64" else values}
    if kind == "batch":
        results, _ = batch.run_batch(state["circuits"], seeds=state["seeds"], shots=case["shots"],
                                     dtype=case["dtype"])
        z = np.array([r.expz for r in results])
        return {"z0": z.astype(np.float32) if case["dtype"] == "complex64" else z,
                "shots": np.stack([r.shots for r in results]).astype(np.int64)}
    if kind == "serve":
        answers = list(state["server"].run_all(state["requests"]).values())
        return {"shots": np.stack([r.shots for r in answers]).astype(np.int64),
                "bits": np.array([int(r.classical[0]) if r.classical else -1 for r in answers],
                                 dtype=np.int64)}
    ex = density.DensityMatrixBackend.run_with_noise_seeded(state["circuit"], state["noise"],
                                                            state["seed"])
    return {"rho": ex.density_matrix().data()}


# ---- the work of a pass ------------------------------------------------------------------------

_FLOPS = {"rz": 6, "ry": 6, "u": 14, "h": 6, "x": 0, "cphase": 1.5, "cx": 0, "cz": 0.5, "swap": 0,
          "rzz": 6, "measure": 7}


def work(case):
    """Bytes: each array that goes in or comes out, once (a register: the state it leaves).
    Flops: a gate's multiplications and additions on the amplitudes that it changes."""
    kind = case["kind"]
    size = 16 if case.get("dtype") != "complex64" else 8
    rng = np.random.default_rng([1, 20])
    if kind in ("run", "steps"):
        n = case["n"]
        ops = _steps(n, rng) if kind == "steps" else _gates(case["circuit"], n, case["depth"], rng)
        flops = float(sum(_FLOPS[o[0]] for o in ops)) * 2.0 ** n
        return {"bytes": size * 2.0 ** n * (2 if case["read"] == "state" else 1), "flops": flops}
    if kind == "energy":
        return {"bytes": size * 2.0 ** case["n"], "flops": 2.0 ** case["n"] * (3 + 5 * case["n"])}
    if kind == "batch":
        draws, flops = Rng.seed_from_u64(1), 0.0
        for _ in range(case["count"]):
            c = workloads.tfim_raw(draws, case["nmin"], case["nmax"], case["smin"], case["smax"])
            flops += len(c) * 8.0 * 2.0 ** c.num_qubits()
        return {"bytes": case["count"] * (8.0 * case["shots"] + 8), "flops": flops}
    if kind == "serve":
        mean = sum(2.0 ** q for q in range(case["nmin"], case["nmax"] + 1)) / (
            case["nmax"] - case["nmin"] + 1)
        q = 0.5 * (case["nmin"] + case["nmax"])
        return {"bytes": case["count"] * 8.0 * (mean + case["shots"]),
                "flops": case["count"] * mean * (0.4 * 2 * q * q * 18 + 0.2 * q * q + 0.2 * 60 * q * 8)}
    n = case["n"]
    ops = len(_gates("layers", n, case["depth"], rng))
    return {"bytes": 16.0 * 4.0 ** n, "flops": ops * 40.0 * 4.0 ** n}


# ---- the same in plain torch, in 64 bits --------------------------------------------------------

def _matrix(what, arg):
    if what == "rz":
        return _rz(arg)
    if what == "ry":
        return _ry(arg)
    if what == "cphase":
        return np.array([[1, 0], [0, np.exp(1j * arg)]])
    return {"u": arg, "h": _H, "x": _X}[what]


class _Register:
    """2^n complex128 amplitudes; one-qubit gates wait until something else touches their qubit
    and are then applied up to three neighbours at a time."""

    def __init__(self, n):
        self.n, self.waiting = n, {}
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.a = torch.zeros(1 << n, dtype=torch.complex128, device=self.dev)
        self.a[0] = 1

    def one(self, q, m):
        self.waiting[q] = m @ self.waiting.get(q, np.eye(2))

    def flush(self):
        q = 0
        while q < self.n:
            if q not in self.waiting:
                q += 1
                continue
            m, w = self.waiting.pop(q), 1
            while w < 3 and q + w in self.waiting:
                m, w = np.kron(self.waiting.pop(q + w), m), w + 1
            u = torch.from_numpy(np.ascontiguousarray(m)).to(self.dev)
            v = self.a.view(-1, 1 << w, 1 << q)
            self.a = (torch.matmul(v.transpose(1, 2), u.T).transpose(1, 2) if q == 0
                      else torch.matmul(u, v)).reshape(-1)
            q += w

    def pair(self, a, b):
        """Views of the amplitudes by the bits (a, b)."""
        hi, lo = max(a, b), min(a, b)
        v = self.a.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
        return lambda i, j: v[:, i, :, j] if a > b else v[:, j, :, i]

    def apply(self, what, q, arg):
        if len(q) == 1 and what != "measure":
            self.one(q[0], _matrix(what, arg))
            return None
        if any(x in self.waiting for x in q):
            self.flush()
        if what == "measure":
            self.flush()
            v = self.a.view(-1, 2, 1 << q[0])
            p1 = float(v[:, 1].abs().square().sum())
            bit = arg < p1
            v[:, 0 if bit else 1] = 0
            self.a *= 1.0 / math.sqrt(p1 if bit else 1.0 - p1)
            return bool(bit)
        at = self.pair(*q)
        if what in ("cx", "swap"):
            x, y = (at(1, 0), at(1, 1)) if what == "cx" else (at(0, 1), at(1, 0))
            t = x.clone()
            x.copy_(y)
            y.copy_(t)
        elif what == "cz":
            at(1, 1).neg_()
        elif what == "cphase":
            at(1, 1).mul_(complex(math.cos(arg), math.sin(arg)))
        else:  # rzz
            even, odd = np.exp(-0.5j * arg), np.exp(0.5j * arg)
            for i in (0, 1):
                for j in (0, 1):
                    at(i, j).mul_(complex(even if i == j else odd))
        return None

    def expectation(self, text):
        """<psi|P|psi> from b = P psi."""
        b = self.a
        for q, p in enumerate(text):
            if p != "I":
                v = b.view(-1, 2, 1 << q)
                x, y = v[:, 0], v[:, 1]
                b = torch.stack({"Z": (x, -y), "X": (y, x), "Y": (-1j * y, 1j * x)}[p],
                                dim=1).reshape(-1)
        return float(torch.vdot(self.a, b).real)


def _read_exact(reg, case, strings, out):
    if case["read"] == "state":
        out["amplitudes"] = reg.a
    else:
        out["marginal"] = reg.a.abs().square().view(-1, 1 << LOW).sum(dim=0)
        out["paulis"] = np.array([reg.expectation(t) for t in strings])
    return out


def _exact_tfim(c):
    """<Z_0> after an Ising Trotter circuit given as op records: Rzz runs as one diagonal."""
    recs, n = c.to_ev()[0], c.num_qubits()
    reg = _Register(n)
    index = torch.arange(1 << n, device=reg.dev)
    phase = torch.zeros(1 << n, dtype=torch.float64, device=reg.dev)
    dirty, seen = False, {}
    step = 2 * n - 1
    for s in range(0, len(recs), step):
        if not seen:  # every step has the same angles
            for r in recs[:n - 1]:
                a = math.atan2(r["m"][1], r["m"][0])
                same = 1 - 2 * (((index >> int(r["q0"])) ^ (index >> int(r["q1"]))) & 1)
                phase += a * same
            seen["d"] = torch.polar(torch.ones_like(phase), phase)
            seen["x"] = [r["m"][:8].view(np.complex128).reshape(2, 2) for r in recs[n - 1:step]]
        if dirty:
            reg.flush()
        reg.a = reg.a * seen["d"]
        for q in range(n):
            reg.one(q, seen["x"][q])
        dirty = True
    reg.flush()
    p = reg.a.abs().square().view(-1, 2).sum(dim=0)
    return float((p[0] - p[1]) / (p[0] + p[1]))


def exact(case, seed):
    rng = np.random.default_rng([seed, 20])
    kind = case["kind"]
    if kind == "run":
        n = case["n"]
        reg = _Register(n)
        for op in _gates(case["circuit"], n, case["depth"], rng):
            reg.apply(*op)
        reg.flush()
        out = {"shots": None} if case["shots"] else {}
        return _read_exact(reg, case, _strings(n, rng), out)
    if kind == "steps":
        n = case["n"]
        reg, bits = _Register(n), []
        for op in _steps(n, rng):
            b = reg.apply(*op)
            if b is not None:
                bits.append(b)
        reg.flush()
        return _read_exact(reg, case, _strings(n, rng), {"bits": bits})
    if kind == "energy":
        n = case["n"]
        reg = _Register(n)
        for op in _gates("layers", n, 2, rng):
            reg.apply(*op)
        reg.flush()
        return {"terms": np.array([reg.expectation(t) for t in _chain(n)])}
    if kind == "batch":
        draws = Rng.seed_from_u64(seed)
        z = [_exact_tfim(workloads.tfim_raw(draws, case["nmin"], case["nmax"], case["smin"],
                                            case["smax"])) for _ in range(case["count"])]
        return {"z0": np.array(z), "shots": None}
    if kind == "serve":
        return None
    n, p = case["n"], case["p"]
    # rho as a vector over 2n qubits: U on the row qubits (the high n), conj(U) on the column qubits
    reg = _Register(2 * n)
    mix = 4.0 * p / 3.0  # depolarizing: rho -> (1 - mix) rho + mix (I/2 on the qubit)

    def noise(q):
        reg.flush()
        at = reg.pair(q + n, q)
        mean = 0.5 * (at(0, 0) + at(1, 1))
        reg.a = reg.a * (1.0 - mix)
        at = reg.pair(q + n, q)
        at(0, 0).add_(mix * mean)
        at(1, 1).add_(mix * mean)

    for what, q, arg in _gates("layers", n, case["depth"], rng):
        if len(q) == 1:
            m = _matrix(what, arg)
            reg.one(q[0] + n, m)
            reg.one(q[0], m.conj())
            noise(q[0])
        else:
            reg.flush()
            reg.apply(what, (q[0] + n, q[1] + n), arg)
            reg.apply(what, q, arg)
            noise(q[0])
            noise(q[1])
    reg.flush()
    return {"rho": reg.a.view(1 << n, 1 << n)}

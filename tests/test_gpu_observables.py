"""Pauli-string expectations on the device against the oracle's restatement
of PauliString::expectation (apply P to a copy, then Re <P psi|psi>,
backend/stabilizer.rs:79-125).

Bars: 1e-12 absolute in complex128 and, in complex64, against the oracle on
the same complex64 amplitudes (double-float sums on the FP32 pipe); the
stabilizer generators of a Clifford state have expectation 1 to 1e-12
(tests/stabilizer.rs:13-25 uses the statevector the same way)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from everett_gb300 import Circuit, algorithms, CudaStateVectorBackend, PauliString, State, workloads
from everett_gb300.error import QubitOutOfRange

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def random_paulis(rng, n, count):
    out = []
    for _ in range(count):
        x = rng.integers(0, 2, n).astype(bool)
        z = rng.integers(0, 2, n).astype(bool)
        out.append(PauliString(x, z, bool(rng.integers(0, 2))))
    return out


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_pauli_expectation_matches_oracle(gpu, dtype):
    rng = np.random.default_rng(11)
    for n in (1, 2, 3, 7, 12, 17):
        amps, _, _ = O.run_seeded(workloads.random_layers(n, 3, seed=n + 3))
        st = State.from_amplitudes(amps, dtype=dtype)
        ref = np.ascontiguousarray(st.amplitudes())
        ps = random_paulis(rng, n, 40)
        # plus diagonal strings sharing x = 0 and strings sharing one X part
        ps += [PauliString([False] * n, rng.integers(0, 2, n).astype(bool)) for _ in range(10)]
        x = rng.integers(0, 2, n).astype(bool)
        ps += [PauliString(x, rng.integers(0, 2, n).astype(bool), bool(rng.integers(0, 2)))
               for _ in range(19)]
        # X parts within qubits 0..2: each index's partner lies in its own
        # aligned block of 8
        for low in ((True,), (False, True), (True, False, True)):
            if len(low) > n:
                continue
            xl = np.zeros(n, dtype=bool)
            xl[:len(low)] = low
            ps += [PauliString(xl, rng.integers(0, 2, n).astype(bool), bool(rng.integers(0, 2)))
                   for _ in range(6)]
        got = st.pauli_expectation(ps)
        for p, g in zip(ps, got):
            xm, zm = p.masks()
            want = O.pauli_expectation(ref, xm, zm, p.neg)
            assert abs(g - want) < 1e-12, (n, dtype, str(p), g, want)
        # grouped evaluation equals one string at a time
        single = np.array([p.expectation(st) for p in ps[:12]])
        assert np.max(np.abs(single - got[:12])) < 1e-13


def test_clifford_state_stabilizers(gpu):
    n = 5
    c = Circuit(n)
    c.h(0)
    for q in range(n - 1):
        c.cnot(q, q + 1)
    c.s(2).h(3)
    st = CudaStateVectorBackend.run(c).state()
    # GHZ stabilizers XXXXX, Z_q Z_{q+1}, conjugated by S on qubit 2 and H on 3
    gens = ["+XXYZX", "+ZZIII", "+IZZII", "+IIZXI", "+IIIXZ"]
    vals = st.pauli_expectation(gens)
    assert np.max(np.abs(vals - 1.0)) < 1e-12, vals
    assert abs(st.pauli_expectation(["-XXYZX"])[0] + 1.0) < 1e-12
    assert abs(st.pauli_expectation(["+ZIIII"])[0]) < 1e-12


def test_pauli_expectation_rejects_foreign_qubits(gpu):
    st = State.zero(3)
    with pytest.raises(ValueError):
        PauliString.parse("+XXXX").expectation(st)
    import ctypes as C
    from everett_gb300 import _native as N
    xm = np.array([1 << 5], dtype=np.uint64)
    zm = np.zeros(1, dtype=np.uint64)
    out = np.zeros(1)
    rc = N.lib().ev_pauli_expectation(st.handle, xm.ctypes.data, zm.ctypes.data, None, 1,
                                      out.ctypes.data)
    assert rc == N.ERR_QUBIT_OUT_OF_RANGE


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_marginal_low_and_phase_estimation(gpu, dtype):
    """most_probable_phase's marginal as a device reduction: identical to the
    oracle's basis-order sums in complex128 (1e-12 in complex64, against the
    oracle on the same complex64 amplitudes), and the reference's
    phase-estimation and superdense assertions hold on the GPU
    (algorithms_phase_estimation.rs:12-36, algorithms_superdense.rs:5-36)."""
    for n, m in [(1, 0), (6, 3), (12, 12), (17, 5)]:
        amps = O.sample_state(n) if n > 1 else np.array([0.6, 0.8j])
        st = State.from_amplitudes(amps, dtype=dtype)
        got = st.marginal_low(m)
        want = O.marginal_low(np.ascontiguousarray(st.amplitudes(), dtype=np.complex128), m)
        if dtype == "complex128":
            assert np.array_equal(got, want), (n, m)
        else:
            assert np.max(np.abs(got - want)) < 1e-12, (n, m)
    for m, phi in [(1, 0.5), (2, 0.25), (2, 0.75), (3, 0.125), (3, 0.875), (4, 0.0)]:
        ex = CudaStateVectorBackend.run(algorithms.phase_estimation(m, phi))
        assert abs(algorithms.most_probable_phase(ex.state(), m) - phi) < 1e-10
    ex = CudaStateVectorBackend.run(algorithms.phase_estimation(4, 0.3))
    assert abs(algorithms.most_probable_phase(ex.state(), 4) - 0.3) <= 1.0 / 16.0 + 1e-10
    for b0 in (False, True):
        for b1 in (False, True):
            ex = CudaStateVectorBackend.run(algorithms.superdense_circuit(b0, b1))
            assert list(ex.classical()) == [b0, b1]


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 11, 12, 13, 19])
def test_many_groups_from_one_read(gpu, n, dtype):
    """Terms of many X parts evaluated from shared-memory tiles (each within
    the tile's qubits), beside X parts too wide for a tile and more Z-only
    terms than one pass takes: registers below, at and above a tile's 2^11
    (complex128) and 2^12 (complex64) amplitudes, both Y parities, signs."""
    rng = np.random.default_rng(n)
    amps, _, _ = O.run_seeded(workloads.random_layers(n, 3, seed=n + 5), parallel=True)
    st = State.from_amplitudes(amps, dtype=dtype)
    ref = np.ascontiguousarray(st.amplitudes())
    texts = []
    for q in range(n):  # every site, and strings from it to the far end
        for p in "XY":
            texts.append("I" * q + p + "I" * (n - q - 1))
        texts.append("-" + "I" * q + "Y" + "Z" * (n - q - 1))
    for q in range(n - 1):
        texts += ["I" * q + p + "I" * (n - q - 2) for p in ("ZZ", "XX", "XY", "YY", "ZX")]
    ps = [PauliString.parse(t) for t in texts] + random_paulis(rng, n, 6)
    ps += [PauliString([False] * n, rng.integers(0, 2, n).astype(bool), bool(rng.integers(0, 2)))
           for _ in range(25)]
    ps = [ps[i] for i in rng.permutation(len(ps))]
    got = st.pauli_expectation(ps)
    for p, g in zip(ps, got):
        xm, zm = p.masks()
        want = O.pauli_expectation(ref, xm, zm, p.neg)
        assert abs(g - want) < 1e-12, (n, dtype, str(p), g, want)


def test_marginal_low_complex64_bits(gpu):
    """complex64 marginals square each part exactly on the integer pipes: the
    f64 sums of the exact squares in basis order, for zero, subnormal, tiny,
    ordinary and huge parts and odd numbers of terms per bin."""
    rng = np.random.default_rng(3)
    n = 11
    a = (rng.normal(size=1 << n) * 10.0 ** rng.integers(-44, 38, 1 << n)).astype(np.float32)
    b = (rng.normal(size=1 << n) * 10.0 ** rng.integers(-44, 38, 1 << n)).astype(np.float32)
    a[:40], b[20:60] = 0.0, 0.0
    amps = a.astype(np.complex128) + 1j * b.astype(np.complex128)
    st = State.from_amplitudes(amps, dtype="complex64")
    x, y = a.astype(np.float64), b.astype(np.float64)
    terms = x * x + y * y  # both squares are exact in f64
    for m in (0, 3, 8, 10, 11):
        want = np.zeros(1 << m)
        for row in terms.reshape(-1, 1 << m):
            want = want + row
        assert np.array_equal(st.marginal_low(m), want), m


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [11, 12, 14])
def test_masks_within_a_tile(gpu, n, dtype):
    """X masks of one and of several bits at every place of a tile (thread
    bits, one slot bit, several, both), with Z bits nowhere, among the thread
    bits and among the slot bits, inside and outside the tile, both Y
    parities: the same bar as above."""
    rng = np.random.default_rng(100 + n)
    amps, _, _ = O.run_seeded(workloads.random_layers(n, 3, seed=n + 9), parallel=True)
    st = State.from_amplitudes(amps, dtype=dtype)
    ref = np.ascontiguousarray(st.amplitudes())
    ps = []
    for width in (1, 2, 3, 5):
        for _ in range(12):
            x = np.zeros(n, dtype=bool)
            x[rng.choice(min(n, 11), width, replace=False)] = True
            z = rng.integers(0, 2, n).astype(bool) & (rng.uniform(size=n) < rng.choice([0.0, 0.2, 0.6]))
            ps.append(PauliString(list(x), list(z), bool(rng.integers(0, 2))))
    for first in range(0, len(ps), 8):  # few masks a call: they share a tile
        got = st.pauli_expectation(ps[first:first + 8])
        for p, g in zip(ps[first:first + 8], got):
            xm, zm = p.masks()
            want = O.pauli_expectation(ref, xm, zm, p.neg)
            assert abs(g - want) < 1e-12, (n, dtype, str(p), g, want)


FULL_PASS = """
import numpy as np
from everett_gb300 import Gate1, State
n = 22
st = State.zero(n, "complex64")
for q in range(n):
    st.apply_1q(q, Gate1.ry(0.1 + 0.05 * q))
chain = ["I" * q + "X" + "I" * (n - q - 1) for q in range(12)]
chain += ["I" * q + "ZZ" + "I" * (n - q - 2) for q in range(8)]
angle = 0.1 + 0.05 * np.arange(n)
want = list(np.sin(angle[:12])) + list(np.cos(angle[:8]) * np.cos(angle[1:9]))
print(np.max(np.abs(st.pauli_expectation(chain) - want)))
"""


def test_full_pauli_passes_fill_the_gpu(gpu):
    """A complex64 tile pass of 20 terms, X and Z, has three blocks on every
    SM in one wave, and the values hold there (22 rotations in single
    precision, each within 3 units of 2^-24: 8e-6 of an expectation)."""
    import torch
    r = subprocess.run([sys.executable, "-c", FULL_PASS], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, EV_DEBUG="1"), cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert float(r.stdout) < 1e-5
    lines = [x for x in r.stderr.splitlines() if "k_pauli_tile 20 terms" in x]
    assert len(lines) == 1 and " 3 CTAs/SM" in lines[0], r.stderr
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert lines[0].endswith(f"grid {min(3 * sms, 1 << (22 - 12))}"), lines


SHARED = """
import numpy as np
import sys
from everett_gb300 import Gate1, PauliString, State
n, dtype, masks, g = int(sys.argv[1]), sys.argv[2], 2, int(sys.argv[3])
st = State.zero(n, dtype)
for q in range(n):
    st.apply_1q(q, Gate1.ry(0.1 + 0.05 * q))
rng = np.random.default_rng(3)
ps, want = [], []
for m in range(masks):
    for t in range(g):
        z = rng.integers(0, 2, n).astype(bool)
        z[m + 3] = False
        x = np.arange(n) == m + 3
        ps.append(PauliString(list(x), list(z)))
        a = 0.1 + 0.05 * np.arange(n)
        want.append(np.prod(np.where(x, np.sin(a), np.where(z, np.cos(a), 1.0))))
print(np.max(np.abs(st.pauli_expectation(ps) - np.array(want))))
"""


@pytest.mark.parametrize("n,dtype,g,tiles", [
    (22, "complex64", 6, 1), (22, "complex64", 7, 0), (23, "complex64", 3, 1), (23, "complex64", 4, 0),
    (24, "complex64", 2, 1), (24, "complex64", 3, 0), (25, "complex64", 1, 1), (25, "complex64", 2, 0),
    (25, "complex64", 8, 0), (22, "complex128", 8, 1), (23, "complex128", 5, 1),
    (23, "complex128", 6, 0), (24, "complex128", 4, 1), (24, "complex128", 5, 0),
    (24, "complex128", 8, 0)])
def test_terms_of_one_mask_share_their_pairs(gpu, n, dtype, g, tiles):
    """Two X masks of g terms each on a large register: from the rule's line
    on each mask takes one read that forms its pairs once, below it both go
    to one tile pass.  Values as above (complex64: n rotations of 2^-22.4
    each, twice)."""
    r = subprocess.run([sys.executable, "-c", SHARED, str(n), dtype, str(g)], capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, EV_DEBUG="1"), cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert float(r.stdout) < (1e-12 if dtype == "complex128" else 1e-5)
    assert sum("k_pauli_tile" in x for x in r.stderr.splitlines()) == tiles, r.stderr


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_more_terms_than_results_wait_on_the_device(gpu, dtype):
    """2500 terms in one call, whose sums come back in several copies: masks
    of one term, of many (both Y parities), wide ones and Z strings, shuffled."""
    n = 13
    rng = np.random.default_rng(8)
    amps, _, _ = O.run_seeded(workloads.random_layers(n, 3, seed=4), parallel=True)
    st = State.from_amplitudes(amps, dtype=dtype)
    ref = np.ascontiguousarray(st.amplitudes())
    xs = [rng.uniform(size=n) < f for f in (0.1, 0.2, 0.3, 1.0) for _ in range(40)]
    ps = random_paulis(rng, n, 300)
    ps += [PauliString([False] * n, rng.integers(0, 2, n).astype(bool)) for _ in range(200)]
    ps += [PauliString(xs[int(rng.integers(len(xs)))], rng.integers(0, 2, n).astype(bool),
                       bool(rng.integers(0, 2))) for _ in range(2000)]
    ps = [ps[i] for i in rng.permutation(len(ps))]
    got = st.pauli_expectation(ps)
    for p, g in zip(ps, got):
        xm, zm = p.masks()
        want = O.pauli_expectation(ref, xm, zm, p.neg)
        assert abs(g - want) < 1e-12, (dtype, str(p), g, want)


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_marginal_sums_of_every_length(gpu, dtype):
    """Sums shorter than, equal to and longer than the amplitudes that are on
    their way together, over zeros and dense values: the f64 sum in basis
    order (complex128 squares as the oracle's norm_sqr: x x + y y, the second
    product rounded into the first's sum once or twice)."""
    n = 12
    rng = np.random.default_rng(5)
    for zeros in (0.0, 0.6, 0.99):
        amps = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        amps[rng.uniform(size=1 << n) < zeros] = 0.0
        if dtype == "complex64":
            amps = amps.astype(np.complex64).astype(np.complex128)
        st = State.from_amplitudes(amps, dtype=dtype)
        terms = amps.real ** 2 + amps.imag ** 2
        for m in range(n + 1):
            want = np.zeros(1 << m)
            for row in terms.reshape(-1, 1 << m):
                want = want + row
            got = st.marginal_low(m)
            if dtype == "complex64":  # exact squares
                assert np.array_equal(got, want), (zeros, m)
            else:  # one rounding more or less per term
                assert np.max(np.abs(got - want)) <= 2.0 ** -51 * (1 << (n - m)) * terms.max(), (zeros, m)


def test_marginal_times_by_length_and_content(gpu):
    """Few long sums: four times the terms take at most five times as long
    (the loads of a register beyond the L2 cache stay ahead of the adds), and
    a state of zeros takes as long as a dense one."""
    import time

    def seconds(st, m):
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            st.marginal_low(m)
            best = min(best, time.perf_counter() - t)
        return best

    def holds(a, b, factor):  # a machine at work may spoil one attempt
        return any(seconds(*a) <= factor * seconds(*b) for _ in range(4))

    short, long = State.zero(22, "complex128"), State.zero(24, "complex128")
    assert holds((long, 8), (short, 8), 5.0)
    sparse = State.zero(24, "complex64")
    dense = CudaStateVectorBackend.run(workloads.random_layers(24, 1, seed=2), dtype="complex64").state()
    assert holds((sparse, 12), (dense, 12), 1.2)

"""The tile pass's default tile per register size (tiles of 2^8, 2^10 and 2^12
amplitudes, rows of 2^2 or 2^4) against the oracle, on both sides of every
edge of the rule, with moves (CNOT, CZ, SWAP) between arithmetic gates on
other qubits, which the pass planner carries across each other.

complex128 equals the oracle (==: the carried moves change no bit);
complex64 keeps fidelity >= 1 - 1e-6."""
import numpy as np
import pytest

import oracle as O
from everett_gb300 import Circuit, CudaStateVectorBackend, Gate1, Gate2, algorithms

pytestmark = pytest.mark.gpu


def interleaved(n, seed, count):
    rng = np.random.default_rng(seed)
    c = Circuit(n)
    for q in range(n):
        c.h(q)
    for _ in range(count):
        q = [int(v) for v in rng.choice(n, min(n, 4), replace=False)]
        k = int(rng.integers(0, 8))
        if n < 2 or k < 2:
            c.rz(q[0], rng.uniform(0, 6)).ry(q[0], rng.uniform(0, 6))
        elif k < 5:
            c.gate2([Gate2.cnot(), Gate2.cz(), Gate2.swap()][k - 2], q[0], q[1])
        elif k == 5:
            c.controlled(q[1:3], Gate1.ry(0.3), q[0])
        elif k == 6:
            c.gate2(Gate2.rzz(rng.uniform(0, 6)), q[0], q[1])
        else:
            c.gate2(Gate2.controlled(Gate1.rx(0.9)), q[0], q[1])
    return c


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 10, 16, 17, 18, 19, 21, 22])
def test_default_tiles_bit_exact(gpu, n):
    c = interleaved(n, n, 160 if n < 18 else 60)
    want, _, rc = O.run_seeded(c, 0, parallel=True)
    assert rc == 0
    got = CudaStateVectorBackend.run(c).state().amplitudes()
    assert np.array_equal(got, want)
    single = CudaStateVectorBackend.run(c, dtype="complex64").state().amplitudes()
    fid = abs(np.vdot(want, single)) ** 2 / (np.vdot(single, single).real * np.vdot(want, want).real)
    assert fid > 1 - 1e-6


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_default_tiles_replayed(gpu, dtype):
    """A prepared run with measurements between its tile passes (passes that
    may start before the previous kernel ends, captured into a graph) equals
    the same run launched kernel by kernel."""
    n = 11
    c = Circuit.with_classical(n, 2)
    c.compose(interleaved(n, 5, 40)).measure(3, 0).x_if(0, 7)
    c.compose(algorithms.qft(n)).measure(n - 1, 1)
    st = CudaStateVectorBackend.run_seeded(c, 9, dtype=dtype)
    again = CudaStateVectorBackend(n, dtype=dtype).state()
    prepared = CudaStateVectorBackend.prepare(again, c)
    for _ in range(3):
        assert prepared.launch(9) == st.classical()
        assert np.array_equal(again.amplitudes(), st.state().amplitudes())
    prepared.close()


def every_record_kind(n, seed, count):
    """1-qubit kinds (real, Rx-like, dense, diagonal, phase, anti-diagonal,
    identity) free and under one to three controls, CNOT, CZ, SWAP, parity
    and general diagonals and a dense 4x4, on random positions."""
    rng = np.random.default_rng(seed)
    ones = [Gate1.h(), Gate1.ry(0.4), Gate1.rx(0.7), Gate1.rz(1.1), Gate1.phase(0.9), Gate1.t(),
            Gate1.x(), Gate1.y(), Gate1.z(), Gate1.id(),
            Gate1(0.6 + 0.1j, -0.3 + 0.2j, 0.25 - 0.7j, 0.1 + 0.05j)]
    unit = np.exp(1j * rng.uniform(0, 6, 4))
    twos = [Gate2.cnot(), Gate2.cz(), Gate2.swap(), Gate2.rzz(0.8), Gate2(np.diag(unit)),
            Gate2(np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))[0])]
    c = Circuit(n)
    for q in range(n):
        c.h(q)
    for _ in range(count):
        q = [int(v) for v in rng.choice(n, 4, replace=False)]
        k = int(rng.integers(0, 3))
        if k == 0:
            c.gate1(ones[int(rng.integers(len(ones)))], q[0])
        elif k == 1:
            c.controlled(q[1:2 + int(rng.integers(3))], ones[int(rng.integers(len(ones)))], q[0])
        else:
            c.gate2(twos[int(rng.integers(len(twos)))], q[0], q[1])
    return c


@pytest.mark.parametrize("n,tile_bits", [(12, 12), (13, 13), (14, 14), (15, 12), (16, 13)])
def test_stages_equal_sweeps(gpu, monkeypatch, n, tile_bits):
    """complex64 records in stages (16 amplitudes a thread in registers)
    against one sweep per record on the same tiles (the 256-thread block
    shape): each amplitude sees the same operations in the same order, so the
    bits agree; and the oracle's amplitudes to the complex64 bar."""
    c = every_record_kind(n, 100 * n + tile_bits, 400)
    staged = CudaStateVectorBackend.run(c, dtype="complex64", tile_bits=tile_bits).state().amplitudes()
    monkeypatch.setenv("EV_TILE_THREADS", "256")
    swept = CudaStateVectorBackend.run(c, dtype="complex64", tile_bits=tile_bits).state().amplitudes()
    assert np.array_equal(staged, swept)
    want, _, _ = O.run_seeded(c, 0, parallel=True)
    want = want / np.linalg.norm(want)
    assert np.max(np.abs(staged - want)) < 1e-5


@pytest.mark.parametrize("n", [15, 20, 23])
def test_default_tiles_at_the_other_edges(gpu, n):
    """The sizes beside the remaining edges: 15 and 20 qubits (complex64
    tiles of 2^8 | 2^10 and 2^10 | 2^12; complex128 between two registers in
    tiles of 2^11), 23 (complex64 tiles of 2^13)."""
    test_default_tiles_bit_exact(gpu, n)

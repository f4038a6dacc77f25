"""complex128 gates on sparse states, whose zero amplitudes skip the
arithmetic, and real matrices of one magnitude (H and its sign variants),
whose products are shared: the oracle's bits, per gate and in tile passes;
a non-finite matrix entry still reaches zero amplitudes."""
import numpy as np
import pytest

import oracle as O
from everett_gb300 import Circuit, CudaStateVectorBackend, Gate1, Gate2, State

pytestmark = pytest.mark.gpu

R = 0.7071067811865476
GATES = [Gate1.h(), Gate1(R, -R, R, R), Gate1(-R, R, R, R), Gate1(-R, -R, -R, R), Gate1(2.0, 2.0, 2.0, -2.0),
         Gate1(R, R, R, np.nextafter(-R, 0)), Gate1.ry(0.7), Gate1.rx(0.4), Gate1.rz(1.3), Gate1.t(),
         Gate1.x(), Gate1.y(), Gate1(0.6 + 0.1j, -0.3 + 0.2j, 0.25 - 0.7j, 0.1 + 0.05j)]


def sparse(n, seed, keep):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    a[rng.random(1 << n) >= keep] = 0.0
    part = rng.random(1 << n) < 0.1
    a[part] = a[part].real
    a[rng.random(1 << n) < 0.02] *= 1e-200
    return a


@pytest.mark.parametrize("n,keep", [(1, 0.5), (5, 0.1), (6, 0.5), (9, 0.03), (9, 0.9), (13, 0.2)])
def test_gates_on_sparse_states(gpu, n, keep):
    base = sparse(n, n, keep)
    st = State.from_amplitudes(base)
    for k in {0, n // 2, n - 1}:
        for g in GATES:
            st.upload(base)
            st.apply_1q(k, g)
            want = base.copy()
            O.apply_1q(want, k, g)
            assert np.array_equal(st.amplitudes(), want), (n, k, g)
            if n > 1:
                st.upload(base)
                st.apply_controlled_1q([(k + 1) % n], k, g)
                want = base.copy()
                O.apply_controlled_1q(want, [(k + 1) % n], k, g)
                assert np.array_equal(st.amplitudes(), want), (n, k, g)


@pytest.mark.parametrize("n,keep", [(2, 0.5), (6, 0.3), (11, 0.05)])
def test_two_qubit_gates_on_sparse_states(gpu, n, keep):
    rng = np.random.default_rng(n)
    base = sparse(n, 50 + n, keep)
    st = State.from_amplitudes(base)
    for g in (Gate2(rng.normal(size=16) + 1j * rng.normal(size=16)), Gate2.rzz(0.7),
              Gate2(np.diag(np.exp(1j * rng.uniform(0, 6, 4)))), Gate2.controlled(Gate1.ry(0.4))):
        for a, b in ((0, n - 1), (n - 1, 0)):
            st.upload(base)
            st.apply_2q(a, b, g)
            want = base.copy()
            O.apply_2q(want, a, b, g)
            assert np.array_equal(st.amplitudes(), want), (n, a, b)


@pytest.mark.parametrize("n", [6, 10, 13, 18])
def test_tiled_from_a_basis_state(gpu, n):
    """Gates that leave most of the register in |0> for long, then fill it."""
    rng = np.random.default_rng(n)
    c = Circuit(n)
    for q in range(n):
        for _ in range(3):
            c.gate1(GATES[int(rng.integers(len(GATES)))], q)
        if q:
            c.gate2([Gate2.cnot(), Gate2.cz(), Gate2.rzz(0.4)][q % 3], q - 1, q)
    want, _, _ = O.run_seeded(c, 0, parallel=True)
    for mode in ("exact", "tiled"):
        assert np.array_equal(CudaStateVectorBackend.run(c, mode=mode).state().amplitudes(), want)


@pytest.mark.parametrize("entry", [np.inf, np.nan])
def test_non_finite_entries_reach_zeros(gpu, entry):
    for g in (Gate1(entry, 0.3j, 0.4, 0.5 + 0.5j), Gate1(complex(0.5, 0.5), 0, 0, complex(entry, 0.5)),
              Gate1(1, 0, 0, complex(entry, 0.5)), Gate1(entry, R, R, R)):
        want = np.zeros(1 << 6, dtype=complex)
        want[0] = 1.0
        st = State.from_amplitudes(want)
        O.apply_1q(want, 2, g)
        st.apply_1q(2, g)
        assert np.array_equal(st.amplitudes(), want, equal_nan=True)
        for two in (Gate2.controlled(g), Gate2(np.diag([0.5 + 0.5j] * 3 + [complex(entry, 0.5)])),
                    Gate2(np.full((4, 4), 0.5 + 0.5j) + np.diag([0, 0, 0, entry]))):
            st2 = State.from_amplitudes(np.eye(1, 1 << 6, dtype=complex)[0])
            want2 = np.eye(1, 1 << 6, dtype=complex)[0].copy()
            O.apply_2q(want2, 4, 1, two)
            st2.apply_2q(4, 1, two)
            assert np.array_equal(st2.amplitudes(), want2, equal_nan=True)
        c = Circuit(6)
        c.gate1(g, 2)
        tiled = CudaStateVectorBackend.run(c).state().amplitudes()
        assert np.array_equal(tiled, want, equal_nan=True)

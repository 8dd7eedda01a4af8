"""States small enough to run whole in shared memory: every gate kind at
sizes below, at and above the three register qubits of a sweep and up to the
route's largest, lists longer than one launch's chunks, and the batch kernel
on the same lists, all against the oracle (and batch against handles)."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from oracle import pyoracle as po
from tests.test_plan import mixed_circuit


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def oracle(n, ops, init=None):
    po.set_fast(True)
    o = po.OracleState(n, 0)
    if init is not None:
        o.set_state(init)
    o.apply(C.ops_to_array(ops))
    v = o.state()
    o.close()
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 2e-5)])
@pytest.mark.parametrize("n,count", [(3, 80), (4, 200), (5, 60), (8, 1500), (9, 120), (10, 300), (11, 200), (12, 250)])
def test_all_gate_kinds(n, count, precision, tol):
    ops = [C.Op(C.RX, [q], 0.3 + q) for q in range(n)] + mixed_circuit(n, count, 90 + n)
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init /= np.linalg.norm(init)
    with qb.QuantumState(n, precision=precision) as st:
        launches = st.launch_count()
        st.execute(ops)
        assert st.launch_count() - launches <= 1 + count // 100
        assert rel_l2(st.get_state_vector(), oracle(n, ops)) < tol
        st.set_state_vector(init)
        st.execute(ops)
        assert rel_l2(st.get_state_vector(), oracle(n, ops, init)) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2])
def test_fewer_qubits_than_a_sweep_takes(n):
    ops = []
    for k in range(40):
        ops += [C.Op(C.H, [k % n]), C.Op(C.RZ, [(k + 1) % n], 0.2 * k), C.Op(C.RY, [k % n], 0.1 * k), C.Op(C.T, [k % n])]
        if n == 2:
            ops += [C.Op(C.CNOT, [k % 2, 1 - k % 2]), C.Op(C.SWAP, [0, 1]), C.Op(C.CPHASE, [0, 1], 0.3)]
    with qb.QuantumState(n) as st:
        st.execute(ops)
        assert rel_l2(st.get_state_vector(), oracle(n, ops)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_batch_circuits_match_handles(precision, tol):
    sizes = [3, 4, 7, 9, 11, 12] + ([13] if precision == "f32" else [])
    with qb.Batch(precision) as b:
        want = []
        for n in sizes:
            ops = [C.Op(C.H, [0])] + mixed_circuit(n, 60 + 40 * n, n)
            masks = [1, (1 << n) - 1, 1 << (n - 1), 0]
            b.add(n, ops, masks)
            with qb.QuantumState(n) as st:
                st.execute(ops)
                want.append(st.expect_z(masks))
        b.run()
        first = b.results()
        b.run()
        assert np.max(np.abs(first - np.concatenate(want))) < tol
        assert np.array_equal(first, b.results())

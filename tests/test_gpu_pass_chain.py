"""Runs of unitary passes carry their norm without measuring it, and a reset
followed by a pass is not written: op lists with resets, re-initialisations
and non-unitary matrices inside them equal the same list given call by call
(the calls re-measure the norm, hence the tolerance of rounding), and the
oracle."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from oracle import pyoracle as po


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def pieces(n):
    a = C.random_layered(n, 5, 7 * n, initial_h=True)
    b = C.random_layered(n, 4, 7 * n + 1)
    return a, b


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), ("f32", 1e-5)])
@pytest.mark.parametrize("jit", [qb.QOA_JIT_OFF, qb.QOA_JIT_SYNC])
@pytest.mark.parametrize("n", [5, 11, 12, 16])
def test_resets_inside_a_list(n, jit, precision, tol):
    a, b = pieces(n)
    reset = [C.Op(C.RESETALL)]
    for ops, last in ((a + reset + b, b), (reset + a + reset + reset + b, b), (a + reset, []), (reset, []), (reset + b + a, b + a)):
        with qb.QuantumState(n, precision=precision) as x, qb.QuantumState(n, precision=precision) as y:
            x.set_jit(jit, min_qubits=11)
            x.execute(a)
            for _ in range(3):  # planned, kept, from the kept plan
                x.execute(ops)
                got = x.get_state_vector()
                y.apply_reset_all()
                for op in last:
                    y.execute([op])
                assert rel_l2(got, y.get_state_vector()) < tol
                assert x.get_status()["zero_norm_resets"] == 0


@pytest.mark.gpu
def test_reinit_inside_a_list():
    a, b = pieces(13)
    with qb.QuantumState(13) as x, qb.QuantumState(12) as y:
        x.execute(a + [C.Op(C.QINIT, [12])] + C.random_layered(12, 3, 5))
        y.execute(C.random_layered(12, 3, 5))
        assert x.n == 12
        assert rel_l2(x.get_state_vector(), y.get_state_vector()) < 1e-13
        x.execute(a[:3] + [C.Op(C.QINIT, [12])])
        v = x.get_state_vector()
        assert v[0] == 1 and np.count_nonzero(v) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("n", [11, 14, 17])
def test_non_unitary_matrices_between_passes(n):
    rng = np.random.default_rng(n)
    a, b = pieces(n)
    ops = list(a)
    for q in range(0, n, 3):
        m = rng.standard_normal(4) + 1j * rng.standard_normal(4)
        ops += [C.Op(C.U1, [q], 0.0, m)] + b[q * n:(q + 1) * n]
    ops += b
    po.set_fast(True)
    o = po.OracleState(n, 0)
    o.apply(C.ops_to_array(ops))
    with qb.QuantumState(n) as st:
        st.execute(ops)
        assert rel_l2(st.get_state_vector(), o.state()) < 1e-12
    o.close()

"""A few 4x4 gates or controlled SWAPs alone in their passes run on their own
kernels: one launch each, the same state as inside a pass, the norm carried
across them, and what is not unitary still measured."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from oracle import pyoracle as po
from tests.test_plan import oracle_state, rel_l2

TOL = {"f64": 1e-12, "f32": 1e-5}


def unitary(seed):
    g = np.random.default_rng(seed)
    return np.linalg.qr(g.standard_normal((4, 4)) + 1j * g.standard_normal((4, 4)))[0].reshape(-1)


def u2(q1, q2, seed=1):
    return C.Op(C.U2, [q1, q2], 0.0, unitary(seed))


def start(n):
    return [C.Op(C.H, [q]) for q in range(n)] + [C.Op(C.RZ, [q], 0.1 + 0.2 * q) for q in range(n)] + \
           [C.Op(C.RX, [q], 0.3 * q) for q in range(n)]


def state_after(n, precision, lists):
    po.set_fast(True)
    with qb.QuantumState(n, precision=precision) as st:
        for ops in lists:
            st.execute(ops)
        got = st.get_state_vector().astype(np.complex128)
    return got, oracle_state(n, [o for ops in lists for o in ops], 0)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [13, 16, 20])
@pytest.mark.parametrize("precision,op", [("f64", u2(2, 11)), ("f64", u2(12, 0)), ("f64", C.Op(C.CSWAP, [12, 0, 7])),
                                          ("f32", C.Op(C.CSWAP, [3, 12, 1]))])
def test_alone_it_is_one_launch(n, precision, op):
    with qb.QuantumState(n, precision=precision) as st:
        st.execute(start(n))
        before = st.launch_count()
        st.execute([op])
        assert st.launch_count() - before == 1
        got = st.get_state_vector().astype(np.complex128)
    assert rel_l2(got, oracle_state(n, start(n) + [op], 0)) < TOL[precision]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [13, 15])
def test_between_passes_and_after_resets(n, precision):
    one = [C.Op(C.CSWAP, [1, 8, n - 1])]
    two = one + [C.Op(C.CSWAP, [n - 2, 0, 9])]
    six = two + [C.Op(C.CSWAP, [3 + k, 4 + k, (9 + k) % n]) for k in range(4)]
    lists = [[start(n), one, start(n)], [start(n) + one], [start(n), two, two], [start(n), six, six],
             [start(n), [C.Op(C.RESETALL)] + one], [start(n), [C.Op(C.RESETALL), C.Op(C.X, [1]), C.Op(C.X, [8])] + one]]
    if precision == "f64":
        w = [u2(0, 10, 3)]
        lists += [[start(n), w, start(n)], [start(n) + w + start(n)], [start(n), [C.Op(C.RESETALL)] + w],
                  [start(n), w + one, w + [u2(10, 12, 4)], w + [u2(10, 12, 4), u2(12, 5, 5)] + one]]
    for ls in lists:
        got, want = state_after(n, precision, ls)
        assert rel_l2(got, want) < TOL[precision]


@pytest.mark.gpu
def test_one_that_is_not_unitary_is_measured():
    n = 13
    m = 3.0 * unitary(7).reshape(4, 4)
    m[2] *= 0.5
    op = C.Op(C.U2, [4, 12], 0.0, m.reshape(-1))
    got, want = state_after(n, "f64", [start(n), [op]])
    assert abs(np.linalg.norm(got) - 1) < 1e-12
    assert rel_l2(got, want) < 1e-12
    with qb.QuantumState(n) as st:
        st.execute(start(n))
        st.execute([C.Op(C.U2, [4, 12], 0.0, np.full(16, np.nan, dtype=complex))])
        assert st.get_status()["nan"]
        assert st.get_probabilities()[0] == 1.0


@pytest.mark.gpu
def test_long_lists_of_them_repeat_alike():
    n = 14
    g = np.random.default_rng(8)
    ops = []
    for k in range(60):
        q = [int(x) for x in g.permutation(n)[:3]]
        ops.append(C.Op(C.CSWAP, q) if k % 3 else u2(q[0], q[1], 100 + k))
    with qb.QuantumState(n) as st:
        out = []
        for _ in range(3):
            st.execute([C.Op(C.QINIT, [n])] + start(n) + ops)
            out.append(st.get_state_vector())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert rel_l2(out[0], oracle_state(n, start(n) + ops, 0)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [13, 17, 19, 20])
def test_short_lists_of_every_mix(n, precision):
    """at each side of the rule's lines, alone and with a gate of a pass beside them"""
    g = np.random.default_rng(n)
    for case in range(14):
        ops = []
        for k in range(1 + case % 7):
            q = [int(x) for x in g.permutation(n)[:3]]
            ops.append(C.Op(C.CSWAP, q) if precision == "f32" or (case + k) % 3 else u2(q[0], q[1], 10 * case + k))
        if case % 4 == 3:
            ops.insert(len(ops) // 2, C.Op(C.CNOT, [0, n - 1]))
        got, want = state_after(n, precision, [start(n), ops, ops])
        assert rel_l2(got, want) < TOL[precision]


@pytest.mark.gpu
@pytest.mark.parametrize("zero", [np.zeros(4, dtype=complex), np.full(4, np.nan, dtype=complex)])
def test_after_a_gate_that_leaves_no_state(zero):
    """A zero or NaN vector is |0..0> to the next gate, whatever kernel runs it."""
    n = 13
    op = u2(12, 1, 6)
    with qb.QuantumState(n) as st, qb.QuantumState(n) as ref:
        st.execute(start(n))
        st.execute([C.Op(C.U1, [3], 0.0, zero)])
        st.execute([op])
        ref.execute([op])
        assert np.max(np.abs(st.get_state_vector() - ref.get_state_vector())) < 1e-15
        st.execute([C.Op(C.U1, [3], 0.0, zero)])
        st.execute([C.Op(C.CSWAP, [1, 2, 12]), C.Op(C.CSWAP, [4, 2, 11])])
        assert st.get_probabilities()[0] == 1.0
        st.execute([op])
        assert np.max(np.abs(st.get_state_vector() - ref.get_state_vector())) < 1e-15

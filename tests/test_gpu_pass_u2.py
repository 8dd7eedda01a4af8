"""4x4 gates and controlled SWAPs inside tile passes: dense lists over every
pair of qubits (lane, register, warp and outside the tile, both operand
orders) against the oracle, interpreter and generated kernels alike, on
handles and in batches."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from oracle import pyoracle as po


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def dense(n, count, seed):
    rng = np.random.default_rng(seed)
    ops = [C.Op(C.RY, [q], 0.4 + q) for q in range(n)]
    for _ in range(count):
        q = [int(x) for x in rng.permutation(n)[:3]]
        k = rng.integers(5)
        if k < 2:
            u, _ = np.linalg.qr(rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)))
            ops.append(C.Op(C.U2, q[:2], 0.0, u.reshape(-1)))
        elif k == 2:
            ops.append(C.Op(C.CSWAP, q))
        elif k == 3:
            ops.append(C.Op(C.CPHASE, q[:2], 0.7))
        else:
            ops.append(C.Op(C.RX, q[:1], 1.1))
    return ops


def oracle(n, ops):
    po.set_fast(True)
    o = po.OracleState(n, 0)
    o.apply(C.ops_to_array(ops))
    v = o.state()
    o.close()
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("search", [False, True])
@pytest.mark.parametrize("n,count", [(13, 120), (14, 60), (16, 150), (18, 80)])
def test_handles(n, count, search):
    ops = dense(n, count, n)
    ref = oracle(n, ops)
    got = []
    for jit in (qb.QOA_JIT_OFF, qb.QOA_JIT_SYNC):
        with qb.QuantumState(n, slot_search=search) as st:
            st.set_jit(jit, min_qubits=11)
            before = st.launch_count()
            st.execute(ops)
            assert st.launch_count() - before < count // 3  # passes, not a launch per gate
            got.append(st.get_state_vector())
    assert np.array_equal(got[0].view(np.float64), got[1].view(np.float64))
    assert rel_l2(got[0], ref) < 1e-12
    with qb.QuantumState(n, precision="f32") as st:
        st.execute(ops)
        assert rel_l2(st.get_state_vector(), ref) < 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_batches(precision, tol):
    with qb.Batch(precision) as b:
        want = []
        for n in (13, 14, 15):
            ops = dense(n, 40, 3 * n)
            masks = [1, (1 << n) - 1, 5 << (n - 4)]
            b.add(n, ops, masks)
            with qb.QuantumState(n) as st:
                st.execute(ops)
                want.append(st.expect_z(masks))
        for _ in range(2):
            b.run()
            assert np.max(np.abs(b.results() - np.concatenate(want))) < tol

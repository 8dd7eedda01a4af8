"""Lists of one gate on states that run whole in shared memory: the gate's own
kernel where the stored vector is the state, the shared-memory launch where it
may not be; the same states either way."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from tests.test_gpu_own_kernels import TOL, start, u2
from tests.test_plan import oracle_state, rel_l2


def gates(n):
    g = [C.Op(C.H, [n - 1]), C.Op(C.X, [0]), C.Op(C.Y, [n // 2]), C.Op(C.Z, [0]), C.Op(C.T, [n - 1]), C.Op(C.RX, [0], 0.7),
         C.Op(C.RY, [n - 1], 4.1), C.Op(C.RZ, [0], 1.3), C.Op(C.P, [n // 2], 0.4),
         C.Op(C.U1, [0], 0.0, np.array([0.6, 0.8j, 0.8j, 0.6]))]
    if n > 1:
        g += [C.Op(C.CNOT, [0, n - 1]), C.Op(C.CZ, [n - 1, 0]), C.Op(C.CPHASE, [0, n - 1], 0.9), C.Op(C.SWAP, [0, n - 1]),
              C.Op(C.CY, [n - 1, 0]), u2(n - 1, 0)]
    if n > 2:
        g += [C.Op(C.CSWAP, [0, 1, 2]), C.Op(C.TOFFOLI, [n - 1, 0, 1])]
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 5, 10, 12])
def test_one_gate_at_a_time(n, precision):
    with qb.QuantumState(n, precision=precision) as st:
        st.execute(start(n))
        for op in gates(n):
            before = st.launch_count()
            st.execute([op])
            assert st.launch_count() - before == 1
        got = st.get_state_vector().astype(np.complex128)
    assert rel_l2(got, oracle_state(n, start(n) + gates(n), 0)) < TOL[precision]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("bad", [np.zeros(4, dtype=complex), np.full(4, np.nan, dtype=complex),
                                 np.array([3.0, 0, 0, 0.5], dtype=complex)])
def test_after_one_that_is_not_unitary(bad, precision):
    n = 6
    with qb.QuantumState(n, precision=precision) as st, qb.QuantumState(n, precision=precision) as ref:
        st.execute(start(n))
        st.execute([C.Op(C.U1, [3], 0.0, bad)])
        kept = st.get_state_vector()
        assert abs(np.linalg.norm(kept) - 1) < TOL[precision]
        for op in gates(n):
            st.execute([op])
        ref.set_state_vector(kept)
        ref.execute(gates(n))
        assert np.max(np.abs(st.get_state_vector() - ref.get_state_vector())) < TOL[precision]

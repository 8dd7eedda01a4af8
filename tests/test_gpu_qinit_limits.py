"""QINIT to a size that cannot be had: an error, and a handle that goes on
working (a state of no memory would be read and written by the next call)."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C


@pytest.mark.gpu
@pytest.mark.parametrize("size", [41, 60, 64, 100, (1 << 31) + 5])
def test_beyond_the_engine_limit(size):
    with qb.QuantumState(5) as st:
        st.execute([C.Op(C.H, [0]), C.Op(C.CNOT, [0, 4])])
        before = st.get_state_vector()
        with pytest.raises(qb.QoaError):
            st.execute([C.Op(C.QINIT, [size])])
        assert st.get_num_qubits() == 5
        assert np.allclose(st.get_state_vector(), before, rtol=0, atol=1e-15)
        with pytest.raises(qb.QoaError):  # what came before it in the list is done
            st.execute([C.Op(C.RESETALL), C.Op(C.X, [1]), C.Op(C.RESETALL), C.Op(C.QINIT, [size])])
        assert st.get_probabilities()[0] == 1.0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 14])
def test_more_than_the_device_has(n):
    with qb.QuantumState(n) as st:
        st.execute([C.Op(C.X, [2])])
        with pytest.raises(qb.QoaError):
            st.execute([C.Op(C.X, [0]), C.Op(C.QINIT, [38])])  # 4 TiB
        assert st.get_num_qubits() == n
        assert st.get_probabilities()[0] == 1.0
        st.execute([C.Op(C.H, [0]), C.Op(C.CNOT, [0, n - 1])])
        p = st.get_probabilities()
        assert abs(p[0] - 0.5) < 1e-15 and abs(p[1 | 1 << (n - 1)] - 0.5) < 1e-15
        assert st.sample(50, np.full(50 * n, 0.75))[0] == 1 | 1 << (n - 1)

"""The order of a pass's gates: lists whose gates mostly commute in part
(diagonal runs, shared controls, SWAPs that relabel tile bits in between), in
both precisions, interpreted and generated, against the oracle."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from oracle import pyoracle as po


def entangled(n, count, seed):
    rng = C.SplitMix64(seed)
    ops = [C.Op(C.H, [q]) for q in range(n)]
    for _ in range(count):
        a, b = rng.below(n), rng.below(n - 1)
        b += b >= a
        k = rng.below(8)
        if k == 0:
            ops.append(C.Op(C.SWAP, [a, b]))
        elif k in (1, 2):
            ops.append(C.Op(C.CNOT, [a, b]))
        elif k == 3:
            ops.append(C.Op(C.CZ, [a, b]))
        elif k == 4:
            ops.append(C.Op(C.CPHASE, [a, b], rng.uniform() * 6))
        elif k == 5:
            ops.append(C.Op(C.RZ, [a], rng.uniform() * 6))
        else:
            ops.append(C.Op(C.RX if k == 6 else C.RY, [a], rng.uniform() * 6))
    return ops


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 2e-5)])
@pytest.mark.parametrize("n,count,search", [(13, 300, False), (14, 90, True), (17, 400, True), (18, 250, False)])
def test_reordered_passes(n, count, search, precision, tol):
    ops = entangled(n, count, 1000 + n)
    po.set_fast(True)
    o = po.OracleState(n, 0)
    o.apply(C.ops_to_array(ops))
    ref = o.state()
    o.close()
    got = []
    for jit in (qb.QOA_JIT_OFF, qb.QOA_JIT_SYNC):
        with qb.QuantumState(n, precision=precision, slot_search=search) as st:
            st.set_jit(jit, min_qubits=11)
            st.execute(ops)
            got.append(st.get_state_vector())
    assert np.array_equal(got[0], got[1])
    assert np.linalg.norm(got[0] - ref) / np.linalg.norm(ref) < tol

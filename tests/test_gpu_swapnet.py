"""Swap networks as one permutation pass: partners among, above and outside a
tile's lowest qubits, few and many outer qubits, both precisions, against the
permuted amplitudes."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-14), ("f32", 1e-6)])
@pytest.mark.parametrize("kind", ["reverse", "low", "high", "random"])
@pytest.mark.parametrize("n", [13, 14, 17, 19])
def test_networks(n, kind, precision, tol):
    if kind == "reverse":
        pairs = [(q, n - 1 - q) for q in range(n // 2)]
    elif kind == "low":
        pairs = [(0, 1), (2, 5), (3, 4)]
    elif kind == "high":
        pairs = [(6, n - 1), (7, n - 2), (8, n - 3)]
    else:
        p = [int(x) for x in np.random.default_rng(n).permutation(n)]
        pairs = [(p[2 * k], p[2 * k + 1]) for k in range(n // 2 - 1)]
    with qb.QuantumState(n, precision=precision) as st:
        st.set_random_state(n)
        before = st.get_state_vector()
        st.execute([C.Op(C.SWAP, list(x)) for x in pairs])
        after = st.get_state_vector()
    idx = np.arange(1 << n)
    src = idx.copy()
    for a, b in pairs:
        bits = ((src >> a) ^ (src >> b)) & 1
        src ^= (bits << a) | (bits << b)
    assert np.linalg.norm(after - before[src]) < tol

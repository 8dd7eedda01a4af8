"""Expectation sweeps against numpy: states smaller than, equal to and larger
than a sweep's 4096-amplitude tile, and mask counts at the edges of the
kernel's variants (16, 64, 256 per sweep), for handles and batch circuits.
FP64 sums of 2^n terms of total weight 1 agree to 1e-13."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C

TOL = 1e-13


def reference(p, masks):
    idx = np.arange(p.size, dtype=np.uint64)
    return np.array([p @ (1.0 - 2.0 * (np.bitwise_count(idx & np.uint64(m)) & 1)) for m in masks])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n,k", [(1, 1), (4, 17), (11, 16), (12, 64), (13, 65), (14, 257), (17, 300)])
def test_expect_z_masks(n, k, precision):
    rng = np.random.default_rng(n * 1000 + k)
    masks = [0, (1 << n) - 1] + [int(x) for x in rng.integers(0, 1 << n, max(0, k - 2))]
    masks = masks[:k]
    with qb.QuantumState(n, precision=precision) as st:
        st.execute(C.ops_to_array(C.variational(n, 3, C.SplitMix64(n))))
        st.execute([C.Op(C.H, [0])])
        p = st.get_probabilities()
        got = st.expect_z(masks)
        again = st.expect_z(masks)
    assert np.max(np.abs(got - reference(p, masks))) < TOL
    assert np.array_equal(got, again)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(13, 1), (13, 15), (14, 16), (15, 63), (13, 64), (16, 255)])
def test_batch_masks_match_handles(n, k):
    rng = np.random.default_rng(k)
    ops = C.ops_to_array(C.variational(n, 2, C.SplitMix64(k)))
    masks = [int(x) for x in rng.integers(0, 1 << n, k)]
    with qb.Batch() as b, qb.QuantumState(n) as st:
        b.add(n, ops, masks)
        b.run()
        st.execute(ops)
        assert np.max(np.abs(b.results() - st.expect_z(masks))) < TOL

"""Shots and expectation values on states above 22 qubits, against numpy: the
shot tree's steps of five (23 qubits) and six bits (26), and sweeps of more
tiles than CTAs, where a CTA adds up several tiles in the same shared memory,
in each of the sweep's variants."""
import numpy as np
import pytest

import qoa_b200 as qb
from tests.test_gpu_expz_sweep import TOL, reference
from tests.test_gpu_sample_tree import walk


@pytest.mark.gpu
@pytest.mark.parametrize("n,precision,mode", [(23, "f64", 0), (23, "f64", 1), (23, "f32", 0), (23, "f32", 1),
                                              (26, "f64", 0), (26, "f32", 1)])
def test_shots_walk_the_marginal_tree(n, precision, mode):
    shots = 203
    u = np.random.default_rng(n + mode).random(shots * n if mode == 0 else shots)
    with qb.QuantumState(n, precision=precision) as st:
        st.set_random_state(n)
        p = st.get_probabilities()
        got = st.sample(shots, u, mode=mode)
    assert np.array_equal(got, walk(p, n, u, mode))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n,k", [(22, 16), (22, 17), (23, 65)])
def test_expect_z_over_many_tiles(n, k, precision):
    masks = [0, (1 << n) - 1] + [int(x) for x in np.random.default_rng(k).integers(0, 1 << n, k - 2)]
    with qb.QuantumState(n, precision=precision) as st:
        st.set_random_state(n + k)
        p = st.get_probabilities()
        got = st.expect_z(masks)
        again = st.expect_z(masks)
    assert np.max(np.abs(got - reference(p, masks))) < TOL
    assert np.array_equal(got, again)

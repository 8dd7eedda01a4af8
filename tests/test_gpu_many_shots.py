"""Many shots at once: the tree of all levels with a thread per shot gives the
shots that a few at a time get from the stored levels, bit for bit, at the
edges of its rule and of its folds (8 levels at the root, 4, 5 and 6 bits a
fold), and costs no more a shot on 20 qubits than on 2."""
import time

import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C

MIB = 1 << 20


def many(n):
    return max(1 << 14, (1 << n) >> 8)


def in_pieces(st, u, per, shots, mode, upto):
    """the first `upto` shots, below the rule's line at a time"""
    step = min(many(st.n) - 1, 1000)
    return np.concatenate([st.sample(min(step, upto - k), u[k * per:min(k + step, upto) * per], mode=mode)
                           for k in range(0, upto, step)])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 12, 16, 20, 23])
def test_same_shots_as_a_few_at_a_time(n, mode, precision):
    shots, per = many(n), n if mode == 0 else 1
    u = np.random.default_rng(n).random(shots * per)
    with qb.QuantumState(n, precision=precision) as st:
        st.set_random_state(40 + n)
        got = st.sample(shots, u, mode=mode)
        assert np.array_equal(got[:4000], in_pieces(st, u, per, shots, mode, 4000))
        assert got.max() < (1 << n)


@pytest.mark.gpu
def test_six_bit_folds_and_a_tree_that_does_not_fit():
    import torch

    n, shots = 26, 1 << 18
    u = np.random.default_rng(2).random(shots)
    with qb.QuantumState(n, precision="f32") as st:
        st.set_random_state(9)
        want = in_pieces(st, u, 1, shots, 1, 3000)
        got = st.sample(shots, u, mode=1)
        assert np.array_equal(got[:3000], want)
        torch.cuda.empty_cache()
        block = torch.empty(torch.cuda.mem_get_info()[0] - 300 * MIB, dtype=torch.uint8, device="cuda")
        try:
            again = st.sample(shots, u, mode=1)  # 512 MiB of levels do not fit: the stored ones
        finally:
            del block
            torch.cuda.empty_cache()
        assert np.array_equal(again, got)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_sparse_and_reset_states(precision):
    n, shots = 11, 1 << 14
    u0, u1 = np.random.default_rng(4).random(shots * n), np.random.default_rng(5).random(shots)
    with qb.QuantumState(n, precision=precision) as st:
        for ops in ([], [C.Op(C.H, [0]), C.Op(C.CNOT, [0, 10])], [C.Op(C.X, [3]), C.Op(C.H, [9])]):
            st.execute([C.Op(C.RESETALL)] + ops)
            assert np.array_equal(st.sample(shots, u0, mode=0)[:2000], in_pieces(st, u0, n, shots, 0, 2000))
            assert np.array_equal(st.sample(shots, u1, mode=1)[:2000], in_pieces(st, u1, 1, shots, 1, 2000))


@pytest.mark.gpu
def test_a_shot_costs_the_same_on_more_qubits():
    shots, t = 1 << 20, {}
    u = np.random.default_rng(6).random(shots)
    for n in (2, 20):
        with qb.QuantumState(n) as st:
            st.set_random_state(1)
            best = 1e9
            for _ in range(12):
                t0 = time.perf_counter()
                st.sample(shots, u, mode=1)
                best = min(best, time.perf_counter() - t0)
            t[n] = best
    assert t[20] < 2 * t[2]  # both mostly copy 16 MB between host and device

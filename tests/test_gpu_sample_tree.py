"""Shots against a walk of the marginal tree in numpy: sizes at the edges of
the stored levels (8-bit root, steps of up to 6 bits), both draw orders and
both precisions. The walk sums the engine's own probabilities with the top
index bit paired first, so outcomes agree exactly except where a uniform
falls within rounding of a boundary (of order 1e-13 a shot)."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C


def walk(p, n, u, mode):
    levels = [p]
    while len(levels[-1]) > 1:
        x = levels[-1]
        levels.append(x[:len(x) // 2] + x[len(x) // 2:])
    h = levels[::-1]  # h[k][prefix]
    out = []
    for us in u.reshape(-1, n) if mode == 0 else u:
        pre, dead = 0, False
        t = 0.0 if mode == 0 else us * h[0][0]
        for q in range(n):
            left = h[q + 1][pre]
            if mode == 1:
                if t >= left:
                    t -= left
                    pre |= 1 << q
                continue
            if dead:
                continue
            tot = h[q][pre]
            p0, p1 = left / tot, h[q + 1][pre | 1 << q] / tot
            b = 0 if us[q] < p0 else 1
            pre |= b << q
            dead = not (p1 if b else p0) > 1e-12
        out.append(pre)
    return np.array(out, dtype=np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 8, 9, 14, 15, 20, 21])
def test_shots_walk_the_marginal_tree(n, mode, precision):
    shots = 301
    rng = np.random.default_rng(100 * n + mode)
    u = rng.random(shots * n if mode == 0 else shots)
    with qb.QuantumState(n, precision=precision) as st:
        st.execute(C.ops_to_array(C.random_layered(n, 4, 50 + n, initial_h=True) if n > 1 else [C.Op(C.RY, [0], 0.9)]))
        p = st.get_probabilities()
        got = st.sample(shots, u, mode=mode)
    assert np.array_equal(got, walk(p, n, u, mode))

"""Batches in which some pass structures are shared widely enough for a
generated kernel and others are not: rounds that mix generated and
interpreted launches equal the interpreter bit for bit, and the kernels
requested are the shared ones only."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shared,lone", [(9, 0), (8, 1), (12, 7), (3, 5)])
def test_mixed_rounds(precision, shared, lone):
    rng = C.SplitMix64(7)
    circs = [(14, C.variational(14, 3, rng)) for _ in range(shared)]
    circs += [(13 + k % 3, C.random_layered(13 + k % 3, 2 + k, 40 + k, initial_h=True)) for k in range(lone)]
    order = np.random.default_rng(shared * 10 + lone).permutation(len(circs))

    def run(jit):
        with qb.Batch(precision) as b:
            b.set_tuning(jit=jit)
            for i in order:
                n, ops = circs[i]
                b.add(n, ops, [1, (1 << n) - 1, 6])
            b.run()
            first = b.results()
            b.run()
            qb.jit_wait()
            b.run()
            return first, b.results(), b.jit_info()

    first, last, info = run(qb.QOA_JIT_ASYNC)
    _, want, _ = run(qb.QOA_JIT_OFF)
    assert np.array_equal(first, want) and np.array_equal(last, want)
    assert info["graph_uses_generated"] == (shared >= 8)
    assert info["ready"] == info["structures"] and (info["structures"] > 0) == (shared >= 8)

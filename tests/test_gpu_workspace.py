"""Scratch that handles keep between calls: an allocation that finds the
device full takes it back, and all handles together keep at most 1 GiB."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C

N = 24                     # complex128: a state of 256 MiB, probabilities in 128 MiB of scratch
MIB = 1 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["create", "qinit", "batch"])
def test_full_device_takes_idle_scratch_back(how):
    import torch

    torch.cuda.empty_cache()
    small = qb.QuantumState(4)
    batch = qb.Batch("f64")
    a = qb.QuantumState(N)
    a.set_random_state(5)
    p = a.get_probabilities()  # keeps 128 MiB
    # 192 MiB stay free: too few for another state, enough with the scratch
    block = torch.empty(torch.cuda.mem_get_info()[0] - 192 * MIB, dtype=torch.uint8, device="cuda")
    try:
        if how == "create":
            with qb.QuantumState(N) as b:
                b.apply_h(0)
                assert b.get_num_qubits() == N
        elif how == "qinit":
            small.execute([C.Op(C.QINIT, [N]), C.Op(C.H, [0])])
            assert abs(small.expect_z([2])[0] - 1.0) < 1e-12
        else:
            batch.add(N, [C.Op(C.X, [3])], [8])
            batch.run()
            assert abs(batch.results()[0] + 1.0) < 1e-12
    finally:
        batch.close()
        small.close()
        del block
        torch.cuda.empty_cache()
    assert np.array_equal(a.get_probabilities(), p)
    a.close()


@pytest.mark.gpu
def test_handles_keep_a_bounded_total():
    import torch

    sts = [qb.QuantumState(N) for _ in range(12)]
    for s in sts:
        s.sync()
    before = torch.cuda.mem_get_info()[0]
    first = sts[0].get_probabilities()
    for s in sts[1:]:
        assert np.array_equal(s.get_probabilities(), first)  # |0..0>
    kept = before - torch.cuda.mem_get_info()[0]
    for s in sts:
        s.close()
    assert kept <= 1024 * MIB + 64 * MIB  # (64: what the kernels' first launch maps)

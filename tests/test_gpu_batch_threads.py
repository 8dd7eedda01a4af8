"""Every accepted block size of the batch's shared-memory kernel launches: the
largest one too, in both precisions, at the largest state the kernel takes."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from tests.test_gpu_batch import F32_TOL, F64_TOL, expected


@pytest.mark.gpu
@pytest.mark.parametrize("precision,nmax,tol", [("f64", 12, F64_TOL), ("f32", 13, F32_TOL)])
@pytest.mark.parametrize("threads", [32, 512, 640, 1024])
def test_every_block_size_runs(precision, nmax, tol, threads):
    circs = C.variational_batch(count=6, nmin=3, nmax=nmax, lmin=1, lmax=2, nmasks=3, seed=29)
    circs[0] = dict(circs[0], **C.variational_batch(count=1, nmin=nmax, nmax=nmax, lmin=2, lmax=2, nmasks=3, seed=30)[0])
    with qb.Batch(precision) as b:
        b.set_tuning(small_threads=threads, small_ctas_per_sm=1)
        for c in circs:
            b.add(c["n"], c["ops"], c["masks"])
        b.run()
        got = b.results()
    assert np.max(np.abs(got - expected(circs))) < tol

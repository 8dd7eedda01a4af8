"""Compiling the generated complex64 passes of a handle costs no more than
their batch form, which stages its coefficients instead of reading them from
the kernel's parameter (no GPU)."""
import time

import qoa_b200 as qb
from qoa_b200 import circuits as C


def ansatz(n, layers):
    ops = []
    for k in range(layers):
        for q in range(n):
            ops += [C.Op(C.RY, [q], 0.1 + 0.01 * (q + k)), C.Op(C.RZ, [q], 0.2 + 0.02 * q)]
        ops += [C.Op(C.CZ, [q, q + 1]) for q in range(n - 1)]
    return ops


def cpu_seconds(arena):
    t0 = time.process_time()  # of all the compiler's threads
    _, npasses = qb.jit_translate(18, ansatz(18, 8), compile=True, precision="f32", arena=arena)
    assert npasses >= 4
    return time.process_time() - t0


def test_parameter_coefficients_compile_as_fast_as_staged_ones():
    qb.jit_translate(13, ansatz(13, 1), compile=True, precision="f32")  # the compiler is loaded
    staged = min(cpu_seconds(True) for _ in range(2))
    direct = min(cpu_seconds(False) for _ in range(2))
    assert direct < 1.05 * staged, (direct, staged)

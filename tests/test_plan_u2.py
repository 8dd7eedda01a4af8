"""Plans and generated text of lists with 4x4 gates and controlled SWAPs (no
GPU): the pass scheduler reports what a complex128 handle runs, both kinds
inside tile passes, and the kernels of such passes compile."""
import numpy as np
import pytest

import qoa_b200 as qb
from qoa_b200 import circuits as C
from tests.plan_emulator import replay
from tests.test_plan import mixed_circuit, oracle_state, rel_l2

N = 13


def circuit():
    u, _ = np.linalg.qr(np.arange(16).reshape(4, 4) + 1j * np.eye(4) + 3 * np.eye(4))
    return ([C.Op(C.H, [q]) for q in range(N)] + [C.Op(C.U2, [3, 9], 0.0, u.reshape(-1))]
            + [C.Op(C.RX, [9], 0.7), C.Op(C.CSWAP, [1, 4, 10])])


def test_plan_has_them_inside_passes():
    ops = circuit()
    plan = qb.plan(N, ops)
    assert len(plan["pass_of"]) == N + 1 + 1 + 3  # the controlled SWAP is three gates
    # 13 qubits, 11 of them in a tile: H on every qubit takes two passes, and nothing breaks them
    assert plan["npasses"] == 2
    assert rel_l2(replay(N, plan), oracle_state(N, ops, 0)) < 1e-12


def test_per_gate_plan_keeps_the_controlled_swap():
    plan = qb.plan(N, circuit(), qb.QOA_FLAG_PER_GATE)
    assert plan["npasses"] == len(plan["pass_of"]) == N + 3


@pytest.mark.parametrize("arena", [False, True])
def test_translate_compiles_the_4x4_gate(arena):
    src, npasses = qb.jit_translate(N, circuit(), compile=True, arena=arena)
    assert npasses == 2
    assert "g2r<" in src


def test_complex64_passes_leave_the_4x4_gate_out():
    # complex64 handles run it on a kernel of its own; the controlled SWAP is in the passes
    src, npasses = qb.jit_translate(N, circuit(), compile=True, precision="f32")
    assert "g2r<" not in src
    assert npasses >= 2


@pytest.mark.parametrize("n,count,seed", [(12, 200, 21), (14, 150, 22)])
def test_passes_of_both_reports_agree(n, count, seed):
    ops = [o for o in mixed_circuit(n, count, seed) if o.opcode != C.SWAP]
    _, npasses = qb.jit_translate(n, ops, compile=True)
    assert qb.plan(n, ops)["npasses"] == npasses  # every step is a tile pass

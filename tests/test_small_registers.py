"""Registers below the pass kernel's size: many gates per kernel, at every
size, past the gates and the entries one kernel holds, against the oracle
and the gate-by-gate mode."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8])
def test_small_registers(gpu_lib, oracle_lib, n, precision):
    """complex128 within 1e-12; complex64 within 120 gates of FP32
    roundings, 120 * 6e-8 < 1e-5. Random gates of up to 4 targets (16
    entries each) with controls, 33 one-qubit gates and a measured chain."""
    circ = C.random_circuit(n, 90, seed=n, max_controls=min(3, n - 1), measure_prob=0.1)
    circ += [("u3", (0.1 * i, 0.2, 0.3), (i % n,), (), ()) for i in range(33)]
    states, bits = [], []
    for lib, mode in ((gpu_lib, qcs_b200.FUSION_GREEDY), (gpu_lib, qcs_b200.FUSION_PLAIN), (oracle_lib, None)):
        kw = {} if mode is None else {"precision": precision, "fusion": mode}
        with qcs_b200.Simulator(lib, n, n, seed=3, **kw) as sim:
            sim.run(circ)
            states.append(sim.statevector())
            bits.append(sim.clbits_string())
    tol = 1e-12 if precision == 128 else 1e-5
    assert bits[0] == bits[2] or precision == 64
    assert bits[0] == bits[1]
    assert np.max(np.abs(states[0] - states[1])) <= tol
    if bits[0] == bits[2]:
        assert np.max(np.abs(states[0] - states[2])) <= tol


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("n", [1, 2, 5, 8])
def test_gates_in_one_kernel_are_the_plain_kernels(gpu_lib, oracle_lib, n, precision):
    """Without measurements: bit for bit the gate-by-gate mode's state, and
    the oracle's within 120 roundings in either precision."""
    circ = C.random_circuit(n, 90, seed=40 + n, max_controls=min(3, n - 1))
    circ += [("u3", (0.1 * i, 0.2, 0.3), (i % n,), (), ()) for i in range(33)]
    states = []
    for lib, mode in ((gpu_lib, qcs_b200.FUSION_GREEDY), (gpu_lib, qcs_b200.FUSION_PLAIN), (oracle_lib, None)):
        kw = {} if mode is None else {"precision": precision, "fusion": mode}
        with qcs_b200.Simulator(lib, n, **kw) as sim:
            # (an uncontrolled swap only relabels qubits in the fused modes)
            sim.run([op for op in circ if op[0] != "swap" or op[3] or op[4]])
            states.append(sim.statevector())
    assert np.array_equal(states[0], states[1])
    assert np.max(np.abs(states[0] - states[2])) <= (1e-12 if precision == 128 else 1e-5)

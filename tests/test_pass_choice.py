"""How automatic mode runs the passes of phase-heavy circuits (plans of a
complex128 register, made on the host without a GPU)."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C


def trotter(n, steps):
    """H on every qubit, then steps of RZZ on neighbours and next neighbours and an RX layer."""
    circ = [("h", (), (q,), (), ()) for q in range(n)]
    for s in range(steps):
        circ += [("rzz", (0.3 + 0.1 * s,), (q, q + 1), (), ()) for q in range(n - 1)]
        circ += [("rzz", (0.2 + 0.1 * s,), (q, q + 2), (), ()) for q in range(n - 2)]
        circ += [("rx", (0.7 - 0.1 * s,), (q,), (), ()) for q in range(n)]
    return circ


def qaoa(n, layers, seed):
    """H on every qubit, then layers of RZZ on the edges of a random 3-regular graph and an RX layer."""
    rng = np.random.default_rng(seed)
    while True:
        edges = rng.permutation(np.repeat(np.arange(n), 3)).reshape(-1, 2)
        if (edges[:, 0] != edges[:, 1]).all():
            break
    circ = [("h", (), (q,), (), ()) for q in range(n)]
    for s in range(layers):
        circ += [("rzz", (0.4 + 0.1 * s,), (int(a), int(b)), (), ()) for a, b in edges]
        circ += [("rx", (0.9 - 0.1 * s,), (q,), (), ()) for q in range(n)]
    return circ


@pytest.mark.parametrize("n", [20, 22, 24, 28])
def test_phases_with_other_gates_are_priced(gpu_lib, n):
    """RZZ layers with an RX layer between them: mostly phases, and two to
    four times as fast as 8 x 8 tensor stages (one pass of the last, short
    layer may stay behind)."""
    s = qcs_b200.plan_summary(gpu_lib, n, trotter(n, 6))
    assert s["tensor_passes"] >= s["passes"] - 1
    s = qcs_b200.plan_summary(gpu_lib, n, qaoa(n, 4, seed=n))
    assert s["tensor_passes"] >= s["passes"] - 1


@pytest.mark.parametrize("n", [20, 24, 28])
def test_hadamards_with_phases_stay_butterflies(gpu_lib, n):
    s = qcs_b200.plan_summary(gpu_lib, n, C.qft(n, seed=1)[0])
    assert s["tensor_passes"] == 0


@pytest.mark.parametrize("n", [16, 20, 24, 28])
def test_qft_passes_are_butterflies(gpu_lib, n):
    s = qcs_b200.plan_summary(gpu_lib, n, C.qft(n, seed=1)[0])
    assert s["kinds"]["butterfly_pass"] == s["passes"]
    # a U3 on every qubit in front: passes that hold one are none
    circ = [("u3", (0.1, 0.2, 0.3), (q,), (), ()) for q in range(n)] + C.qft(n, seed=1)[0]
    s = qcs_b200.plan_summary(gpu_lib, n, circ)
    assert 0 < s["kinds"]["butterfly_pass"] + s["tensor_passes"] <= s["passes"]
    assert s["kinds"]["butterfly_pass"] < s["passes"]


@pytest.mark.parametrize("n", [10, 11, 15, 19])
def test_small_registers_take_8x8_stages(gpu_lib, n):
    """From 11 qubits (one chunk of a tensor pass) and 24 gates a pass on."""
    s = qcs_b200.plan_summary(gpu_lib, n, C.layered_u3_cz_cx_toffoli(n, 8, seed=1))
    assert s["tensor_passes"] == s["tensor8_passes"]
    assert (s["tensor8_passes"] >= 0.5 * s["passes"]) == (n >= 11)
    short = [("u3", (0.1, 0.2, 0.3), (q % n,), (), ()) for q in range(23)]
    assert qcs_b200.plan_summary(gpu_lib, n, short)["tensor_passes"] == 0

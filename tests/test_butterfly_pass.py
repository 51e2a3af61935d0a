"""Butterfly passes: flushes of Hadamard gates and diagonals (QFT, layers of H
with phases between them), on registers of one chunk and up, with stages that
do and do not hold the low qubits, an even and an odd number of H, basis
inputs whose X gates end in an H, against the CPU oracle."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C

pytestmark = pytest.mark.gpu


def hadamard_phases(n, seed):
    """H on a random half of the qubits, phases of every sort, H on others, phases again."""
    rng = np.random.default_rng(seed)
    circ = [("x", (), (int(q),), (), ()) for q in rng.permutation(n)[: n // 3]]
    for _ in range(2):
        circ += [("h", (), (int(q),), (), ()) for q in sorted(rng.permutation(n)[: n // 2 + 1], reverse=True)]
        for _ in range(2 * n):
            a, b = (int(q) for q in rng.choice(n, 2, replace=False))
            circ.append([("p", (float(rng.uniform(-3, 3)),), (a,), (), (b,)), ("rz", (float(rng.uniform(-3, 3)),), (a,), (), ()),
                         ("rzz", (float(rng.uniform(-3, 3)),), (a, b), (), ()), ("s", (), (a,), (), (b,)),
                         ("t", (), (a,), (b,), ())][int(rng.integers(0, 5))])
    return circ


CASES = {
    "qft": lambda n: C.qft(n, seed=n)[0],
    "inverse_order": lambda n: [("h", (), (q,), (), ()) for q in range(n)] + C.qft(n, seed=n, swaps=False)[0],
    "phases": lambda n: hadamard_phases(n, n),
}


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("n", [11, 12, 14, 17, 19, 21])
def test_hadamard_and_phase_circuits(gpu_lib, oracle_lib, n, case, precision):
    """complex128 within 1e-12 (at most n H per flush and a product of
    phases each); complex64 within 1e-5 of the largest amplitude."""
    circ = CASES[case](n)
    rng = np.random.default_rng(n)
    start = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    start /= np.linalg.norm(start)
    states = []
    for lib in (gpu_lib, oracle_lib):
        kw = {"precision": precision, "fusion": qcs_b200.FUSION_GREEDY} if lib is gpu_lib else {}
        with qcs_b200.Simulator(lib, n, **kw) as sim:
            sim.set_statevector(start)
            sim.run(circ)
            states.append(sim.statevector())
    got, ref = states
    tol = 1e-12 if precision == 128 else 1e-5 * np.max(np.abs(ref))
    assert np.max(np.abs(got - ref)) <= tol


def test_qft_of_a_basis_state(gpu_lib):
    n = 16
    circ, x = C.qft(n, seed=4)
    with qcs_b200.Simulator(gpu_lib, n) as sim:
        sim.run(circ)
        got = sim.statevector()
    k = np.arange(1 << n)
    want = np.exp(2j * np.pi * ((x * k) % (1 << n)) / (1 << n)) / np.sqrt(1 << n)
    assert np.max(np.abs(got - want)) <= 1e-14


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("n", [22, 23])
def test_qft_with_several_chunks_per_block(gpu_lib, n, precision):
    """2048 and 4096 chunks on at most 1184 (complex128: 592) blocks, every
    pass a butterfly; the transform of a basis state in closed form."""
    circ, x = C.qft(n, seed=n)
    s = qcs_b200.plan_summary(gpu_lib, n, circ)
    assert s["kinds"]["butterfly_pass"] == s["passes"]
    with qcs_b200.Simulator(gpu_lib, n, precision=precision, fusion=qcs_b200.FUSION_GREEDY) as sim:
        sim.set_tensor_passes(qcs_b200.TENSOR_NEVER)
        sim.run(circ)
        got = sim.statevector()
    k = np.arange(1 << n)
    want = np.exp(2j * np.pi * ((x * k) % (1 << n)) / (1 << n)) / np.sqrt(1 << n)
    # relative to the amplitudes, all of one size: n H and n / 2 phases per
    # amplitude in each precision
    assert np.max(np.abs(got - want)) * np.sqrt(1 << n) <= (1e-13 if precision == 128 else 1e-4)


@pytest.mark.parametrize("precision", [128, 64])
def test_phases_with_several_chunks_per_block(gpu_lib, oracle_lib, precision):
    """Stages that hold the low qubits and ones that leave them alone."""
    n = 22
    circ = hadamard_phases(n, 5)
    states = []
    for lib in (gpu_lib, oracle_lib):
        kw = {"precision": precision, "fusion": qcs_b200.FUSION_GREEDY} if lib is gpu_lib else {}
        with qcs_b200.Simulator(lib, n, **kw) as sim:
            if lib is gpu_lib:
                sim.set_tensor_passes(qcs_b200.TENSOR_NEVER)
            sim.set_state("flat")
            sim.run(circ)
            states.append(sim.statevector())
    got, ref = states
    tol = 1e-12 if precision == 128 else 1e-5
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))

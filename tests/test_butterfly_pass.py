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

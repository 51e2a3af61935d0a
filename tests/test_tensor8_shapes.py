"""8 x 8 tensor passes at the sizes where the kernel changes shape (one chunk,
eight warps per chunk up to 256 chunks, four above), with the low qubits
dense, as conditions and untouched in the last stages, against the oracle."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C

pytestmark = pytest.mark.gpu


def circuit(n, low, seed):
    rng = np.random.default_rng(seed)
    circ = C.layered_u3_cz_cx_toffoli(n, 2, seed)
    qubits = list(range(3, n))
    for _ in range(6):
        a, b = (int(q) for q in rng.choice(qubits, 2, replace=False))
        if low == "dense":
            a = int(rng.integers(0, 3))
        circ.append(("u3", tuple(rng.uniform(-3, 3, 3)), (a,), (), (int(rng.integers(0, 3)),) if low == "condition" else ()))
        circ.append(("x", (), (b,), (), (int(rng.integers(0, 3)),) if low == "condition" else (a,)))
    return circ


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("low", ["dense", "condition", "untouched"])
@pytest.mark.parametrize("n", [11, 12, 13, 18, 19, 20])
def test_shapes(gpu_lib, oracle_lib, n, low, precision):
    """complex128 within 1e-12; complex64 within 1e-5 of the largest
    amplitude (split-TF32 products, 2^-21 each, over a few stages)."""
    circ = circuit(n, low, n)
    rng = np.random.default_rng(n)
    start = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    start /= np.linalg.norm(start)
    states = []
    for lib in (gpu_lib, oracle_lib):
        kw = {"precision": precision, "fusion": qcs_b200.FUSION_GREEDY} if lib is gpu_lib else {}
        with qcs_b200.Simulator(lib, n, **kw) as sim:
            if lib is gpu_lib:
                sim.set_tensor_passes(qcs_b200.TENSOR_ALWAYS_8X8)
            sim.set_statevector(start)
            sim.run(circ)
            states.append(sim.statevector())
            if lib is gpu_lib:
                assert sim.stats()["tensor8_passes"] > 0
    got, ref = states
    tol = 1e-12 if precision == 128 else 1e-5 * np.max(np.abs(ref))
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("low", ["dense", "condition", "untouched"])
@pytest.mark.parametrize("n", [21, 22])
def test_shapes_with_several_chunks_per_block(gpu_lib, oracle_lib, n, low, precision):
    """1024 and 2048 chunks on at most 888 (complex64: 1184) blocks: a block
    refills its buffer behind the last stage. Tolerances as above."""
    circ = circuit(n, low, n)
    states = []
    for lib in (gpu_lib, oracle_lib):
        kw = {"precision": precision, "fusion": qcs_b200.FUSION_GREEDY} if lib is gpu_lib else {}
        with qcs_b200.Simulator(lib, n, **kw) as sim:
            if lib is gpu_lib:
                sim.set_tensor_passes(qcs_b200.TENSOR_ALWAYS_8X8)
            sim.run(circ)
            states.append(sim.statevector())
            if lib is gpu_lib:
                assert sim.stats()["tensor8_passes"] > 0
    got, ref = states
    tol = 1e-12 if precision == 128 else 1e-5 * np.max(np.abs(ref))
    assert np.max(np.abs(got - ref)) <= tol

"""Reductions over the register: the <Z> sums at the sizes where the kernel
changes shape (below one tile, one tile, several tiles of one block each,
several tiles per block), against numpy sums of the state read back."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C


def random_state(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 10, 11, 12, 13, 14, 18, 20, 21])
def test_z_sums_match_numpy(gpu_lib, n, precision):
    """Both sides add 2^n non-negative terms in FP64 in blocked order: each
    sum is within ~100 roundings (tiles of a block, a thread's loads, the
    trees over threads and blocks) of exact, 1.2e-14 of the norm."""
    mapping = [int(q) for q in np.random.default_rng(n).permutation(n)]
    with qcs_b200.Simulator(gpu_lib, n, precision=precision, mapping=mapping) as sim:
        sim.set_statevector(random_state(n, 7 + n))
        p = np.abs(sim.statevector()) ** 2
        z, norm = sim.expectation_z()
        again, _ = sim.expectation_z()
    total = p.sum()
    want = [1.0 - 2.0 * p.reshape(-1, 2, 1 << q)[:, 1, :].sum() / total for q in range(n)]
    assert abs(norm / total - 1.0) <= 2.5e-14
    assert np.max(np.abs(z - np.array(want))) <= 5e-14
    assert np.array_equal(z, again)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("n", [20, 21, 22, 25, 26, 27])
def test_samples_do_not_depend_on_the_qubit_order(gpu_lib, n, precision):
    """Registers deeper than the sampler's tree (20 levels): the qubits below
    the leaves on lane bits of the leaf sums (reversed order: all of them up
    to 25 qubits), above them, and mixed. The outcomes are those of the
    identity order, which the sequential measurements check; a draw decides
    otherwise only within the rounding of a state computed in another order,
    1e-14 of a probability (complex64: 1e-5, one shot in 128 x n draws at
    most)."""
    circ = C.layered_u3_cz(n, 1, seed=n)
    orders = [list(range(n)), list(reversed(range(n))), [int(q) for q in np.random.default_rng(n).permutation(n)]]
    shots = []
    for mapping in orders:
        with qcs_b200.Simulator(gpu_lib, n, precision=precision, mapping=mapping, seed=17) as sim:
            sim.run(circ)
            shots.append(sim.sample(128))
    for other in shots[1:]:
        assert np.count_nonzero(shots[0] != other) <= (0 if precision == 128 else 1)

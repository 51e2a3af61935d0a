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

"""Rounding of complex128 passes, against 80-bit arithmetic on the CPU."""

import cmath
import math

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import circuits as C

pytestmark = pytest.mark.gpu

N = 13


def extended_state(circ, n):
    """The state in 80-bit arithmetic, the gates' entries in 64 bits as the library holds them (u3, x, z)."""
    psi = np.zeros(1 << n, dtype=np.clongdouble)
    psi[0] = 1
    index = np.arange(1 << n)
    for op, p, (t,), neg, pos in circ:
        if op == "u3":
            c, s = math.cos(0.5 * p[0]), math.sin(0.5 * p[0])
            m = [c, -cmath.exp(1j * p[2]) * s, cmath.exp(1j * p[1]) * s, cmath.exp(1j * (p[1] + p[2])) * c]
        else:
            m = {"x": [0, 1, 1, 0], "z": [1, 0, 0, -1]}[op]
        assert not neg
        mask = sum(1 << q for q in pos)
        i0 = index[(index & (mask | (1 << t))) == mask]
        a, b = psi[i0], psi[i0 | (1 << t)]
        m = [np.clongdouble(x) for x in m]
        psi[i0], psi[i0 | (1 << t)] = m[0] * a + m[1] * b, m[2] * a + m[3] * b
    return psi


CIRCUITS = {"layered": lambda seed: C.layered_u3_cz_cx_toffoli(N, 12, seed), "matching": lambda seed: C.u3_random_matching(N, 12, seed)}


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no 80-bit long double on this machine")
@pytest.mark.parametrize("circuit", sorted(CIRCUITS))
def test_tensor_stages_round_no_more_than_gates(gpu_lib, circuit):
    """The 2-norm of the error over six circuits: automatic mode (four
    products per complex one) at most that of the register path (gate by
    gate), measured 0.80-0.90 of it; forced 8 x 8 stages (three products) at
    most 1.3 of it, measured 1.10-1.22. An error is a sum over 2^13
    amplitudes, so that a ratio of these sums varies by 1-2%."""
    modes = {"auto": qcs_b200.TENSOR_AUTO, "gates": qcs_b200.TENSOR_NEVER, "three": qcs_b200.TENSOR_ALWAYS_8X8}
    err = dict.fromkeys(modes, 0.0)
    for seed in range(6):
        circ = CIRCUITS[circuit](seed)
        want = extended_state(circ, N)
        for name, mode in modes.items():
            with qcs_b200.Simulator(gpu_lib, N, fusion=qcs_b200.FUSION_GREEDY) as sim:
                sim.set_tensor_passes(mode)
                sim.run(circ)
                d = sim.statevector().astype(np.clongdouble) - want
                assert (sim.stats()["tensor8_passes"] > 0) == (name != "gates")
            err[name] += float(np.sum(d.real**2 + d.imag**2))
    assert math.sqrt(err["auto"] / err["gates"]) <= 1.0
    assert math.sqrt(err["three"] / err["gates"]) <= 1.3

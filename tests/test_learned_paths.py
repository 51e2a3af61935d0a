"""The learned planner's passes run as the executor's own choice unless the
model predicts another way to be faster: under a model that predicts the same
time for every pass, the learned plan takes the paths of the greedy one."""

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import FUSION_GREEDY, FUSION_LEARNED
from qcs_b200 import circuits as C
from test_pass_choice import trotter

pytestmark = pytest.mark.gpu

MIX = ["u3", "x", "h", "rz", "p", "ry", "swap", "rzz", "rxx", "sx", "s", "t", "y", "iswap"]
CASES = {
    # below the size at which greedy passes are priced: 8 x 8 stages at once
    "layered_17": (17, lambda: C.layered_u3_cz_cx_toffoli(17, 6, seed=3)),
    # conditions that need stages scheduled within a tensor pass's limits
    "random_20": (20, lambda: C.random_circuit(20, 240, seed=11, max_controls=2, gates=MIX)),
    "trotter_20": (20, lambda: trotter(20, 4)),
    # butterflies
    "qft_20": (20, lambda: C.qft(20, seed=2)[0]),
}


@pytest.fixture(scope="module")
def flat_model(gpu_lib):
    model = qcs_b200.CostModel(gpu_lib, seed=1)
    rng = np.random.default_rng(0)
    model.train(rng.uniform(1, 20, (64, qcs_b200.PASS_FEATURES)), np.zeros(64), epochs=1, batch=64)
    params, scaling = model.params()
    model.set_params(np.zeros_like(params), scaling)
    yield model
    model.close()


@pytest.mark.parametrize("case", sorted(CASES))
def test_learned_passes_take_the_executors_paths(gpu_lib, oracle_lib, flat_model, case):
    n, make = CASES[case]
    circ = make()
    stats = []
    for mode in (FUSION_GREEDY, FUSION_LEARNED):
        with qcs_b200.Simulator(gpu_lib, n, fusion=mode) as sim:
            sim.set_cost_model(flat_model if mode == FUSION_LEARNED else None)
            sim.run(circ)
            sim.synchronize()
            assert sim.planner_judge()["learned_plan"] == (mode == FUSION_LEARNED)
            stats.append(sim.stats())
            got = sim.statevector()
    with qcs_b200.Simulator(oracle_lib, n) as sim:
        sim.run(circ)
        assert np.max(np.abs(got - sim.statevector())) <= 1e-12
    greedy, learned = stats
    # (the cut moves by a few gates: as many passes or fewer, a pass of which
    # may fall to the other path)
    assert learned["fused_passes"] <= greedy["fused_passes"]
    assert learned["plain_gate_kernels"] == greedy["plain_gate_kernels"]
    for key in ("tensor_passes", "tensor8_passes"):
        assert abs(learned[key] / learned["fused_passes"] - greedy[key] / greedy["fused_passes"]) <= 0.2, key

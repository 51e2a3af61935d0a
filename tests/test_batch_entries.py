"""Gate entries of a batch, evaluated on the GPU: every parametrised gate of
at most two targets, with and without controls, before and after
set_parameters, against the CPU oracle."""

import time

import numpy as np
import pytest

import qcs_b200
from qcs_b200 import GATES

pytestmark = pytest.mark.gpu
N = 10


def circuit(rng, names):
    """h on every qubit, then each gate on random qubits, half of them controlled."""
    circ = [("h", (), (q,), (), ()) for q in range(N)]
    for i, name in enumerate(names):
        npar, nt = GATES[name]
        qs = [int(q) for q in rng.permutation(N)]
        ctrls, neg = ((qs[nt],), (qs[nt + 1],)) if i % 2 else ((), ())
        circ.append((name, tuple(rng.uniform(-7.0, 7.0, npar)), tuple(qs[:nt]), neg, ctrls))
    return circ


@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("name", [g for g, (npar, nt) in GATES.items() if npar > 0 and nt <= 2] + ["mixed"])
def test_batch_entries_match_oracle(gpu_lib, oracle_lib, name, precision):
    """Tolerance: an entry is a product of at most three sines and cosines,
    each within 2 ulp, over at most 20 gates: 1e-12 holds for complex128;
    complex64 entries are rounded once to FP32 (6e-8 each): 5e-6."""
    rng = np.random.default_rng(len(name))
    names = [name] * 6 if name != "mixed" else [g for g, (_, nt) in GATES.items() if nt <= 2]
    circ = circuit(rng, names)
    new = [(op, tuple(rng.uniform(-7.0, 7.0, len(p))), t, neg, pos) for op, p, t, neg, pos in circ]
    with qcs_b200.Batch(gpu_lib, precision) as batch:
        for _ in range(3):
            batch.add_circuit(N, circ)
        batch.run()
        first = batch.statevector(2)
        params = [x for op in circ for x in op[1]]
        batch.set_parameters(params * 2 + [x for op in new for x in op[1]])
        batch.run()
        states = [first, batch.statevector(0), batch.statevector(2)]
    tol = 1e-12 if precision == 128 else 5e-6
    for got, ops in zip(states, (circ, circ, new)):
        with qcs_b200.Simulator(oracle_lib, N) as sim:
            sim.run(ops)
            assert np.max(np.abs(got - sim.statevector())) <= tol


@pytest.mark.parametrize("tensor", [0, 2])
@pytest.mark.parametrize("precision", [128, 64])
def test_gates_that_differ_in_their_sub_indices_only(gpu_lib, oracle_lib, precision, tensor):
    """xx_plus_yy and xx_minus_yy have the same 2 x 2 block, on |01>, |10>
    and on |00>, |11>: circuits that differ in nothing else have plans of
    their own, while u3 and u, p and u1 share one. Tolerances as above."""
    n = 11
    pre = [("u3", (0.3 + q, 0.2, 0.9 - q), (q,), (), ()) for q in range(n)]
    swapped = {"xx_plus_yy": "xx_minus_yy", "u3": "u", "p": "u1"}
    a = pre + [("p", (0.4,), (3,), (), (1,)), ("xx_plus_yy", (0.7, 0.4), (2, 5), (), ()),
               ("xx_plus_yy", (1.1, -0.6), (9, 0), (4,), (7,))]
    b = [(swapped["xx_plus_yy"], *op[1:]) if op[0] == "xx_plus_yy" else op for op in a]
    c = [(swapped[op[0]], *op[1:]) if op[0] in ("u3", "p") else op for op in a]
    with qcs_b200.Batch(gpu_lib, precision) as batch:
        batch.set_tensor_passes(tensor)
        for circ in (a, b, c, b):
            batch.add_circuit(n, circ)
        batch.run()
        assert batch.info()["groups"] == 2
        states, z = [batch.statevector(i) for i in range(4)], batch.expectation_z()
    tol = 1e-12 if precision == 128 else 5e-6
    for i, circ in enumerate((a, b, c, b)):
        with qcs_b200.Simulator(oracle_lib, n) as sim:
            sim.run(circ)
            assert np.max(np.abs(states[i] - sim.statevector())) <= tol, i
            assert np.max(np.abs(z[i] - sim.expectation_z()[0])) <= tol, i


def test_first_run_grows_with_the_number_of_structures(gpu_lib):
    """A first run plans and tunes each structure by itself: four times as
    many different circuits take about four times as long (measured 4.0; with
    the entries of all structures uploaded for every candidate 9.4). The
    smaller batch is the better of two, so that a slow first call does not
    stand for it."""
    rng = np.random.default_rng(2)
    circuits = []
    for _ in range(1200):
        circ = []
        for k in range(200):
            a, b = (int(q) for q in rng.choice(N, 2, replace=False))
            circ.append(("ry", (0.1 * k,), (a,), (), ()) if k % 2 else ("x", (), (a,), (), (b,)))
        circuits.append(circ)

    def first_run(count):
        with qcs_b200.Batch(gpu_lib, 64) as batch:
            for circ in circuits[:count]:
                batch.add_circuit(N, circ)
            t0 = time.perf_counter()
            batch.run()
            t = time.perf_counter() - t0
            assert batch.info()["groups"] == count
        return t

    few = min(first_run(300), first_run(300))
    assert first_run(1200) <= 6.5 * few


def test_device_memory_of_a_batch_is_what_it_needs(gpu_lib):
    """4000 registers of 10 qubits with 300 U3 gates each: the amplitudes
    (64 MiB), at most four entries per gate (74 MiB), the parameters (28 MiB)
    and 24 MiB for the work lists, the tuner's spare and the allocator's
    granularity."""
    import torch

    count, gates = 4000, 300
    rng = np.random.default_rng(1)
    circ = [("u3", tuple(rng.uniform(-3, 3, 3)), (i % N,), (), ((i // N + i) % N,) if (i // N) % N else ()) for i in range(gates)]
    circ = [op for op in circ if op[2] != op[4]]
    with qcs_b200.Batch(gpu_lib, 128) as warm:   # what a first batch of the process loads
        warm.add_circuit(N, circ)
        warm.run()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with qcs_b200.Batch(gpu_lib, 128) as batch:
        for _ in range(count):
            batch.add_circuit(N, circ)
        batch.run()
        assert batch.info()["groups"] == 1
        used = before - torch.cuda.mem_get_info()[0]
    need = count * (16 * 2**N + 4 * 16 * len(circ) + 24 * len(circ))
    assert used <= need + (24 << 20)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no 80-bit long double on this machine")
def test_sines_and_cosines_of_entries(gpu_lib):
    """p(x) on |1> leaves e^{ix}: small and large angles, near multiples of
    pi / 2 and beyond the range of the own reduction, in ulp of 80-bit
    results. The own series is within 0.66 ulp, root mean square 0.29 (0.5
    and 0.289 would be rounding alone); CUDA's sincos, beyond 2^40, within 2."""
    rng = np.random.default_rng(3)
    own = [rng.uniform(-s, s, 400) for s in (1e-9, 0.5, 7.0, 1e3, 1e6, 1e11)]
    own += [np.arange(-200, 200) * (np.pi / 2), np.arange(-200, 200) * (np.pi / 4), np.array([0.0, 2.0**40, -(2.0**40)])]
    own = np.concatenate(own)
    far = rng.uniform(-1e15, 1e15, 400)
    x = np.concatenate([own, far])
    with qcs_b200.Batch(gpu_lib, 128) as batch:
        for v in x:
            batch.add_circuit(9, [("x", (), (0,), (), ()), ("p", (float(v),), (0,), (), ())])
        batch.run()
        got = np.array([batch.statevector(i)[1] for i in range(len(x))])
    want = np.cos(x.astype(np.longdouble)), np.sin(x.astype(np.longdouble))
    err = []
    for part, w in zip((got.real, got.imag), want):
        e = np.abs((part - w) / np.spacing(np.maximum(np.abs(w.astype(float)), 2.0**-60)))
        # where a part is close to nothing, its error counts against one ulp of 1
        err.append(np.where(np.abs(w) < 1e-9, np.abs(part - w) / 2.0**-53, e).astype(float))
    err = np.array(err)
    mine = err[:, : len(own)]
    assert mine.max() <= 0.70 and np.sqrt(np.mean(mine**2)) <= 0.30
    assert err[:, len(own):].max() <= 2.0

"""Which complex128 segments go to the fixed-point blocks (compiler._FIXED_SPREAD)
and which keep the tile sweeps, by how far their ops spread amplitudes."""
import numpy as np
import pytest

from qaravan_gb300 import workloads
from qaravan_gb300.circuits import Circuit
from qaravan_gb300.compiler import DenseStep, Op, SweepStep, compile_ops, spreading
from qaravan_gb300.gates import Gate
from qaravan_gb300.statevector import circuit_ops, gates_to_ops


def _plan(circ, n):
    ops = gates_to_ops(circuit_ops(circ), n)
    return compile_ops(ops, n, mode="fixed", width=5, max_sweep_k=4, itemsize=16, device_fusion=True, pack=True)


def _ansatz(n):
    return workloads.hea_circuit(n, 2, np.random.default_rng(1).uniform(0.5, 2.5, (2, n, 2)))


def test_spreading_of_gates():
    rng = np.random.default_rng(0)
    h = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
    small = np.array([[np.cos(0.05), -1j * np.sin(0.05)], [-1j * np.sin(0.05), np.cos(0.05)]])
    dft = np.exp(2j * np.pi * np.outer(np.arange(4), np.arange(4)) / 4) / 2
    assert spreading([h, np.diag([1, 1j]), small, np.eye(4)[[0, 1, 3, 2]], dft]) == [1.0, 0.0, 0.0, 0.0, 2.0]
    assert spreading([]) == []
    assert 1.5 < np.mean(spreading([workloads.haar_unitary(4, rng) for _ in range(50)])) <= 2.0


@pytest.mark.parametrize("n,make,kind", [
    (17, lambda n: workloads.brickwork_circuit(n, 2, 5), DenseStep),
    (18, lambda n: workloads.brickwork_circuit(n, 1, 5), DenseStep),
    (17, _ansatz, SweepStep), (18, _ansatz, SweepStep), (19, _ansatz, DenseStep),
    (17, lambda n: workloads.tfi_trotter_circuit(n, 0.05, 2), SweepStep),
    (20, lambda n: workloads.tfi_trotter_circuit(n, 0.05, 2), SweepStep),
    (20, lambda n: Circuit([Gate("p", [q, q + 1], np.diag(np.exp(1j * np.arange(4)))) for q in range(n - 1)], n=n),
     SweepStep)])
def test_routes(n, make, kind):
    plan = _plan(make(n), n)
    assert plan.steps and all(type(s) is kind for s in plan.steps)
    if kind is DenseStep:
        assert all(s.fixed and len(s.bits) == 5 for s in plan.steps)


def _pairs(n, layers):
    rng = np.random.default_rng(7)
    return Circuit([Gate("u", [q, q + 1], workloads.haar_unitary(4, rng)) for j in range(layers)
                    for q in range(j % 2, n - 1, 2)], n=n)


@pytest.mark.parametrize("n,layers,kind", [(17, 1, SweepStep), (17, 2, DenseStep), (17, 3, SweepStep), (18, 3, SweepStep),
                                           (18, 6, DenseStep), (19, 2, DenseStep), (20, 1, SweepStep),
                                           (20, 2, DenseStep), (25, 1, SweepStep), (25, 3, DenseStep)])
def test_too_few_ops_for_the_passes(n, layers, kind):
    steps = _plan(_pairs(n, layers), n).steps  # (a narrow tail is a sweep behind the passes)
    assert type(steps[0]) is kind and sum(type(s) is kind for s in steps) >= len(steps) - 1


@pytest.mark.parametrize("n,depth,seed", [(19, 2, 1), (20, 20, 1), (25, 8, 1), (25, 3, 2), (22, 5, 4)])
def test_narrow_tail_in_sweeps(n, depth, seed):
    """The last blocks of up to 3 bits run as a tile sweep behind the passes: every op once, in an order that
    keeps each bit's ops as they were."""
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(n, depth, seed)), n)
    plan = _plan(workloads.brickwork_circuit(n, depth, seed), n)
    kinds = "".join("D" if isinstance(s, DenseStep) else "S" for s in plan.steps)
    assert kinds.strip("D").strip("S") == "" and kinds.startswith("D")
    seen = []
    for s in plan.steps:
        for mat in [s.mat] if isinstance(s, DenseStep) else [m for _, m in s.ops]:
            seen += [i for i, _ in plan.matrices[mat].entries]
    assert sorted(seen) == list(range(len(ops)))
    for b in range(n):
        mine = [i for i in seen if b in ops[i].bits]
        assert mine == sorted(mine)
    assert all(len(bits) <= 3 for s in plan.steps if isinstance(s, SweepStep) for bits, _ in s.ops)


def test_one_gate():
    g = Circuit([Gate("u", [3, 4], workloads.haar_unitary(4, np.random.default_rng(0)))], n=20)
    assert [type(s) for s in _plan(g, 20).steps] == [SweepStep]


def test_segments_are_judged_by_themselves():
    """A reset cuts the circuit: Haar gates on one side, phases on the other."""
    n, rng = 17, np.random.default_rng(2)
    haar = workloads.brickwork_circuit(n, 2, 5).gate_list
    phases = [Gate("p", [q, q + 1], np.diag(np.exp(1j * rng.random(4)))) for q in range(n - 1)]
    a, b = gates_to_ops(haar, n), gates_to_ops(phases, n)
    plan = compile_ops(a + [None] + b, n, mode="fixed", width=5, max_sweep_k=4, itemsize=16, device_fusion=True)
    kinds = [type(s).__name__ for s in plan.steps]
    cut = kinds.index("NormalizeStep")
    assert set(kinds[:cut]) == {"DenseStep"} and set(kinds[cut + 1:]) == {"SweepStep"}


def test_the_same_structure_with_other_matrices():
    """The plan kept for a structure is not taken for matrices that spread less."""
    n = 17
    spread = workloads.brickwork_circuit(n, 1, 5)
    idle = Circuit([Gate("i", list(g.indices), np.eye(g.matrix.shape[0], dtype=complex)) for g in spread.gate_list], n=n)
    for _ in range(2):
        assert all(s.fixed for s in _plan(spread, n).steps)
        assert all(type(s) is SweepStep for s in _plan(idle, n).steps)


def test_other_ops_keep_the_sweeps():
    n, rng = 17, np.random.default_rng(3)
    gates = workloads.brickwork_circuit(n, 1, 5).gate_list
    wide = Gate("U", [int(q) for q in rng.permutation(n)[:6]], workloads.haar_unitary(64, rng))
    assert not any(getattr(s, "fixed", False) for s in _plan(Circuit(gates + [wide], n=n), n).steps)
    proj = gates_to_ops(gates, n) + [Op([3], np.diag([1.0, 0.0]).astype(complex))]
    plan = compile_ops(proj, n, mode="fixed", width=5, max_sweep_k=4, itemsize=16, device_fusion=True)
    assert all(type(s) is SweepStep for s in plan.steps)

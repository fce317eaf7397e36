"""Frontier fusion (``compiler.fuse_frontier``): its blocks, applied in order, are
the circuit, for every op exactly once, within the width; and ``compile_ops(pack=True)``
never has more dense passes than without."""
import numpy as np
import pytest

from qaravan_gb300 import workloads
from qaravan_gb300.compiler import DenseStep, Op, compile_ops, embed, fuse_frontier, fuse_symbolic, recipe_matrix


def _ops(n, count, kmax, seed, near):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        k = int(rng.integers(1, kmax + 1))
        if near:
            q = int(rng.integers(0, n - k + 1))
            bits = [q + int(x) for x in rng.permutation(k)]
        else:
            bits = [int(x) for x in rng.permutation(n)[:k]]
        out.append(Op(bits, workloads.haar_unitary(2 ** k, rng)))
    return out


def _product(seq, n):
    full = list(range(n - 1, -1, -1))
    m = np.eye(2 ** n, dtype=complex)
    for bits, mat in seq:
        m = embed(mat, bits, full) @ m
    return m


@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("n,count,kmax,width", [(2, 5, 2, 2), (6, 1, 1, 6), (6, 40, 2, 2), (6, 40, 3, 4), (7, 60, 2, 6),
                                                (5, 30, 2, 6), (7, 30, 4, 5)])
def test_blocks_are_the_circuit(n, count, kmax, width, near):
    ops = _ops(n, count, kmax, 10 * n + count + width, near)
    want = _product([(o.bits, o.matrix) for o in ops], n)
    blocks = fuse_frontier(ops, width)
    assert sorted(i for b in blocks for i in b.ops) == list(range(count))
    for b in blocks:
        assert len(b.bits) <= width and set(x for i in b.ops for x in ops[i].bits) <= set(b.bits)
    got = _product([(ops[i].bits, ops[i].matrix) for b in blocks for i in b.ops], n)
    assert np.max(np.abs(got - want)) < 1e-12
    plan = compile_ops(ops, n, mode="fused", width=width, device_fusion=True, pack=True)
    got = _product([(s.bits, recipe_matrix(plan.matrices[s.mat], plan.op_matrices)) for s in plan.steps], n)
    assert np.max(np.abs(got - want)) < 1e-12
    assert len(plan.steps) <= len(fuse_symbolic(ops, width))


def test_brickwork_passes():
    """28 qubits, depth 20: 62 blocks of 6 qubits (72 in the ops' order)."""
    from qaravan_gb300.statevector import circuit_ops, gates_to_ops
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(28, 20, 1)), 28)
    assert len(fuse_symbolic(ops, 6)) == 72
    plan = compile_ops(ops, 28, mode="fused", width=6, device_fusion=True, pack=True)
    assert len(plan.steps) == 62 and all(isinstance(s, DenseStep) and s.unitary for s in plan.steps)


def test_too_wide_op():
    with pytest.raises(ValueError):
        fuse_frontier([Op([0, 1, 2], np.eye(8))], 2)

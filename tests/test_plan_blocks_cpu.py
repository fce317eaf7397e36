"""The native fusion planner (``qgb_plan_blocks``) against its restatement in
Python: the same blocks, bits and op orders, over near and far ops, one to six bits wide, mixed
widths, idle bits, repeated ops, brickwork circuits and noisy layer lists, and what it refuses.
"""
import numpy as np
import pytest

from qaravan_gb300 import _lib, workloads
from qaravan_gb300.compiler import Op, SymBlock, fuse_fewest, fuse_frontier, fuse_symbolic
from qaravan_gb300.density_matrix import DensityMatrixSim
from qaravan_gb300.statevector import circuit_ops, gates_to_ops


def in_order(ops, width):
    """The order-driven planner restated in Python."""
    blocks: list = []
    last: dict = {}
    for oi, op in enumerate(ops):
        bits = list(op.bits)
        if len(bits) > width:
            raise ValueError(f"op on {len(bits)} bits exceeds fusion width {width}")
        deps = [last[b] for b in bits if b in last]
        cand = max(deps) if deps else None
        if cand is not None and blocks[cand] is not None and len(set(blocks[cand].bits) | set(bits)) <= width:
            blk = blocks[cand]
            u = sorted(set(blk.bits) | set(bits), reverse=True)
            blk.ops.append(oi)
            blk.bits = u
            for b in bits:
                last[b] = cand
            for j in sorted({d for d in deps if d != cand}, reverse=True):
                bj = blocks[j]
                if bj is None or not set(bj.bits) <= set(u):
                    continue
                if any(blocks[i] is not None and set(blocks[i].bits) & set(bj.bits) for i in range(j + 1, cand)):
                    continue
                blk.ops = bj.ops + blk.ops
                blocks[j] = None
                for b in bj.bits:
                    if last.get(b) == j:
                        last[b] = cand
            continue
        blocks.append(SymBlock(sorted(bits, reverse=True), [oi]))
        for b in bits:
            last[b] = len(blocks) - 1
    return [(b.bits, b.ops) for b in blocks if b is not None]


def frontier(ops, width):
    """The frontier planner restated in Python."""
    N = len(ops)
    obits = [tuple(op.bits) for op in ops]
    queue: dict = {}  # bit -> its ops in order
    for i, bits in enumerate(obits):
        if len(bits) > width:
            raise ValueError(f"op on {len(bits)} bits exceeds fusion width {width}")
        for b in bits:
            queue.setdefault(b, []).append(i)
    for qb in queue.values():
        qb.append(-1)  # no further op
    head = dict.fromkeys(queue, 0)
    weight = [1.0 if len(b) > 1 else 1e-3 for b in obits]

    def take(bits, pos, got):
        """Continues the in-order application on ``bits`` from ``pos`` (updated);
        appends the ops taken to ``got`` and returns their weight."""
        total, work = 0.0, list(bits)
        while work:
            b = work.pop()
            while True:
                i = queue[b][pos[b]]
                if i < 0:
                    break
                ib = obits[i]
                ok = True
                for y in ib:
                    if y not in pos or queue[y][pos[y]] != i:
                        ok = False
                        break
                if not ok:
                    break
                got.append(i)
                total += weight[i]
                for y in ib:
                    pos[y] += 1
                    if y != b and y not in work:
                        work.append(y)
        return total

    def grow(start):
        pos = {b: head[b] for b in obits[start]}
        got: list = []
        total = take(obits[start], pos, got)
        seen = set(pos)
        while len(pos) < width:
            best = None
            tried = set()
            for b in sorted(pos):
                i = queue[b][pos[b]]
                if i < 0:
                    continue
                ext = tuple(sorted(y for y in obits[i] if y not in pos))
                if not ext or len(pos) + len(ext) > width or ext in tried:
                    continue
                tried.add(ext)
                seen.update(ext)
                p2 = dict(pos)
                for y in ext:
                    p2[y] = head[y]
                g2: list = []
                gain = take(list(p2), p2, g2) / len(ext)
                if best is None or gain > best[0]:
                    best = (gain, p2, g2)
            if best is None:
                break
            total += best[0] * (len(best[1]) - len(pos))
            pos = best[1]
            got += best[2]
        return total, pos, got, seen

    cache: dict = {}  # start op -> its grown set, while nothing it looked at has moved
    blocks, done = [], 0
    while done < N:
        best = None
        for b in queue:
            i = queue[b][head[b]]
            if i < 0 or obits[i][0] != b or any(queue[y][head[y]] != i for y in obits[i]):
                continue
            hit = cache.get(i)
            if hit is None:
                hit = cache[i] = grow(i)
            if best is None or hit[0] > best[0]:
                best = hit
        _, pos, got, _ = best
        blocks.append((sorted(pos, reverse=True), got))
        done += len(got)
        head.update(pos)
        moved = set(pos)
        cache = {i: hit for i, hit in cache.items() if not (hit[3] & moved)}
    return blocks


def _same(ops, width):
    n, one, two = len(ops), in_order(ops, width), frontier(ops, width)
    back = [(bits, [n - 1 - i for i in reversed(o)]) for bits, o in reversed(frontier(ops[::-1], width))]
    for plan, want in ((fuse_symbolic, one), (fuse_frontier, two), (fuse_fewest, min(one, two, back, key=len))):
        assert [(b.bits, b.ops) for b in plan(ops, width)] == want


def _random(n, count, kmax, seed, near):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        k = int(rng.integers(1, kmax + 1))
        q = int(rng.integers(0, n - k + 1))
        out.append(Op([q + int(x) for x in rng.permutation(k)] if near else [int(x) for x in rng.permutation(n)[:k]],
                      None))
    return out


@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("n,count,kmax,width", [(1, 3, 1, 1), (2, 9, 2, 2), (5, 40, 3, 3), (6, 60, 2, 6), (9, 80, 2, 6),
                                                (20, 200, 3, 5), (28, 150, 6, 6), (40, 120, 2, 4), (68, 150, 2, 6)])
def test_random_ops(n, count, kmax, width, seed, near):
    _same(_random(n, count, kmax, 100 * n + seed, near), width)


@pytest.mark.parametrize("n,depth,width", [(7, 3, 6), (13, 4, 6), (17, 5, 5), (28, 6, 6)])
def test_circuits(n, depth, width):
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(n, depth, n)), n)
    _same(ops, width)


def test_layer_lists_of_channels():
    sim = DensityMatrixSim.__new__(DensityMatrixSim)
    sim.circ, sim.num_sites, sim.nm = workloads.noisy_brickwork_circuit(7, 3, 1), 7, None
    _same([o for o in sim.op_sequence() if o is not None], 6)


def test_nothing_and_what_is_refused():
    assert fuse_frontier([], 4) == []
    for bits in ([0, 0], [70], [-1]):
        with pytest.raises(_lib.QgbError):
            fuse_frontier([Op(bits, None)], 2)
    with pytest.raises(ValueError):
        fuse_frontier([Op([0, 1, 2], None)], 2)
    L = _lib.lib()
    assert L.qgb_plan_blocks(1, None, None, 3, 2, None, None, None, None) == _lib.QGB_EINVAL
    assert L.qgb_plan_blocks(1, None, None, -1, 2, None, None, None, None) == _lib.QGB_EINVAL
    assert L.qgb_plan_blocks(3, None, None, 0, 2, None, None, None, None) == _lib.QGB_EINVAL
    assert L.qgb_plan_blocks(2, None, None, 0, 2, None, None, None, None) == 0

"""Tensor-core passes that start before the previous launch has finished read
their operator before they wait for it (csrc/dense_tc.cu, csrc/dense_oz.cu), so
only a pass behind another one of the same plan may start early. Here the
operator is written by the very launch before: by a kernel before a single
gate, and by the fusion kernel before a new plan's first pass. 13 to 20 qubits
(one to 128 tiles, all within the early-start limit); the same plans under
graph capture and on a second stream.
"""
import numpy as np
import pytest
import torch

from qaravan_gb300 import _lib, workloads
from qaravan_gb300.compiler import compile_ops
from qaravan_gb300.engine import Executor, set_norm_restore
from qaravan_gb300.statevector import circuit_ops, gates_to_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _state(n, dtype, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    return torch.from_numpy(v / np.linalg.norm(v)).to("cuda", dtype)


@pytest.mark.parametrize("n", [13, 19])
@pytest.mark.parametrize("k", [5, 6])
def test_operator_written_by_the_launch_before(n, k):
    rng = np.random.default_rng(10 * n + k)
    ops = torch.from_numpy(np.stack([workloads.haar_unitary(2 ** k, rng) for _ in range(24)])).to("cuda", torch.complex64)
    sites = _lib.int_array([int(q) for q in rng.permutation(n)[:k]])
    L, st = _lib.lib(), _lib.stream_ptr(ops.device)
    out = []
    for wait in (True, False):
        v, op = _state(n, torch.complex64, n), torch.zeros_like(ops[0])
        torch.cuda.synchronize()
        for m in ops:
            torch.mul(m, 1.0, out=op)
            if wait:
                torch.cuda.synchronize()
            _lib.check(L.qgb_op_action(v.data_ptr(), _lib.QGB_C64, n, sites, k, op.data_ptr(), 0, 1, 0, st), "op_action")
        out.append(v)
    assert torch.equal(out[0], out[1])


def _plan(n, dtype, mode, seed):
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(n, 3, seed)), n)
    isz = 8 if dtype == torch.complex64 else 16
    width = 3 if mode == "sweep" else 6 if isz == 8 else 5
    return compile_ops(ops, n, mode=mode, width=width, itemsize=isz, device_fusion=True, pack=True)


@pytest.mark.parametrize("norm", ["row", "off"])
@pytest.mark.parametrize("n,dtype,mode", [(13, torch.complex64, "fused"), (19, torch.complex64, "fused"),
                                          (13, torch.complex128, "fixed"), (18, torch.complex128, "fixed")])
def test_first_pass_behind_the_fusion_kernel(n, dtype, mode, norm):
    set_norm_restore(norm)
    try:
        for seed in range(8):
            plan, got = _plan(n, dtype, mode, seed), []
            for wait in (True, False):
                v = _state(n, dtype, seed)
                torch.cuda.synchronize()
                ex = Executor(plan, dtype)
                if wait:
                    torch.cuda.synchronize()
                got.append(ex.run(v))
            assert torch.equal(got[0], got[1])
    finally:
        set_norm_restore("chain")


@pytest.mark.parametrize("n,dtype,mode", [(16, torch.complex64, "fused"), (20, torch.complex64, "fused"),
                                          (16, torch.complex128, "fixed"), (16, torch.complex128, "sweep")])
def test_capture_and_a_second_stream(n, dtype, mode):
    set_norm_restore("off")
    try:
        ex = Executor(_plan(n, dtype, mode, 3), dtype)
        first = _state(n, dtype, 5)
        want = ex.run(first.clone())
        side = torch.cuda.Stream()
        v = first.clone()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            ex.run(v)
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(v, want)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ex.run(v)
        for _ in range(3):
            v.copy_(first)
            g.replay()
            assert torch.equal(v, want)
    finally:
        set_norm_restore("chain")

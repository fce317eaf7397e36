"""What a plan's first run sets up: the norm chain's buffer only where a pass is a
chain link, and a call table that holds what the steps say."""
import pytest
import torch

from qaravan_gb300 import _lib, workloads
from qaravan_gb300.compiler import DenseStep, compile_ops
from qaravan_gb300.engine import Executor
from qaravan_gb300.statevector import circuit_ops, gates_to_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


@pytest.mark.parametrize("n,dtype,mode,width,links", [(8, torch.complex64, "sweep", 4, False),
                                                      (12, torch.complex64, "fused", 4, False),
                                                      (14, torch.complex128, "sweep", 3, False),
                                                      (14, torch.complex128, "fixed", 5, False),
                                                      (14, torch.complex64, "fused", 6, True)])
def test_chain_buffer_only_with_links(n, dtype, mode, width, links):
    isz = 8 if dtype == torch.complex64 else 16
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(n, 3, 1)), n)
    plan = compile_ops(ops, n, mode=mode, width=width, itemsize=isz, max_sweep_k=4, device_fusion=True, pack=True)
    ex = Executor(plan, dtype)
    state = torch.zeros(2 ** n, dtype=dtype, device="cuda")
    state[0] = 1
    ex.run(state)
    assert (getattr(ex, "_chain", None) is not None) == links
    (table, _, count, _), = ex._calls.values()
    assert count == len(plan.steps) == len(table)
    for c, s in zip(table, plan.steps):
        if isinstance(s, DenseStep):
            want = _lib.QGB_CALL_CHAIN if links else _lib.QGB_CALL_FIXED if s.fixed else _lib.QGB_CALL_ROWS
            assert (c["kind"], c["k"], c["mat"]) == (want, len(s.bits), ex.mat_offsets[s.mat])
            assert c["sites"].tolist()[:c["k"]] == [n - 1 - b for b in s.bits]
        else:
            assert c["kind"] == _lib.QGB_CALL_SWEEP and c["sweep"] != 0

"""Tile sweeps of a batch whose states lie further apart than 2^n: every state
gets what it gets alone, bit for bit, and the elements between the states stay as
they were. Strides whose batch offsets share bits with the tile's own index
(2^n + 8) and with the tile number's place (2^n + 2^(n-1)), one tile and several
per state, few states (clusters) and many (one CTA per tile), in complex64,
double-float and float64, and the TMA kernel.
"""
import numpy as np
import pytest
import torch

from qaravan_gb300 import _lib, workloads
from qaravan_gb300.compiler import SweepStep, compile_ops
from qaravan_gb300.engine import Executor
from qaravan_gb300.statevector import circuit_ops, gates_to_ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _check(n, tile, batch, extra, dtype):
    ops = gates_to_ops(circuit_ops(workloads.brickwork_circuit(n, 2, 90 + n)), n)
    isz = 8 if dtype == torch.complex64 else 16
    plan = compile_ops(ops, n, mode="sweep", width=3, tile_bits=tile, max_sweep_k=4, itemsize=isz, device_fusion=True)
    assert all(isinstance(s, SweepStep) for s in plan.steps)
    ex = Executor(plan, dtype)
    stride, rng = 2 ** n + extra, np.random.default_rng(n + batch)
    v = rng.standard_normal((batch, stride)) + 1j * rng.standard_normal((batch, stride))
    x = torch.from_numpy(v).to("cuda", dtype)
    want = x.clone()
    for i in (range(batch) if batch < 10 else (0, 1, batch - 1)):
        want[i, :2 ** n] = ex.run(want[i, :2 ** n].clone())
    ex.run(x, batch=batch, stride=stride)
    assert torch.equal(x[:, 2 ** n:], want[:, 2 ** n:])
    for i in (range(batch) if batch < 10 else (0, 1, batch - 1)):
        assert torch.equal(x[i], want[i]), i


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,tile,batch,extra", [(10, 13, 3, 8), (10, 13, 5, 2), (10, 13, 160, 8), (12, 10, 4, 8),
                                                (12, 10, 3, 2 ** 11), (12, 10, 50, 2 ** 11 + 8), (14, 12, 2, 2 ** 13),
                                                (16, 12, 3, 2 ** 15 + 8), (16, 12, 12, 2 ** 14 + 2)])
def test_padded_batches(n, tile, batch, extra, dtype):
    _check(n, tile, batch, extra, dtype)


def test_padded_batches_float64():
    L = _lib.lib()
    L.qgb_set_c128_arith(0)
    try:
        _check(12, 10, 3, 2 ** 11 + 8, torch.complex128)
    finally:
        L.qgb_set_c128_arith(1)


def test_padded_batches_tma():
    L = _lib.lib()
    L.qgb_set_sweep_impl(1)
    try:
        _check(14, 12, 3, 2 ** 13 + 16, torch.complex64)
    finally:
        L.qgb_set_sweep_impl(0)

"""5-qubit complex128 blocks in fixed point on the tensor cores (csrc/dense_oz.cu)
against NumPy: one tile and several, targets low, high and mixed in any order
(rows written directly and through shared memory), zero rows, rows of very
different scale, values that are not finite, the ops the kernel leaves to
others, and whole circuits on the default path.

Tolerance: components are kept to 2^-50 of their row's largest, the operator to
2^-51 of its largest entry, so one block's error is below
64 (2^-50 + 2^-51) max|row| max|w| < 9e-14 max|row| (typically 1e-15)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu

EPS = 9e-14


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _apply(v, m, sites, n):
    k = len(sites)
    t = np.tensordot(m.reshape([2] * (2 * k)), v.reshape([2] * n), axes=(list(range(k, 2 * k)), sites))
    return np.moveaxis(t, list(range(k)), sites).reshape(-1)


def _run(v, m, sites, n):
    from qaravan_gb300 import _lib
    st = torch.from_numpy(v.copy()).cuda()
    op = torch.from_numpy(np.ascontiguousarray(m)).cuda()
    L = _lib.lib()
    call = _lib.Call(kind=_lib.QGB_CALL_FIXED, k=len(sites), mat=0)
    for j, q in enumerate(sites):
        call.sites[j] = q
    _lib.check(L.qgb_run_calls(st.data_ptr(), 1, n, ctypes.byref(call), 1, op.data_ptr(), None, None,
                               _lib.stream_ptr(st.device)), "run_calls")
    _lib.check(L.qgb_check_status(None))
    return st.cpu().numpy()


SITES = [[0, 1, 2, 3, 4], [-5, -4, -3, -2, -1], [-1, 0, 5, -3, 2], [4, 3, 2, 1, 0], [-4, -8, 1, -2, 6], [-6, -5, -4, 0, 3]]


@pytest.mark.parametrize("n", [12, 13, 16, 20])
@pytest.mark.parametrize("sites", SITES)
def test_block_against_numpy(n, sites):
    from qaravan_gb300 import workloads
    rng = np.random.default_rng(n)
    sites = [s % n for s in sites]
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    m = workloads.haar_unitary(32, rng)
    assert np.max(np.abs(_run(v, m, sites, n) - _apply(v, m, sites, n))) < EPS * np.max(np.abs(v))


def test_rows_of_different_scale():
    """Each group is scaled by itself: zero groups stay zero, small ones keep their accuracy."""
    from qaravan_gb300 import workloads
    n, rng = 14, np.random.default_rng(1)
    sites = [1, 4, 6, 9, 12]
    m = workloads.haar_unitary(32, rng)
    t = (rng.standard_normal([2] * n) + 1j * rng.standard_normal([2] * n))
    rest = [q for q in range(n) if q not in sites]
    scale = 10.0 ** rng.integers(-280, 280, [2] * len(rest))
    scale[0, 0] = 0.0
    full = np.ones([2] * n) * np.moveaxis(scale.reshape([2] * len(rest) + [1] * 5), range(n), rest + sites)
    v = (t * full).reshape(-1)
    got, want = _run(v, m, sites, n).reshape([2] * n), _apply(v, m, sites, n).reshape([2] * n)
    err = np.max(np.abs(got - want), axis=tuple(sites))
    big = np.max(np.abs(v.reshape([2] * n)), axis=tuple(sites))
    assert np.all(err <= EPS * big)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_stay_in_their_group(bad):
    from qaravan_gb300 import workloads
    n, rng = 13, np.random.default_rng(2)
    sites = [0, 3, 5, 8, 11]
    v = rng.standard_normal(2 ** n) + 0j
    v[7] = bad
    got = _run(v, workloads.haar_unitary(32, rng), sites, n).reshape([2] * n)
    hit = np.zeros([2] * n, bool)
    hit.reshape(-1)[7] = True
    hit = np.broadcast_to(np.any(hit, axis=tuple(sites), keepdims=True), hit.shape)
    assert not np.any(np.isfinite(got[hit])) and np.all(np.isfinite(got[~hit]))


@pytest.mark.parametrize("k,n", [(4, 14), (5, 11), (6, 14)])
def test_other_blocks_run_elsewhere(k, n):
    from qaravan_gb300 import workloads
    rng = np.random.default_rng(k)
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    m = workloads.haar_unitary(2 ** k, rng)
    sites = [int(q) for q in rng.permutation(n)[:k]]
    assert np.max(np.abs(_run(v, m, sites, n) - _apply(v, m, sites, n))) < 1e-13 * np.max(np.abs(v)) * 2 ** k


@pytest.mark.parametrize("n,depth", [(17, 2), (18, 1)])
def test_default_complex128_path(n, depth):
    from qaravan_gb300 import StatevectorSim, workloads
    gates = workloads.brickwork_gates(n, depth, 5)
    sim = StatevectorSim(workloads.brickwork_circuit(n, depth, 5), dtype=torch.complex128)
    assert (sim.mode, sim.fusion_width) == ("fixed", 5)
    assert all(len(s.bits) == 5 for s in sim.compile().plan.steps)
    assert np.max(np.abs(sim.get_statevector().cpu().numpy() - ref.run_sv(gates, n))) < 1e-13


def test_reset_and_wide_gates_keep_the_sweeps():
    """A projector or a gate of 6 qubits is not a fixed-point block: its segment runs as before."""
    from qaravan_gb300 import StatevectorSim, workloads
    from qaravan_gb300.circuits import Circuit
    from qaravan_gb300.gates import Gate, Reset
    n, rng = 17, np.random.default_rng(3)
    gates = workloads.brickwork_circuit(n, 1, 5).gate_list
    wide = Gate("U", [int(q) for q in rng.permutation(n)[:6]], workloads.haar_unitary(64, rng))
    for extra in (wide, Reset([3], "0")):
        circ = Circuit(gates + [extra], n)
        a = StatevectorSim(circ, dtype=torch.complex128)
        b = StatevectorSim(circ, dtype=torch.complex128, mode="sweep", fusion_width=3, tile_bits=13)
        plan, ref_plan = a.compile().plan, b.compile().plan
        assert [type(s) for s in plan.steps] == [type(s) for s in ref_plan.steps]
        assert torch.equal(a.get_statevector(), b.get_statevector())


def test_same_kernel_with_the_norm_off():
    """Norm restoring is a complex64 matter: without it complex128 blocks run as they do."""
    from qaravan_gb300 import StatevectorSim, engine, workloads
    circ = workloads.brickwork_circuit(17, 1, 5)
    a = StatevectorSim(circ, dtype=torch.complex128).get_statevector()
    engine.set_norm_restore("off")
    try:
        b = StatevectorSim(circ, dtype=torch.complex128).get_statevector()
    finally:
        engine.set_norm_restore("chain")
    assert torch.equal(a, b)


def test_other_entries_keep_their_arithmetic():
    """Blocks asked for as fused, the unitary entry of the C ABI and another width run as before."""
    from qaravan_gb300 import StatevectorSim, _lib, workloads
    n, rng = 17, np.random.default_rng(4)
    circ = workloads.brickwork_circuit(n, 1, 5)
    assert not any(s.fixed for s in StatevectorSim(circ, dtype=torch.complex128, mode="fused", fusion_width=5).compile().plan.steps)
    assert StatevectorSim(circ, dtype=torch.complex128, fusion_width=4).mode == "sweep"
    v = rng.standard_normal(2 ** 12) + 1j * rng.standard_normal(2 ** 12)
    m = workloads.haar_unitary(32, rng)
    st, op = torch.from_numpy(v.copy()).cuda(), torch.from_numpy(m.copy()).cuda()
    L, sites = _lib.lib(), [0, 1, 2, 3, 4]
    _lib.check(L.qgb_op_action_unitary(st.data_ptr(), 1, 12, _lib.int_array(sites), 5, op.data_ptr(), 0, 1, 0,
                                       _lib.stream_ptr(st.device)), "op_action")
    # float64 sums of 64 products: far below the fixed-point kernel's 2^-50 of the row
    err = np.abs(st.cpu().numpy() - _apply(v, m, sites, 12))
    assert np.max(err) < 128 * 2.0 ** -53 * np.max(np.abs(v))


def test_steps_one_by_one():
    """A plan run step by step (with events) gives the one-call run's state."""
    from qaravan_gb300 import StatevectorSim, workloads
    sim = StatevectorSim(workloads.brickwork_circuit(17, 1, 5), dtype=torch.complex128)
    want = sim.run().reshape(-1).clone()
    sim.initialize_state()
    sim.compile().run(sim.state, events=[])
    assert torch.equal(sim.state.reshape(-1), want)

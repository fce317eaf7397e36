"""Every amplitude's own accuracy in the fixed-point blocks (csrc/dense_oz.cu).

The kernel keeps the 32 amplitudes of a group to 2^-50 of the largest, so an
output is left to it only where the block draws it from large amplitudes, and is
formed in double-float elsewhere. Against the same sums in extended precision,
with B_i = sum_j |U_ij| |x_j| of output i and M its group's largest component:

* certified outputs have B_i >= M / 32, and their error is at most
  (5.7 * 1.42 * 2^-50 + 46 * 1.42 * 2^-51 + 2^-47) M < 2^-43.9 M < 2^-38 B_i (every
  component of the row rounded by 2^-50 M, every entry of the block by 2^-51, the
  dropped digit pairs); in a row of at most 8 components, all within 1/8 of the
  largest, one product is enough: B_i >= M / 128 and an error below 2^-45.4 M;
* the others carry 48 bits through 32 products: below 2^-41 B_i.

A random block on random amplitudes stays within 2.5e-15 of the norm (rounding
the components and the entries to their last place, 1.4 * 2^-50; without the
smallest digits that are summed it is 2e-14).
"""
import ctypes

import numpy as np
import pytest
import torch

from qaravan_gb300 import _lib, workloads

pytestmark = pytest.mark.gpu

BOUND = 2.0 ** -38


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _run(v, m, sites, n):
    st, op = torch.from_numpy(v.copy()).cuda(), torch.from_numpy(np.ascontiguousarray(m)).cuda()
    L = _lib.lib()
    call = _lib.Call(kind=_lib.QGB_CALL_FIXED, k=5, mat=0)
    for j, q in enumerate(sites):
        call.sites[j] = q
    _lib.check(L.qgb_run_calls(st.data_ptr(), _lib.QGB_C128, n, ctypes.byref(call), 1, op.data_ptr(), None, None,
                               _lib.stream_ptr(st.device)), "run_calls")
    _lib.check(L.qgb_check_status(None))
    return st.cpu().numpy()


def _groups(v, sites, n):
    return np.moveaxis(v.reshape([2] * n), sites, range(5)).reshape(32, -1)


def _compare(v, m, sites, n):
    """(errors, B) per amplitude, extended precision."""
    x, u = _groups(v, sites, n).astype(np.clongdouble), m.astype(np.clongdouble)
    want = np.zeros_like(x)
    for j in range(32):  # (no BLAS for extended precision)
        want += u[:, j:j + 1] * x[j:j + 1]
    got = _groups(_run(v, m, sites, n), sites, n).astype(np.clongdouble)
    return np.abs(got - want).astype(float), (np.abs(m) @ np.abs(_groups(v, sites, n)))


def _phases(rng):
    return np.diag(np.exp(2j * np.pi * rng.random(32)))


def _permutation(rng):
    return np.eye(32)[rng.permutation(32)].astype(complex)


def _small_rotations(rng):
    m = np.eye(1)
    for th in 1e-3 * rng.standard_normal(5):
        m = np.kron(m, np.array([[np.cos(th), -1j * np.sin(th)], [-1j * np.sin(th), np.cos(th)]]))
    return m


def _pair(rng):
    """A Haar pair gate beside three idle sites."""
    return np.kron(np.eye(8), workloads.haar_unitary(4, rng))


def _haar(rng):
    return workloads.haar_unitary(32, rng)


BLOCKS = {f.__name__[1:]: f for f in (_phases, _permutation, _small_rotations, _pair, _haar)}


def _random(n, rng):
    return rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)


def _tail(n, rng, low=1e-12):
    """One large amplitude a group or so, the rest about `low` of it."""
    return _random(n, rng) * np.where(rng.random(2 ** n) < 0.04, 1.0, low)


STATES = {"random": _random, "tail_1e-12": _tail, "tail_1e-17": lambda n, rng: _tail(n, rng, 1e-17),
          "spread": lambda n, rng: _random(n, rng) * 10.0 ** rng.uniform(-25, 0, 2 ** n),
          "basis": lambda n, rng: np.eye(1, 2 ** n, 5, dtype=complex)[0],
          "small_numbers": lambda n, rng: _tail(n, rng) * 1e-290}


@pytest.mark.parametrize("sites", [[0, 1, 2, 3, 4], [8, 9, 10, 11, 12], [12, 0, 5, 10, 2], [4, 6, 8, 3, 7]])
@pytest.mark.parametrize("state", list(STATES))
@pytest.mark.parametrize("block", list(BLOCKS))
def test_every_amplitude(block, state, sites):
    n, rng = 13, np.random.default_rng(len(block) + 10 * len(state) + sites[0])
    v, m = STATES[state](n, rng).astype(complex), BLOCKS[block](rng).astype(complex)
    err, b = _compare(v, m, sites, n)
    assert np.all(err <= BOUND * b + 1e-307)


@pytest.mark.parametrize("sites", [[0, 1, 2, 3, 4], [8, 9, 10, 11, 12]])
def test_last_digits(sites):
    rng = np.random.default_rng(2)
    v = _random(13, rng)
    err, _ = _compare(v, _haar(rng), sites, 13)
    assert np.sqrt((err ** 2).sum() / (np.abs(v) ** 2).sum()) < 2.5e-15


@pytest.mark.parametrize("kind", ["phases", "rotations", "permutations", "haar"])
def test_circuits_by_default(kind):
    """17 qubits, the default path, from a state with a tail: every amplitude to 2e-11 of what the
    circuit draws it from (up to 6 blocks of 2^-38)."""
    from qaravan_gb300 import StatevectorSim
    from qaravan_gb300.circuits import Circuit
    from qaravan_gb300.gates import Gate
    n, rng = 17, np.random.default_rng(9)
    gates = []
    for l in range(2):
        for q in range(l, n - 1, 2):
            if kind == "haar":
                gates.append(Gate("u", [q, q + 1], workloads.haar_unitary(4, rng)))
            elif kind == "phases":
                gates.append(Gate("u", [q, q + 1], np.diag(np.exp(2j * np.pi * rng.random(4)))))
            elif kind == "permutations":
                gates.append(Gate("u", [q, q + 1], np.eye(4)[rng.permutation(4)].astype(complex)))
            else:
                th = 1e-3 * rng.standard_normal()
                gates.append(Gate("u", [q], np.array([[np.cos(th), -1j * np.sin(th)], [-1j * np.sin(th), np.cos(th)]])))
    v = _tail(n, rng)
    got = StatevectorSim(Circuit(gates, n=n), init_state=v, dtype=torch.complex128).run().reshape(-1).cpu().numpy()
    x, b = v.astype(np.clongdouble), np.abs(v)
    for g in gates:
        k = len(g.indices)
        for what in (0, 1):
            y, m = (x, g.matrix.astype(np.clongdouble)) if what == 0 else (b, np.abs(g.matrix))
            t = np.moveaxis(y.reshape([2] * n), g.indices, range(k)).reshape(2 ** k, -1)
            t = sum(m[:, j:j + 1] * t[j:j + 1] for j in range(2 ** k))
            t = np.moveaxis(t.reshape([2] * n), range(k), g.indices).reshape(-1)
            x, b = (t, b) if what == 0 else (x, t)
    assert np.all(np.abs(got - x).astype(float) <= 6 * BOUND * b)


@pytest.mark.parametrize("n,depth", [(19, 4), (20, 20), (22, 3)])
def test_passes_and_the_sweep_behind_them(n, depth):
    """Whole circuits with a narrow tail against float64 sweeps: below 1e-13 of the norm (double-float sweeps
    leave 5e-14 after such circuits, the passes less)."""
    from qaravan_gb300 import StatevectorSim
    circ = workloads.brickwork_circuit(n, depth, 3)
    L = _lib.lib()
    _lib.check(L.qgb_set_c128_arith(0))
    try:
        want = StatevectorSim(circ, dtype=torch.complex128, mode="sweep", fusion_width=3, tile_bits=13).run()
    finally:
        _lib.check(L.qgb_set_c128_arith(1))
    got = StatevectorSim(circ, dtype=torch.complex128).run()
    assert torch.linalg.vector_norm(got - want).item() < 1e-13

"""The adjoint tile sweep's index map and straight-line programs: permutations at
the start, the middle and the end of runs (CNOT both ways, SWAP, X), rotation
pairs on one, two and three bits in and out of order, single rotations of every
kind, more than 32 derivatives per pass, one and several tiles per chunk, tiles
smaller than a block of threads. Energies and gradients against the per-gate
reverse steps: complex128 to 1e-10 of the largest entry, complex64 to 2e-5 (the
complex64 gradient bar of the suite)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

X = np.array([[0, 1], [1, 0]], complex)
CX = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], complex)
XC = np.array([[1, 0, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0], [0, 1, 0, 0]], complex)
SWAP = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], complex)


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _gates(n, count, rng):
    gates, p = [], 0
    kinds = ["pair", "pair", "RX", "RY", "RZ", "RZZ", "CX", "CX", "XC", "SWAP", "X", "dense"]
    for _ in range(count):
        kind = kinds[int(rng.integers(0, len(kinds)))]
        a, b = (int(q) for q in rng.permutation(n)[:2])
        if kind == "pair":  # the reverse sweep meets RZ, then RY
            gates += [("RY", [a], p), ("RZ", [a], p + 1)]
            p += 2
        elif kind in ("RX", "RY", "RZ"):
            gates.append((kind, [a], p))
            p += 1
        elif kind == "RZZ":
            gates.append((kind, [a, b], p))
            p += 1
        elif kind == "X":
            gates.append(("fixed", [a], X))
        elif kind == "dense":
            q, r = np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))
            gates.append(("fixed", [a, b], q * (np.diag(r) / np.abs(np.diag(r)))))
        else:
            gates.append(("fixed", [a, b], {"CX": CX, "XC": XC, "SWAP": SWAP}[kind]))
    return gates, p


def _both(n, gates, nparams, sets, dtype, terms, rng):
    from qaravan_gb300.adjoint import BatchedAnsatz
    th = rng.uniform(0, 2 * np.pi, (sets, max(nparams, 1)))
    out = []
    for kw in ({}, {"tile_bits": 0}):
        e, g = BatchedAnsatz(n, gates, nparams=max(nparams, 1), dtype=dtype, **kw).energy_and_grad(th, terms)
        out.append((e.cpu().numpy(), g.cpu().numpy()))
    return out


def _check(got, want, dtype):
    tol = 2e-5 if dtype == torch.complex64 else 1e-10
    for a, b in zip(got, want):
        assert np.max(np.abs(a - b)) < tol * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,count,sets", [(3, 30, 2), (5, 60, 3), (11, 150, 2), (12, 120, 1), (13, 200, 5)])
def test_random_circuits(n, count, sets, dtype):
    from qaravan_gb300.hamiltonians import TFI
    rng = np.random.default_rng(n * 1000 + count)
    gates, p = _gates(n, count, rng)
    got, want = _both(n, gates, p, sets, dtype, TFI(n, 1.0, 0.7).pauli_sum(), rng)
    _check(got, want, dtype)


@pytest.mark.parametrize("dtype,n,layers,sets", [(torch.complex64, 14, 4, 200), (torch.complex64, 4, 3, 9),
                                                 (torch.complex128, 12, 3, 3), (torch.complex64, 16, 3, 1)])
def test_ladder_ansatz(dtype, n, layers, sets):
    from qaravan_gb300.adjoint import BatchedAnsatz
    from qaravan_gb300.hamiltonians import TFI
    ba = BatchedAnsatz.hea(n, layers, dtype=dtype)
    got, want = _both(n, ba.gates, ba.nparams, sets, dtype, TFI(n, 1.0, 1.0).pauli_sum(), np.random.default_rng(n))
    _check(got, want, dtype)

"""Pauli sums of complex128 states by shared-memory tiles (csrc/pauli_tiles.cu): values
that are not finite, zero coefficients, sums of many passes, and a sum with one mask too wide for
a tile (the general kernels), each term against the same term alone, which the general
kernel takes.

Tolerance: float64 sums of 2^n products of a unit vector, 2^-53 each, in another
order: 1e-13.
"""
import numpy as np
import pytest
import torch

from qaravan_gb300 import _lib
from qaravan_gb300.statevector import pauli_expectations

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _apply(psi, n, terms):
    out = torch.full_like(psi, 7.0)
    _lib.check(_lib.lib().qgb_pauli_apply(psi.data_ptr(), out.data_ptr(), _lib.QGB_C128, n,
                                          "".join(s for _, s in terms).encode(), _lib.double_array([c for c, _ in terms]),
                                          len(terms), 1, 0, _lib.stream_ptr(psi.device)), "pauli_apply")
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [5, 11, 13])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_special_values(n, bad):
    """They reach every term that reads them with a coefficient that is not zero, and, applied, their partners only."""
    def at(q, p):
        return "i" * q + p + "i" * (n - q - len(p))
    terms = [(1.0, at(0, "z")), (0.5, at(n - 1, "z")), (1.0, at(0, "zz")), (1.0, at(0, "x")), (2.0, at(n - 2, "yx")),
             (1.0, at(1, "y")), (0.0, at(2, "x")), (0.0, at(1, "z"))]
    psi = torch.zeros(2 ** n, dtype=torch.complex128, device="cuda")
    psi[5] = complex(bad, 0.0)
    psi[2] = 0.5
    many = pauli_expectations(psi, n, terms).cpu().numpy()
    single = np.array([pauli_expectations(psi, n, [t]).cpu().numpy()[0] for t in terms])
    assert np.array_equal(np.isfinite(many), np.isfinite(single))
    assert np.array_equal(many[np.isposinf(single)], single[np.isposinf(single)])
    got = _apply(psi, n, terms[:6])
    idx = np.arange(2 ** n)
    hit = np.zeros(2 ** n, bool)
    for _, s in terms[:6]:
        x = sum(1 << (n - 1 - q) for q, c in enumerate(s) if c in "xy")
        hit |= (idx ^ x) == 5
    assert not np.isfinite(got[hit]).any() and np.isfinite(got[~hit]).all()


@pytest.mark.parametrize("n,count,wide", [(9, 1000, False), (14, 300, False), (16, 300, True)])
def test_many_passes(n, count, wide):
    rng = np.random.default_rng(n)
    letters, terms = np.array(list("ixyz")), []
    for _ in range(count):
        w = int(rng.integers(1, min(n, 8) + 1))
        q = int(rng.integers(0, n - w + 1))
        terms.append((float(rng.uniform(-1, 1)), "i" * q + "".join(letters[rng.integers(0, 4, w)]) + "i" * (n - q - w)))
    if wide:  # more X bits above the lowest three than a tile holds
        terms.insert(7, (1.0, "x" * n))
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    psi = torch.from_numpy(v / np.linalg.norm(v)).cuda()
    many = pauli_expectations(psi, n, terms).cpu().numpy()
    single = np.array([pauli_expectations(psi, n, [t]).cpu().numpy()[0] for t in terms])
    assert np.max(np.abs(many - single)) < 1e-13


def _times(psi, n, s):
    """P psi for a Pauli string, site 0 most significant."""
    idx = np.arange(2 ** n)
    src = idx ^ sum(1 << (n - 1 - q) for q, c in enumerate(s) if c in "xy")
    out = psi[src]
    for q, c in enumerate(s):
        b = (src >> (n - 1 - q)) & 1
        if c == "z":
            out = out * (1 - 2 * b)
        elif c == "y":  # Y|0> = i|1>, Y|1> = -i|0>
            out = out * np.where(b == 0, 1j, -1j)
    return out


@pytest.mark.parametrize("n,kind", [(15, "diagonal"), (16, "diagonal"), (17, "diagonal"), (19, "chain"), (20, "chain"),
                                    (21, "chain"), (20, "one")])
def test_applied_on_both_sides_of_the_rule(n, kind):
    """The tile form from 20 qubits (16 for diagonal sums), in several passes that add to `out`, and the
    general kernel below: at most two roundings a term and amplitude, 2^-53 each, in either."""
    rng = np.random.default_rng(n)
    if kind == "diagonal":
        terms = [(float(rng.uniform(-1, 1)), "".join(rng.choice(list("iz"), n))) for _ in range(100)]
    elif kind == "one":
        terms = [(0.7, "i" * (n - 3) + "yxz")]
    else:
        terms = [(float(rng.uniform(-1, 1)), "i" * q + p + "i" * (n - q - len(p))) for p in ("z", "yy", "xz")
                 for q in range(0, n - len(p) + 1, 2)]
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    want = sum(c * _times(v, n, s) for c, s in terms)
    got = _apply(torch.from_numpy(v).cuda(), n, terms)
    assert np.max(np.abs(got - want)) < 4 * len(terms) * 2.0 ** -53 * np.max(np.abs(v))

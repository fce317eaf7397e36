"""Pauli sums by shared-memory tiles (csrc/pauli_tiles.cu): expectation values
and H psi of many terms against a float64 NumPy restatement, at the edges of the
rules: one partial tile, one full tile, several tiles and passes, more terms
than a pass holds, masks of many bits (linear runs), masks too wide for a tile
and states off the 16-byte alignment (both the general kernels), batches.

Tolerances: complex64 sums are float32 chains of at most 16 + 16 + 16 roundings
of parts of sum |psi|^2 = 1 per unit coefficient (48 * 2^-24 = 3e-6); an applied
amplitude has at most two roundings per term. complex128 the same at 2^-53,
taken as 1e-13.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _apply(psi, n, s):
    """P psi for a Pauli string, site 0 most significant."""
    idx = np.arange(2 ** n)
    x = sum(1 << (n - 1 - q) for q, c in enumerate(s) if c in "xy")
    out = psi[idx ^ x].astype(np.complex128)
    src = idx ^ x
    for q, c in enumerate(s):
        b = (src >> (n - 1 - q)) & 1
        if c == "z":
            out = out * (1 - 2 * b)
        elif c == "y":  # Y|0> = i|1>, Y|1> = -i|0>
            out = out * np.where(b == 0, 1j, -1j)
    return out


def _strings(n, kind, count, rng):
    if kind == "chain":  # Ising and Heisenberg chain terms
        out = ["i" * q + p + "i" * (n - q - 1) for p in "xyz" for q in range(n)]
        out += ["i" * q + p + "i" * (n - q - 2) for p in ("xx", "yy", "zz", "xy") for q in range(n - 1)]
        return out
    letters = np.array(list("ixyz"))
    if kind == "dense":
        return ["".join(letters[rng.integers(0, 4, n)]) for _ in range(count)]
    out = []  # "diag" and "near": long strings over few neighbouring sites
    for _ in range(count):
        if kind == "diag":
            out.append("".join(np.array(list("iz"))[rng.integers(0, 2, n)]))
        else:
            w = min(n, 6)
            q = int(rng.integers(0, n - w + 1))
            out.append("i" * q + "".join(letters[rng.integers(0, 4, w)]) + "i" * (n - q - w))
    return out


def _state(n, batch, dtype, rng):
    v = rng.standard_normal((batch, 2 ** n)) + 1j * rng.standard_normal((batch, 2 ** n))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return torch.from_numpy(v).to("cuda", dtype)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,kind,count,batch", [(4, "chain", 0, 1), (5, "chain", 0, 1), (7, "dense", 40, 3),
                                                (11, "near", 30, 1), (12, "dense", 100, 1), (13, "chain", 0, 2),
                                                (13, "diag", 120, 1), (16, "near", 60, 1), (17, "dense", 6, 1),
                                                (18, "chain", 0, 1)])
def test_expectation_and_apply(n, kind, count, batch, dtype):
    from qaravan_gb300 import _lib
    from qaravan_gb300.statevector import pauli_expectations
    rng = np.random.default_rng(n * 100 + count)
    strings = _strings(n, kind, count, rng)
    coeff = rng.uniform(-1.0, 1.0, len(strings))
    psi = _state(n, batch, dtype, rng)
    host = psi.cpu().numpy().astype(np.complex128)
    want = np.array([[c * np.vdot(v, _apply(v, n, s)).real for c, s in zip(coeff, strings)] for v in host])
    got = pauli_expectations(psi.reshape(-1), n, list(zip(coeff, strings)), batch=batch, stride=2 ** n)
    tol = 3e-6 if dtype == torch.complex64 else 1e-13
    assert np.max(np.abs(got.cpu().numpy().reshape(batch, -1) - want)) < tol
    if len(strings) > 128:
        strings, coeff = strings[:128], coeff[:128]
    out = torch.full_like(psi, float("nan"))
    _lib.check(_lib.lib().qgb_pauli_apply(psi.data_ptr(), out.data_ptr(), _lib.dtype_code(dtype), n,
                                          "".join(strings).encode(), _lib.double_array(coeff), len(strings), batch,
                                          2 ** n, _lib.stream_ptr(psi.device)), "pauli_apply")
    ref = np.stack([sum(c * _apply(v, n, s) for c, s in zip(coeff, strings)) for v in host])
    eps = 2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -53
    assert np.max(np.abs(out.cpu().numpy() - ref)) < 4 * len(strings) * eps * np.max(np.abs(host))


def test_unaligned_state_takes_the_general_kernels():
    from qaravan_gb300.statevector import pauli_expectations
    n, rng = 9, np.random.default_rng(3)
    buf = torch.zeros(2 ** n + 1, dtype=torch.complex64, device="cuda")
    buf[1:] = _state(n, 1, torch.complex64, rng).reshape(-1)
    terms = [(1.0, s) for s in _strings(n, "chain", 0, rng)]
    a = pauli_expectations(buf[1:], n, terms).cpu().numpy()
    b = pauli_expectations(buf[1:].clone(), n, terms).cpu().numpy()
    assert np.max(np.abs(a - b)) < 3e-6


def test_special_values_reach_the_result():
    """A NaN or an infinity in the state reaches every term that reads it, in both forms."""
    from qaravan_gb300.statevector import pauli_expectations
    n = 13
    terms = [(1.0, "z" + "i" * (n - 1)), (1.0, "x" + "i" * (n - 1)), (0.0, "y" + "i" * (n - 1))]
    for bad in (float("nan"), float("inf")):
        psi = torch.zeros(2 ** n, dtype=torch.complex64, device="cuda")
        psi[5] = bad
        many = pauli_expectations(psi, n, terms).cpu().numpy()
        single = np.array([pauli_expectations(psi, n, [t]).cpu().numpy()[0] for t in terms])
        assert np.array_equal(np.isfinite(many), np.isfinite(single))

"""The work a user of this framework has it do, as measurable cases.

Each case is one call (or the few calls that belong together) through the
public entry points, on inputs made from a seed. ``listed()`` names twelve of
them over the real range of sizes, ``draw()`` gives more of the same ranges,
``exact()`` is the same result in 64-bit arithmetic with plain torch (GPU) on
the same inputs, and ``work()`` the bytes and operations a pass cannot do
without: inputs read once, outputs written once, every gate's own product.

Kinds:

* ``op``: ``tensorQ.op_action``, one gate on one state.
* ``sv``: ``StatevectorSim.run()`` of a simulator whose circuit is compiled, the
  Haar brickwork of this repository's benchmark (depth unit: SU(2) on every
  site, SU(4) on the even and the odd pairs), from |0..0> or a given state.
* ``pauli``: the transverse-field Ising energy terms of a state, one float64 each.
* ``dm``: ``DensityMatrixSim.run()`` of the noisy brickwork (depolarising
  channel after every two-qubit gate) from a compiled simulator.
* ``dm_batch``: ``DensityMatrixBatch`` of uneven noisy brickworks.
* ``traj``: ``TrajectorySim`` on the Ising Trotter circuit, depolarising and
  damping after every gate, and the Pauli expectations of every trajectory.
* ``grad``: one step of a variational loop: circuit from a parameter tensor,
  ``adjoint_energy`` and its backward.
* ``grad_batch``: ``BatchedAnsatz.energy_and_grad``, many parameter sets at once.
"""
from __future__ import annotations

import numpy as np
import torch

import qaravan_gb300 as qg
from qaravan_gb300 import tensorQ, workloads
from qaravan_gb300.adjoint import BatchedAnsatz, adjoint_energy
from qaravan_gb300.batch import DensityMatrixBatch
from qaravan_gb300.circuits import Circuit
from qaravan_gb300.density_matrix import DensityMatrixSim
from qaravan_gb300.gates import ID, Gate
from qaravan_gb300.hamiltonians import TFI
from qaravan_gb300.noise import depolarizing
from qaravan_gb300.statevector import StatevectorSim, pauli_expectations
from qaravan_gb300.trajectories import TrajectorySim, z_terms

DEV = "cuda"
P_DEP = 1e-3   # depolarising probability after a gate, as in the benchmark's noisy workloads
GAMMA = 5e-4   # amplitude damping of the trajectory workload
DT = 0.05      # Trotter step of the trajectory workload


def listed():
    return [
        # one gate applied by hand to a small state: the shortest call there is
        {"name": "op_10q_c64", "kind": "op", "n": 10, "k": 2, "bits": 64},
        # the benchmark's CPU-sized circuit in the reference's NumPy precision: launches count
        {"name": "sv_12q_c128", "kind": "sv", "n": 12, "depth": 20, "bits": 128, "start": "zero"},
        # an ordinary circuit whose state stays in cache, from a given state
        {"name": "sv_19q_c64", "kind": "sv", "n": 19, "depth": 20, "bits": 64, "start": "random"},
        # the benchmark's headline circuit
        {"name": "sv_28q_c64", "kind": "sv", "n": 28, "depth": 20, "bits": 64, "start": "zero"},
        # double precision, odd size, state well beyond the cache
        {"name": "sv_25q_c128", "kind": "sv", "n": 25, "depth": 8, "bits": 128, "start": "zero"},
        # energy of a large state, term by term
        {"name": "pauli_27q_c64", "kind": "pauli", "n": 27, "bits": 64},
        # a small noisy circuit
        {"name": "dm_6q_c64", "kind": "dm", "n": 6, "depth": 10, "bits": 64},
        # the largest single density matrix of the benchmark
        {"name": "dm_13q_c64", "kind": "dm", "n": 13, "depth": 10, "bits": 64},
        # uneven batch, as in the benchmark's 256-circuit batch, with fewer circuits
        {"name": "dm_batch_16", "kind": "dm_batch", "count": 16, "n_min": 6, "n_max": 12, "depth_min": 10,
         "depth_max": 20},
        # the benchmark's 1024 trajectories over a quarter of its Trotter steps
        {"name": "traj_20q_1024", "kind": "traj", "n": 20, "ntraj": 1024, "steps": 10},
        # the benchmark's 24-qubit ansatz at half its layers
        {"name": "grad_24q", "kind": "grad", "n": 24, "layers": 20, "bits": 64},
        # the benchmark's 64 parameter sets of 20 qubits at a quarter of its layers
        {"name": "grad_batch_64x20q", "kind": "grad_batch", "n": 20, "layers": 10, "sets": 64},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["op", "sv", "sv", "sv", "pauli", "dm", "dm", "dm_batch", "traj", "grad", "grad_batch"])
    if kind == "op":
        return {"kind": kind, "n": rng.randint(4, 27), "k": rng.randint(1, 3), "bits": rng.choice([64, 128])}
    if kind == "sv":
        bits = rng.choice([64, 64, 128])
        return {"kind": kind, "n": rng.randint(5, 27 if bits == 64 else 25), "bits": bits,
                "depth": rng.randint(2, 20 if bits == 64 else 8), "start": rng.choice(["zero", "random"])}
    if kind == "pauli":
        return {"kind": kind, "n": rng.randint(6, 27), "bits": rng.choice([64, 128])}
    if kind == "dm":
        bits = rng.choice([64, 64, 128])
        return {"kind": kind, "n": rng.randint(3, 13 if bits == 64 else 10), "depth": rng.randint(2, 10), "bits": bits}
    if kind == "dm_batch":
        lo = rng.randint(4, 8)
        return {"kind": kind, "count": rng.randint(2, 16), "n_min": lo, "n_max": rng.randint(lo, 12), "depth_min": 4,
                "depth_max": rng.randint(5, 20)}
    if kind == "traj":
        n = rng.randint(8, 20)
        return {"kind": kind, "n": n, "ntraj": _log(rng, 16, 1024), "steps": rng.randint(2, 10)}
    if kind == "grad":
        return {"kind": kind, "n": rng.randint(8, 24), "layers": rng.randint(2, 20), "bits": rng.choice([64, 64, 128])}
    return {"kind": kind, "n": rng.randint(8, 20), "layers": rng.randint(2, 10), "sets": _log(rng, 2, 64)}


# ------------------------------------------------------------------ inputs

def _dtype(case):
    return torch.complex64 if case.get("bits", 64) == 64 else torch.complex128


def _haar(d, count, rng):
    """``count`` Haar unitaries: QR of complex Gaussian matrices, R's phases divided out."""
    z = rng.standard_normal((count, d, d)) + 1j * rng.standard_normal((count, d, d))
    q, r = np.linalg.qr(z)
    ph = np.einsum("gii->gi", r)
    return q * (ph / np.abs(ph))[:, None, :]


def _brickwork(n, depth, seed):
    """[(sites, matrix)]: per depth unit SU(2) on every site, SU(4) on even pairs, then on odd pairs."""
    rng = np.random.default_rng(seed)
    pairs = [(i, i + 1) for i in range(0, n - 1, 2)] + [(i, i + 1) for i in range(1, n - 1, 2)]
    out = []
    for _ in range(depth):
        out += [([q], m) for q, m in enumerate(_haar(2, n, rng))]
        out += [(list(p), m) for p, m in zip(pairs, _haar(4, len(pairs), rng))]
    return out


def _circuit(gates, n):
    return Circuit([Gate("rand_U", s, m) for s, m in gates], n=n)


def _noisy_circuit(gates, n):
    """The gates with a depolarising channel on both sites of every two-qubit gate,
    as the layer list ``workloads.noisy_brickwork_circuit`` builds."""
    dep = depolarizing(P_DEP)
    seq = []
    for s, m in gates:
        seq.append(Gate("rand_U", s, m))
        if len(s) == 2:
            seq += [ID(2, 0.0, [q], nm=dep) for q in s]
    c = _circuit(gates, n)
    c.layers = [[g] for g in seq]
    c.built = True
    return c


def _random_state(n, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(2 ** n, 2, generator=g, device=DEV, dtype=torch.float32 if dtype == torch.complex64 else torch.float64)
    x = torch.view_as_complex(x)
    return x / torch.linalg.vector_norm(x)


def _batch_specs(case, seed):
    rng = np.random.default_rng(seed)
    # sizes from the case alone, so that every seed costs the same; gates from the seed
    sizes = np.random.default_rng(case["count"] * 1000 + case["n_max"] * 10 + case["n_min"])
    ns = sizes.integers(case["n_min"], case["n_max"] + 1, case["count"])
    ds = sizes.integers(case["depth_min"], case["depth_max"] + 1, case["count"])
    return [(int(a), int(b), int(c)) for a, b, c in zip(ns, ds, rng.integers(0, 2 ** 31 - 1, case["count"]))]


def _params(case, seed, sets=1):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, 2 * np.pi, size=(sets, case["layers"], case["n"], 2))


def _op_inputs(case, seed):
    rng = np.random.default_rng(seed)
    sites = [int(q) for q in np.random.default_rng(case["n"] + case["k"]).permutation(case["n"])[:case["k"]]]
    return sites, _haar(2 ** case["k"], 1, rng)[0]


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    s = {"case": case}
    if kind == "op":
        sites, m = _op_inputs(case, seed)
        s["sites"] = sites
        s["op"] = torch.from_numpy(m).to(DEV, _dtype(case))
        s["psi"] = _random_state(n, _dtype(case), seed)
    elif kind == "sv":
        init = _random_state(n, _dtype(case), seed) if case["start"] == "random" else None
        s["sim"] = StatevectorSim(_circuit(_brickwork(n, case["depth"], seed), n), init_state=init,
                                  dtype=_dtype(case))
        s["sim"].compile()
    elif kind == "pauli":
        s["psi"] = _random_state(n, _dtype(case), seed)
        s["terms"] = TFI(n, jz=1.0, h=1.0).pauli_sum()
    elif kind == "dm":
        s["sim"] = DensityMatrixSim(_noisy_circuit(_brickwork(n, case["depth"], seed), n), dtype=_dtype(case))
        s["sim"].compile()
    elif kind == "dm_batch":
        sims = [DensityMatrixSim(_noisy_circuit(_brickwork(a, d, x), a)) for a, d, x in _batch_specs(case, seed)]
        s["batch"] = DensityMatrixBatch(sims)
    elif kind == "traj":
        circ = TFI(n, jz=1.0, h=1.0).trotter_circ(DT, case["steps"])
        s["sim"] = TrajectorySim(circ, case["ntraj"], p_dep=P_DEP, gamma=GAMMA, seed=seed)
        s["terms"] = z_terms(n)
    elif kind == "grad":
        s["params"] = torch.tensor(_params(case, seed)[0], dtype=torch.float64)
        s["terms"] = TFI(n, jz=1.0, h=1.0).pauli_sum()
    elif kind == "grad_batch":
        s["ansatz"] = BatchedAnsatz.hea(n, case["layers"])
        s["params"] = torch.from_numpy(_params(case, seed, case["sets"]).reshape(case["sets"], -1)).to(DEV)
        s["terms"] = TFI(n, jz=1.0, h=1.0).pauli_sum()
    else:
        raise ValueError(kind)
    return s


def run(s):
    case = s["case"]
    kind, n = case["kind"], case.get("n")
    if kind == "op":
        return tensorQ.op_action(s["op"], s["sites"], s["psi"])
    if kind in ("sv", "dm"):
        return s["sim"].run(progress_bar=False)
    if kind == "pauli":
        return pauli_expectations(s["psi"], n, s["terms"])
    if kind == "dm_batch":
        res = s["batch"].run().results()
        return {"trace": np.array([r["trace"] for r in res]), "purity": np.array([r["purity"] for r in res]),
                "z": np.concatenate([r["z"] for r in res]),
                "rho": [s["batch"].density_matrix(i) for i in range(len(res))]}
    if kind == "traj":
        states = s["sim"].run()
        return {"states": states, "expectations": s["sim"].expectations(s["terms"])}
    if kind == "grad":
        th = s["params"].clone().requires_grad_(True)
        sim = qg.StatevectorSim(workloads.hea_circuit(n, case["layers"], th), dtype=_dtype(case))
        e = adjoint_energy(sim, s["terms"])
        e.backward()
        return {"energy": e.detach(), "grad": th.grad}
    e, g = s["ansatz"].energy_and_grad(s["params"], s["terms"])
    return {"energy": e, "grad": g}


# -------------------------------------------------------------------- work

def _brick_counts(n, depth):
    return n * depth, (n - 1) * depth


def work(case):
    kind, n = case["kind"], case.get("n")
    amp = case.get("bits", 64) // 4 // 2  # bytes of one amplitude
    if kind == "op":
        return {"bytes": 2 * 2 ** n * amp + 4 ** case["k"] * amp, "flops": 8 * 2 ** (n + case["k"])}
    if kind == "sv":
        one, two = _brick_counts(n, case["depth"])
        reads = 2 ** n * amp if case["start"] == "random" else 0
        return {"bytes": 2 ** n * amp + reads + (4 * one + 16 * two) * 16, "flops": 2 ** n * (16 * one + 32 * two)}
    if kind == "pauli":
        return {"bytes": 2 ** n * amp + 8 * (2 * n - 1), "flops": 2 ** n * (3 * (n - 1) + 4 * n)}
    if kind in ("dm", "dm_batch"):
        circs = [(n, case["depth"])] if kind == "dm" else [(a, d) for a, d, _ in _batch_specs(case, 0)]
        out = {"bytes": 0, "flops": 0}
        for a, d in circs:
            one, two = _brick_counts(a, d)
            out["bytes"] += 4 ** a * amp + (4 * one + 16 * two) * 16
            # a gate on the ket and the bra side; two channels of four Kraus products on 2 bits each per pair
            out["flops"] += 4 ** a * (2 * 16 * one + 2 * 32 * two + 2 * two * 32)
        return out
    if kind == "traj":
        one, two = n * case["steps"], (n - 1) * case["steps"]
        amps = case["ntraj"] * 2 ** n
        # RX products, ZZ phases, the damping factor of every touched site; the states written once
        return {"bytes": amps * 8 + case["ntraj"] * (2 * n - 1) * 8, "flops": amps * (16 * one + 6 * two + 2 * (one + 2 * two))}
    sets = case.get("sets", 1)
    amps = sets * 2 ** n
    rot = 2 * n * case["layers"]
    # forward products, the same backwards on state and co-state, and one derivative per rotation; the ladder only permutes
    return {"bytes": sets * rot * 16 + 8 * sets, "flops": amps * rot * (3 * 10 + 4)}


# ---------------------------------------------------- the same in 64 bits

def _apply(x, m, sites, n):
    """``m`` on one or two ``sites`` of ``x`` (..., 2^n) by a plain matrix product, complex128."""
    m = torch.as_tensor(m, dtype=torch.complex128, device=x.device)
    k = len(sites)
    order = sorted(range(k), key=lambda j: sites[j])
    if order != list(range(k)):  # rows and columns re-ordered to ascending sites
        m = m.reshape([2] * (2 * k)).permute(order + [k + j for j in order]).reshape(2 ** k, 2 ** k)
    sites = sorted(sites)
    lead = x.numel() // 2 ** n
    dims, prev = [lead], -1
    for q in sites:
        dims += [2 ** (q - prev - 1), 2]
        prev = q
    dims.append(2 ** (n - 1 - prev))
    axes = [2 + 2 * j for j in range(k)]
    rest = [a for a in range(len(dims)) if a not in axes]
    y = x.reshape(dims).permute(axes + rest)
    shape = y.shape
    y = (m @ y.reshape(2 ** k, -1)).reshape(shape)
    back = np.argsort(axes + rest).tolist()
    return y.permute(back).reshape(x.shape)


def _merge(gates):
    """Single-qubit gates folded into the next two-qubit gate of their site (fewer passes, same product)."""
    wait, out = {}, []
    for s, m in gates:
        if len(s) == 1:
            wait[s[0]] = m @ wait[s[0]] if s[0] in wait else m
        else:
            eye = np.eye(2)
            out.append((s, m @ np.kron(wait.pop(s[0], eye), wait.pop(s[1], eye))))
    return out + [([q], m) for q, m in wait.items()]


def _basis(n):
    x = torch.zeros(2 ** n, dtype=torch.complex128, device=DEV)
    x[0] = 1
    return x


def _exact_dm(n, depth, seed):
    x = _basis(2 * n)
    kr = [np.sqrt(1 - P_DEP) * np.eye(2)] + [np.sqrt(P_DEP / 3) * np.array(p) for p in
                                            ([[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]])]
    channel = sum(np.kron(a, np.conj(a)) for a in kr)  # (ket, bra)
    for s, m in _merge(_brickwork(n, depth, seed)):
        x = _apply(x, m, s, 2 * n)
        x = _apply(x, np.conj(m), [n + q for q in s], 2 * n)
        if len(s) == 2:
            for q in s:
                x = _apply(x, channel, [q, n + q], 2 * n)
    return x


def _flip(x, n, q):
    """X on site q: the two halves exchanged."""
    v = x.reshape(-1, 2 ** q, 2, 2 ** (n - 1 - q))
    return v.flip(2).reshape(x.shape)


def _sign(x, n, q):
    """Z on site q."""
    v = x.reshape(-1, 2 ** q, 2, 2 ** (n - 1 - q)).clone()
    v[:, :, 1] *= -1
    return v.reshape(x.shape)


def _cnot(x, n, control, target):
    """Adjacent control and target = control + 1."""
    v = x.reshape(-1, 2 ** control, 2, 2, 2 ** (n - 2 - control)).clone()
    v[:, :, 1] = v[:, :, 1].flip(2)
    return v.reshape(x.shape)


def _turn(x, n, q, kind, th):
    """exp(-i th P) on site q, one angle per leading row; P = Y or Z."""
    v = x.reshape(th.numel(), 2 ** q, 2, 2 ** (n - 1 - q))
    c, s = torch.cos(th).view(-1, 1, 1), torch.sin(th).view(-1, 1, 1)
    a, b = v[:, :, 0], v[:, :, 1]
    if kind == "y":
        out = torch.stack([c * a - s * b, s * a + c * b], dim=2)
    else:
        ph = torch.complex(c, -s)
        out = torch.stack([ph * a, ph.conj() * b], dim=2)
    return out.reshape(x.shape)


def _exact_grad(n, params):
    """Energies and angle gradients of the ansatz: forward, H psi, then gate by gate backwards."""
    th = torch.as_tensor(params, dtype=torch.float64, device=DEV)
    sets, layers = th.shape[0], th.shape[1]
    x = torch.zeros(sets, 2 ** n, dtype=torch.complex128, device=DEV)
    x[:, 0] = 1
    for l in range(layers):
        for q in range(n):
            x = _turn(x, n, q, "y", th[:, l, q, 0])
            x = _turn(x, n, q, "z", th[:, l, q, 1])
        for q in range(n - 1):
            x = _cnot(x, n, q, q + 1)
    lam = torch.zeros_like(x)
    for q in range(n):
        lam += _flip(x, n, q)
        if q < n - 1:
            lam += _sign(_sign(x, n, q), n, q + 1)
    energy = (lam.conj() * x).sum(dim=1).real
    grad = torch.zeros(sets, layers, n, 2, dtype=torch.float64, device=DEV)
    for l in reversed(range(layers)):
        for q in reversed(range(n - 1)):
            x, lam = _cnot(x, n, q, q + 1), _cnot(lam, n, q, q + 1)
        for q in reversed(range(n)):
            for j, kind in ((1, "z"), (0, "y")):
                u = x.reshape(sets, -1, 2, 2 ** (n - 1 - q))
                w = lam.reshape(u.shape)
                if kind == "z":
                    ip = (w[:, :, 0].conj() * u[:, :, 0]).sum((1, 2)) - (w[:, :, 1].conj() * u[:, :, 1]).sum((1, 2))
                    g = 2 * ip.imag
                else:  # <w| Y |u> = -i w0* u1 + i w1* u0
                    ip = (w[:, :, 1].conj() * u[:, :, 0]).sum((1, 2)) - (w[:, :, 0].conj() * u[:, :, 1]).sum((1, 2))
                    g = 2 * ip.real
                grad[:, l, q, j] = g
                x = _turn(x, n, q, kind, -th[:, l, q, j])
                lam = _turn(lam, n, q, kind, -th[:, l, q, j])
    return energy, grad


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "op":
        sites, m = _op_inputs(case, seed)
        m = m.astype(np.complex64).astype(np.complex128) if case["bits"] == 64 else m
        x = _random_state(n, _dtype(case), seed).to(torch.complex128)
        if case["k"] <= 2:
            return _apply(x, m, sites, n)
        y = torch.tensordot(torch.from_numpy(m).to(DEV).reshape([2] * 6), x.reshape([2] * n), dims=([3, 4, 5], sites))
        return torch.movedim(y, [0, 1, 2], sites).reshape(-1)
    if kind == "sv":
        x = _random_state(n, _dtype(case), seed).to(torch.complex128) if case["start"] == "random" else _basis(n)
        for s, m in _merge(_brickwork(n, case["depth"], seed)):
            x = _apply(x, m, s, n)
        return x.reshape([2] * n)
    if kind == "pauli":
        x = _random_state(n, _dtype(case), seed).to(torch.complex128)
        p = x.real ** 2 + x.imag ** 2
        zz, xs = [], []
        for q in range(n - 1):
            v = p.reshape(2 ** q, 2, 2, -1).sum((0, 3))
            zz.append(v[0, 0] + v[1, 1] - v[0, 1] - v[1, 0])
        for q in range(n):
            v = x.reshape(2 ** q, 2, -1)
            xs.append(2 * (v[:, 0].conj() * v[:, 1]).sum().real)
        return torch.stack(zz + xs)
    if kind == "dm":
        return _exact_dm(n, case["depth"], seed)
    if kind == "dm_batch":
        rho = [_exact_dm(a, d, x).reshape(2 ** a, 2 ** a) for a, d, x in _batch_specs(case, seed)]
        z = []
        for r in rho:
            a = int(r.shape[0]).bit_length() - 1
            d = r.diagonal().real
            z += [(v[:, 0] - v[:, 1]).sum().item() for v in (d.reshape(2 ** q, 2, -1) for q in range(a))]
        return {"trace": np.array([r.diagonal().sum().real.item() for r in rho]),
                "purity": np.array([(r.abs() ** 2).sum().item() for r in rho]), "z": np.array(z), "rho": rho}
    if kind == "traj":  # drawn from the library's own random stream
        return None
    energy, grad = _exact_grad(n, _params(case, seed, case.get("sets", 1)))
    if kind == "grad":
        return {"energy": energy[0], "grad": grad[0].cpu()}
    return {"energy": energy, "grad": grad.reshape(case["sets"], -1)}

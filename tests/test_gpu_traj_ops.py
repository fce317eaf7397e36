"""Every kind of op of the persistent trajectory kernel (general, x rotation, real
and diagonal one-site ops, diagonal and general two-site ops) on every pair of
positions of a register group, with runs long enough that the lanes' weights are
summed several times, with and without damping and replayed jumps, for groups of
1 to 4 bits and tiles of fewer groups than threads up to several groups a thread.

Tolerance: an op rounds each component at most 8 times (products, sums, K0,
prescale), so after N ops the error is below 8 N u with u the unit roundoff of
the dtype; the oracle's own rounding is added to it for complex128."""
import numpy as np
import pytest
import torch

from test_trajectories import _replay_jumps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _gates(n, rng):
    from qaravan_gb300 import workloads
    from qaravan_gb300.gates import Gate
    th = rng.uniform(0.2, 1.2, 8)
    c, s = np.cos, np.sin
    one = [lambda: workloads.haar_unitary(2, rng),
           lambda: np.array([[c(th[0]), -1j * s(th[0])], [-1j * s(th[0]), c(th[0])]]),
           lambda: np.array([[c(th[1]), -s(th[1])], [s(th[1]), c(th[1])]]),
           lambda: np.array([[1, 1], [1, -1]]) / np.sqrt(2),
           lambda: np.diag([1, np.exp(1j * th[2])])]
    two = [lambda: np.diag(np.exp(1j * rng.uniform(0, 6, 4))), lambda: workloads.haar_unitary(4, rng)]
    out = []
    sites = [int(q) for q in rng.permutation(n)]
    for i in range(0, n, 4):  # groups of four sites: all kinds, all ordered pairs
        grp = sites[i:i + 4]
        for j, q in enumerate(grp):
            out += [Gate("U", [q], one[(j + k) % 5]()) for k in range(3)]
        for a in grp:
            for b in grp:
                if a != b:
                    out.append(Gate("U", [a, b], two[(a + b + i) % 2]()))
                    out.append(Gate("U", [b], one[(a + 2 * b) % 5]()))
    return out


@pytest.mark.parametrize("dtype,n,tile", [(torch.complex64, 1, 13), (torch.complex64, 2, 13), (torch.complex64, 3, 13),
                                          (torch.complex64, 4, 13), (torch.complex64, 9, 13), (torch.complex64, 13, 13),
                                          (torch.complex64, 13, 10), (torch.complex64, 14, 14),
                                          (torch.complex128, 3, 12), (torch.complex128, 12, 12),
                                          (torch.complex128, 13, 13)])
@pytest.mark.parametrize("p,gamma", [(0.2, 0.08), (0.0, 0.02), (0.2, 0.0)])
def test_kinds_against_oracle(dtype, n, tile, p, gamma):
    from qaravan_gb300.circuits import Circuit
    from qaravan_gb300.trajectories import TrajectorySim
    T, seed = 3, 5
    gates = _gates(n, np.random.default_rng(n))
    sim = TrajectorySim(Circuit(gates, n=n), T, p_dep=p, gamma=gamma, seed=seed, dtype=dtype, log=True, tile_bits=tile)
    assert sim.mode == "persistent"
    states = sim.run().cpu().numpy().reshape(T, -1)
    tol = 8 * len(gates) * (2.0 ** -24 if dtype == torch.complex64 else 2.0 ** -53 * 2)
    for t in range(T):
        exp = _replay_jumps(sim.gates, n, t, seed, p, gamma, sim.jumps(t) if gamma > 0 else [])
        assert np.max(np.abs(states[t] - exp)) < tol

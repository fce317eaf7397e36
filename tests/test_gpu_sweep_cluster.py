"""Tile sweeps over thread-block clusters (csrc/sweep_cluster.cu) against the
one-CTA-per-tile kernels: the same rows summed in the same order, so one state
(few tiles: clusters) equals, bit for bit, the first of 160 copies (tiles for
every SM: the general kernels), whose last copy equals it too. Sizes: parts of
less than a warp, one thread per amplitude, several rows per thread, 1 to 16
CTAs per tile, one to 32 tiles; ops inside a part, across parts, on all rank
bits; more ops than a sweep and more matrices than a staged chunk hold.
"""
import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def _gates(n, width, count, rng):
    """Random dense gates on random sites (any order, any distance)."""
    from qaravan_gb300.gates import Gate
    from qaravan_gb300.workloads import haar_unitary
    out = []
    for _ in range(count):
        k = int(rng.integers(1, min(width, n) + 1))
        sites = [int(q) for q in rng.permutation(n)[:k]]
        out.append(Gate("g", sites, haar_unitary(2 ** k, rng)))
    return out


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,width,tile,low", [(1, 1, 13, None), (3, 3, 13, None), (5, 4, 13, None), (7, 2, 13, None),
                                              (8, 3, 13, None), (10, 4, 13, None), (11, 3, 13, None),
                                              (13, 4, 13, None), (14, 3, 12, 2), (15, 4, 13, 5), (17, 3, 13, None),
                                              (18, 2, 13, 3), (9, 5, 13, None)])
def test_clusters_equal_the_general_kernels(n, width, tile, low, dtype):
    from qaravan_gb300 import compiler
    from qaravan_gb300.engine import Executor
    from qaravan_gb300.statevector import gates_to_ops
    if dtype == torch.complex128:
        width = min(width, 4)
    rng = np.random.default_rng(1000 * n + width)
    gates = _gates(n, width, 90 if n < 14 else 40, rng)
    plan = compiler.compile_ops(gates_to_ops(gates, n), n, mode="sweep", width=width, tile_bits=tile, low_bits=low,
                                max_sweep_k=5 if dtype == torch.complex64 else 4,
                                itemsize=8 if dtype == torch.complex64 else 16)
    assert all(isinstance(s, compiler.SweepStep) for s in plan.steps)
    ex = Executor(plan, dtype, "cuda")
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    v /= np.linalg.norm(v)
    one = torch.from_numpy(v).to("cuda", dtype)
    many = one.repeat(160)
    ex.run(one)
    ex.run(many, batch=160, stride=2 ** n)
    many = many.reshape(160, -1)
    assert torch.equal(many[0], one) and torch.equal(many[159], one)
    exp = ref.run_sv(gates, n, v)
    assert np.max(np.abs(one.cpu().numpy() - exp)) < (1e-5 if dtype == torch.complex64 else 1e-12)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_batches_with_their_own_matrices(dtype):
    """Five states with different matrices in one launch of clusters, against each alone."""
    from qaravan_gb300 import compiler
    from qaravan_gb300.engine import Executor
    from qaravan_gb300.statevector import gates_to_ops
    n, batch, rng = 10, 5, np.random.default_rng(7)
    sets = [_gates(n, 3, 12, np.random.default_rng(5)) for _ in range(batch)]
    for g in sets:  # the same sites, other matrices
        for x in g:
            x.matrix = x.matrix @ np.diag(np.exp(2j * np.pi * rng.random(x.matrix.shape[0])))
    isz = 8 if dtype == torch.complex64 else 16
    exs = [Executor(compiler.compile_ops(gates_to_ops(g, n), n, mode="sweep", width=3, tile_bits=13, itemsize=isz),
                    dtype, "cuda") for g in sets]
    v = rng.standard_normal((batch, 2 ** n)) + 1j * rng.standard_normal((batch, 2 ** n))
    st = torch.from_numpy(v).to("cuda", dtype)
    want = st.clone()
    for i, ex in enumerate(exs):
        ex.run(want[i])
    stride = (exs[0].mats.numel() + 1) // 2 * 2
    mats = torch.zeros(batch, stride, dtype=dtype, device="cuda")
    for i, ex in enumerate(exs):
        mats[i, :ex.mats.numel()] = ex.mats
    exs[0].run(st, batch=batch, stride=2 ** n, mats=mats, mat_stride=stride)
    assert torch.equal(st, want)

"""The norm chain of a plan run in one call, whose first epoch is cut so that the last
pass opens one: chains of 1 to 14 links (every length of the first epoch, up to three
whole ones) end with a norm within the drift of the passes that no later link corrects.

The last pass corrects all before it (lengths of 1 + 4 k links, and with the shorter first
epoch all others): its own loss (round-toward-zero sums, 1e-7 to 2e-7) and the squares' float32
rounding remain, 3e-7.
"""
import numpy as np
import pytest
import torch

from qaravan_gb300 import _lib, workloads
from qaravan_gb300.compiler import DenseStep, Plan
from qaravan_gb300.engine import Executor

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built(cuda_ok):
    from qaravan_gb300 import build
    build.build()


def test_epoch_of_the_library():
    assert _lib.lib().qgb_chain_epoch() == 4


@pytest.mark.parametrize("links", range(1, 15))
def test_norm_after_a_chain(links):
    n, rng = 16, np.random.default_rng(links)
    plan = Plan(nbits=n)
    for _ in range(links):
        bits = sorted((int(b) for b in rng.permutation(n)[:6]), reverse=True)
        plan.steps.append(DenseStep(bits, plan.add_matrix(workloads.haar_unitary(64, rng)), True))
    ex = Executor(plan, torch.complex64)
    v = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    state = torch.from_numpy(v / np.linalg.norm(v)).to("cuda", torch.complex64)

    def norm(x):
        return float(torch.linalg.vector_norm(x.to(torch.complex128)))

    start = norm(state)
    ex.run(state)
    assert abs(norm(state) / start - 1) < 3e-7

"""Which mode a complex128 simulator settles on when fixed-point blocks are asked
for, chosen by default or remembered by the autotuner."""
import pytest
import torch

from qaravan_gb300 import _lib, autotune, workloads
from qaravan_gb300.statevector import StatevectorSim


@pytest.fixture(autouse=True)
def built(tmp_path, monkeypatch):
    from qaravan_gb300 import build
    build.build()
    monkeypatch.setenv("QGB_AUTOTUNE_CACHE", str(tmp_path / "autotune.json"))
    monkeypatch.delenv("QGB_AUTOTUNE", raising=False)


def _sim(n=17, **kw):
    sim = StatevectorSim(workloads.brickwork_circuit(n, 1, 5), dtype=torch.complex128, **kw)
    return sim.mode, sim.fusion_width


@pytest.mark.parametrize("width,want", [(None, ("fixed", 5)), (5, ("fixed", 5)), (4, ("sweep", 4)), (3, ("sweep", 3))])
def test_width_asked_for(width, want):
    assert _sim(mode="fixed", fusion_width=width) == want
    assert _sim(fusion_width=width) == want

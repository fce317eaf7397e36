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


@pytest.mark.parametrize("switch", ["arithmetic", "tensor cores"])
def test_blocks_switched_off(switch):
    """A remembered choice, the default and the mode by name: sweeps, not 5-qubit float64 blocks."""
    L = _lib.lib()
    autotune.store("sv", 17, torch.complex128, ("fixed", 5, 13), [])
    assert _sim() == ("fixed", 5)
    impl = L.qgb_get_dense_impl()
    _lib.check(L.qgb_set_c128_arith(0) if switch == "arithmetic" else L.qgb_set_dense_impl(0))
    try:
        assert autotune.choose_sv(17, torch.complex128) == ("sweep", 3, 13)
        assert _sim() == _sim(mode="fixed") == _sim(18) == ("sweep", 3)
    finally:
        _lib.check(L.qgb_set_c128_arith(1))
        _lib.check(L.qgb_set_dense_impl(impl))
    assert _sim() == ("fixed", 5)

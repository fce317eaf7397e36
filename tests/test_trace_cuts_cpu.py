"""Where the trace chain of density matrices measures (engine.trace_cuts): at
whole-channel cuts, at least four tensor-core passes apart, and, of the four ways
to begin, the one that leaves the end closest to two passes behind the last."""
import numpy as np
import pytest

from qaravan_gb300.engine import _TRACE_EPOCH, _TRACE_TAIL, trace_cuts


def _steps(spec):
    """w / W: a tensor-core pass, open / whole; c / C: a CUDA-core block; n: renormalisation; s: a sweep."""
    kind = {"n": ("normalize",), "s": ("sweep", None)}
    return [kind.get(x) or ("dense", None, 6, 0, True, x.isupper(), x in "wW", False) for x in spec]


def _behind(spec, cut):
    """Tensor-core passes behind a cut, up to the next renormalisation."""
    return sum(x in "wW" for x in spec[cut + 1:].split("n")[0])


@pytest.mark.parametrize("count", range(1, 40))
def test_all_whole(count):
    cuts = sorted(trace_cuts(_steps("W" * count)))
    assert all(b - a >= _TRACE_EPOCH for a, b in zip(cuts, cuts[1:]))
    if count <= _TRACE_EPOCH:
        assert not cuts
    elif count >= _TRACE_EPOCH + _TRACE_TAIL:
        assert _TRACE_EPOCH <= cuts[0] + 1 < 2 * _TRACE_EPOCH and count - 1 - cuts[-1] == _TRACE_TAIL
        assert all(b - a == _TRACE_EPOCH for a, b in zip(cuts, cuts[1:]))
    else:
        assert cuts == [_TRACE_EPOCH - 1]


@pytest.mark.parametrize("spec,want", [("wwCwwWwCnW", [5]), ("WWWWWWnWWWWWW", [3, 10]), ("wwwwwwww", []), ("WWWWC", []),
                                       ("WWWWCw", [3]), ("WWwWcWsWW", [5]), ("", []), ("CCCC", []), ("nn", [])])
def test_cuts(spec, want):
    assert sorted(trace_cuts(_steps(spec))) == want


@pytest.mark.parametrize("seed", range(30))
def test_random_plans(seed):
    rng = np.random.default_rng(seed)
    spec = "".join(rng.choice(list("wWWWcCns"), size=60, p=[0.2, 0.2, 0.2, 0.2, 0.05, 0.05, 0.05, 0.05]))
    cuts = trace_cuts(_steps(spec))
    for c in cuts:
        assert spec[c].isupper() and _behind(spec, c) >= 1
    begin = 0
    for part in spec.split("n"):
        mine = sorted(c - begin for c in cuts if begin <= c < begin + len(part))
        tc = [i for i, x in enumerate(part) if x in "wW"]
        marks = [sum(t <= c for t in tc) for c in mine]
        assert all(b - a >= _TRACE_EPOCH for a, b in zip([0] + marks, marks))
        begin += len(part) + 1

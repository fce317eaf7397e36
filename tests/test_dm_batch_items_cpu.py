"""Items of the persistent density-matrix batch (host code): every pass's tiles are
dealt exactly once, a round is one wave of items unless that takes items of more
than 32 tiles and more than one wave of the pass alone, no item is smaller than 8
tiles unless its pass is, and an item waits for exactly the items of its circuit's
earlier passes."""
import numpy as np
import pytest

ITEM = np.dtype([("pass", "<i4"), ("need", "<u4"), ("t0", "<u4"), ("ntiles", "<u4"), ("tstride", "<u4"),
                 ("last_items", "<i4"), ("last0", "<i8")])


@pytest.fixture(scope="module")
def lib():
    from qaravan_gb300 import _lib, build
    build.build()
    return _lib.lib()


@pytest.mark.parametrize("circuits", [[(7, 1)], [(8, 3), (14, 2)], [(9, 4), (8, 6), (8, 1)], [(12, 5), (11, 7), (11, 6), (10, 2)],
                                      [(8, 9)] * 20, [(13, 3), (7, 8)]])
@pytest.mark.parametrize("sms", [1, 4, 152])
def test_items(lib, circuits, sms):
    from qaravan_gb300.batch import _DMB_CIRC, _DMB_PASS
    npass = sum(k for _, k in circuits)
    c, p = np.zeros(len(circuits), dtype=_DMB_CIRC), np.zeros(npass, dtype=_DMB_PASS)
    first = 0
    for i, (n, k) in enumerate(circuits):
        c[i] = (4096, n, first, k, i)
        for j in range(k):
            p[first + j]["mat"], p[first + j]["circ"], p[first + j]["tslot"] = 8192, i, -1
            p[first + j]["bits"] = [0, 1, 2, 3, 4, 5]
            p[first + j]["flags"] = (8 if j == 0 else 0) | (4 if j == k - 1 else 0)
        first += k
    total = lib.qgb_dm_batch_items(c.ctypes.data, len(c), sms)
    nbytes = lib.qgb_dm_batch_table_bytes(len(c), npass, total)
    buf = np.zeros(nbytes, dtype=np.uint8)
    assert lib.qgb_dm_batch_build(buf.ctypes.data, nbytes, c.ctypes.data, len(c), p.ctypes.data, npass, sms) == 0
    off = nbytes - (total * ITEM.itemsize + 255) // 256 * 256
    items = buf[off:off + total * ITEM.itemsize].view(ITEM)
    work, fin = items[items["ntiles"] > 0], items[items["ntiles"] == 0]
    assert len(fin) == len(circuits)
    rounds = {}
    for i, (n, k) in enumerate(circuits):
        tiles, before = 2 ** (2 * n - 13), 0
        for j in range(k):
            mine = work[work["pass"] == c[i]["first_pass"] + j]
            got = np.concatenate([x["t0"] + x["tstride"] * np.arange(x["ntiles"]) for x in mine])
            assert np.array_equal(np.sort(got), np.arange(tiles))
            assert np.all(mine["need"] == before)
            assert len(mine) == 1 or mine["ntiles"].max() >= 8
            most = max(32, -(-tiles // sms))
            assert mine["ntiles"].max() <= most
            rounds.setdefault(j, []).append((len(mine), mine["ntiles"].max() == most or len(mine) == -(-tiles // most)))
            before += len(mine)
        assert fin[i]["need"] == before and fin[i]["last_items"] == len(mine)
    for r, counts in rounds.items():  # a wave: at most one item a pass beyond the SMs (the rounding up)
        assert sum(k for k, _ in counts) <= sms + len(counts) or any(capped for _, capped in counts)

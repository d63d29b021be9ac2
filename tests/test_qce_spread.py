"""The spread layout of the edge-buffer decoder (slots of short columns moved to
their row's CTA): the row side and the column side name the same place for
every edge slot, no two slots share a place, all places lie in the CTA's shared
memory, every other descriptor is the unspread layout's."""
import numpy as np
import pytest

from atsc3_b200 import codes as C
from atsc3_b200 import native as N
from test_qce_tables import SLOT, qce_tables, zones

SMAX = 232448


@pytest.mark.parametrize("rate,n,cluster", [
    ("6/15", 64800, 6), ("10/15", 64800, 6), ("13/15", 64800, 14), ("8/15", 64800, 9),
    ("8/15", 16200, 3), ("11/15", 16200, 14), ("6/15", 16200, 6), ("11/15", 16200, 2),
    ("7/15", 64800, 7), ("2/15", 16200, 3)])
def test_spread_slots(rate, n, cluster):
    K, QA, QB = zones(rate, n)
    rowptr, addr = [np.ascontiguousarray(a, np.int32) for a in C.address_rows(rate, n)]
    meta = np.zeros(64, np.int32)
    args = [n, K, QA, QB, rowptr.ctypes.data, addr.ctypes.data, cluster, SMAX]
    N.call("atsc3_ldpc_qce_spread_host", *args, meta.ctypes.data, None, None, None)
    rdesc = np.zeros((meta[0], 4), np.int32)
    itab = np.zeros((meta[1], 4), np.int32)
    xtab = np.zeros(max(1, meta[2]), np.uint32)
    N.call("atsc3_ldpc_qce_spread_host", *args, meta.ctypes.data, rdesc.ctypes.data,
           itab.ctypes.data, xtab.ctypes.data)
    smem, buf, xt, slots = (int(v) for v in meta[3:7])
    xb, ib = meta[7:7 + cluster + 1], meta[24:24 + cluster + 1]
    _, _, _, pm, prd, rptr, cdesc, ccols, _, _, pit, _ = qce_tables(rate, n, cluster)
    assert smem <= SMAX and smem == buf + slots * SLOT
    if cluster < 3 or meta[2] == 0:
        assert np.array_equal(rdesc, prd)
        return
    assert xt + 4 * int(np.diff(xb).max()) <= buf
    grow = buf - int(pm[7])
    # unspread place of every slot -> (column, index)
    slot_of = {(int(cdesc[g, 3]) & 0xFF, int(cdesc[g, 1]) + i * SLOT): (g, i)
               for g in range(n // 360) for i in range(cdesc[g, 0])}
    place = {}
    for old, new in zip(prd, rdesc):
        g, i = slot_of[(int(old[0]) & 0xFF, int(old[1]))]
        assert (new[0] & ~0xFF) == (old[0] & ~0xFF) and np.array_equal(new[2:], old[2:])
        place[(g, i)] = (int(new[0]) & 0xFF, int(new[1]))
    assert len(set(place.values())) == len(place)      # one place per slot
    assert all(c < cluster and buf <= o <= smem - SLOT and (o - buf) % SLOT == 0
               for c, o in place.values())
    # column side: the same places, every item of the unspread list once
    moved = 0
    for c in range(cluster):
        for x, y, z, w in itab[ib[c]:ib[c + 1]]:
            g, mm = divmod(int(y), 360)
            own = int(cdesc[g, 3]) & 0xFF
            assert own == c
            for i in range(z & 0xFF):
                if z & (1 << 27):
                    assert (x >> 16) == mm
                    v = int(xtab[xb[c] + (x & 0xFFFF) + i])
                    got = (v >> 20, v & 0xFFFFF)
                    moved += got[0] != c
                else:
                    got = (c, int(x) - 4 * mm + i * SLOT)
                assert got == place[(g, i)]
                if not z & (1 << 27):
                    assert got == (own, int(cdesc[g, 1]) + i * SLOT + grow)
    assert moved > 0
    key = lambda t: sorted((int(y), int(z) & ~(1 << 27), int(w)) for _, y, z, w in t)
    assert key(itab) == key(pit)

"""The phase correction's float32 screen: decisions of cells at the points,
on the boundaries between two of them and far out equal the float64 hypot's
first minimum, for mirrored, unmirrored and tiny alphabets and for symbol
counts that take one CTA or a cluster each; results agree with the oracle."""
import numpy as np
import pytest

import oracle
from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu


def _pool(mods, nsym, per, seed):
    rng = np.random.default_rng(seed)
    al = []
    for m in mods:
        p = np.array(C.alphabet(m.rstrip("*"), "9/15"), np.complex128)
        if m.endswith("*"):
            p[1] *= 1.01                     # no mirror images any more
        al.append(p)
    n = nsym * per
    region = rng.choice(np.array([0, 0, 1, 2, 3], np.uint8), n)
    x = np.zeros(n, np.complex128)
    for r, p in enumerate(al):
        a, b = p[rng.integers(0, len(p), (2, n))]
        kind = rng.integers(0, 4, n)
        v = np.select([kind == 0, kind == 1, kind == 2], [a, (a + b) / 2, a.real + 0j],
                      a + 0.02 * (rng.standard_normal(n) + 1j * rng.standard_normal(n)))
        x[region == r] = v[region == r]
    x[region == 3] = 0.5
    dummy = np.where(rng.random(n) < 0.5, 1.0, -1.0).astype(np.complex128)
    x[region == 2] = dummy[region == 2]
    if len(al) == 1:
        region[region == 1] = 0
    return x, np.repeat(np.arange(nsym), per), al, region, dummy


@pytest.mark.parametrize("mods,nsym,per", [
    (("QPSK", "16QAM"), 1, 1), (("16QAM", "64QAM"), 3, 257), (("256QAM", "64QAM*"), 2, 4099),
    (("256QAM*",), 1, 9000), (("4096QAM", "1024QAM"), 1, 600), (("64QAM", "QPSK"), 700, 9)])
def test_cpe_screen_vs_oracle(mods, nsym, per):
    from atsc3_b200.cpe import cpe_correct
    pool, sym, al, region, dummy = _pool(mods, nsym, per, nsym + per)
    for iters in (0, 1, 3):
        r = region.copy()
        # the oracle has no fourth region: it takes those cells as known zeros
        d = np.where(r == 3, 0, dummy)
        want, wg = oracle.cpe_correct(pool, sym, al, np.where(r == 3, 2, r), d, iters=iters)
        got, gg = cpe_correct(pool, sym, al, r, dummy, iters=iters)
        # a symbol without a known or decided cell has no gain: 0 / 0 on both sides
        ok = np.isfinite(want)
        assert np.array_equal(ok, np.isfinite(got))
        if ok.any():
            assert np.max(np.abs(got - want)[ok]) <= 1e-12 * np.max(np.abs(want[ok]))
        for s in wg:
            assert (abs(gg[s] - wg[s]) <= 1e-12 * abs(wg[s]) if np.isfinite(wg[s])
                    else not np.isfinite(gg[s]))

"""Phase correction over alphabet sizes around 48 KB of tables a CTA (4096
points): every size corrects, as the oracle does."""
import numpy as np
import pytest

import oracle
from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m0,m1", [(4096, 0), (4080, 16), (4081, 0), (4064, 0), (4096, 8)])
def test_cpe_alphabet_sizes(m0, m1):
    from atsc3_b200.cpe import cpe_correct
    big = np.array(C.alphabet("4096QAM", "9/15"), np.complex128)
    small = np.array(C.alphabet("16QAM", "9/15"), np.complex128)
    al = [big[:m0]] + ([small[:m1]] if m1 else [])
    rng = np.random.default_rng(m0 + m1)
    n = 900
    region = rng.integers(0, 2 if m1 else 1, n).astype(np.uint8)
    pool = np.where(region == 0, al[0][rng.integers(0, m0, n)],
                    al[-1][rng.integers(0, len(al[-1]), n)])
    pool = pool * np.exp(0.002j) + 1e-3 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    sym = np.repeat(np.arange(3), n // 3)
    dummy = np.zeros(n, np.complex128)
    want, wg = oracle.cpe_correct(pool, sym, al, region, dummy, iters=2)
    got, gg = cpe_correct(pool, sym, al, region, dummy, iters=2)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    for s in wg:
        assert abs(gg[s] - wg[s]) <= 1e-12 * abs(wg[s])

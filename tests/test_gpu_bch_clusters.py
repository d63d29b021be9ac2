"""The BCH check over cluster sizes and ragged lengths: message lengths that are
not whole 32-bit words, batches that take eight CTAs a codeword, fewer and one,
syndrome words, flag and payload against the oracle."""
import numpy as np
import pytest

import oracle
from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,n,nblk", [
    ("2/15", 16200, 3), ("11/15", 16200, 149), ("6/15", 16200, 1200), ("13/15", 64800, 2)])
def test_bch_check_clusters(rate, n, nblk):
    import torch
    from atsc3_b200 import bch as B
    K, kp = C.kldpc(rate, n), C.kpayload(rate, n)
    rng = np.random.default_rng(nblk)
    msg = oracle.bch_encode(rng.integers(0, 2, (3, kp)).astype(np.uint8), n)
    bits = msg[np.arange(nblk) % 3].copy()
    hit = rng.random(nblk) < 0.5
    bits[hit, rng.integers(0, K, hit.sum())] ^= 1
    width = (n + 31) // 32 * 4
    packed = np.packbits(np.pad(bits, ((0, 0), (0, width * 8 - K))), axis=1)
    o = B.bch_check(torch.from_numpy(packed).cuda(), K, n, kp)
    syn = B.syndromes_to_ints(o["syn"].cpu().numpy())
    pick = rng.choice(nblk, min(nblk, 12), replace=False)
    assert [syn[i] for i in pick] == list(oracle.bch_syndrome(bits[pick], n))
    assert np.array_equal(o["ok"].cpu().numpy(), [int(s == 0) for s in syn])
    assert np.array_equal(o["ok"].cpu().numpy() == 0, hit)
    want = np.packbits(bits[:, :kp] ^ C.scrambler_sequence(kp)[None], axis=1)
    assert np.array_equal(o["payload"].cpu().numpy(), want)

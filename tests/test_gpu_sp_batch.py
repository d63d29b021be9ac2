"""The sum-product kernel's list of blocks still decoding: batches that end at
different iterations, more blocks than one launch takes, and the same decode
one iteration a call, against the oracle."""
import numpy as np
import pytest

import oracle
from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu
RATE, N = "10/15", 16200


@pytest.mark.parametrize("nblk", [1, 9, 258])
def test_sp_batches_vs_oracle(nblk):
    import torch
    from atsc3_b200 import ldpc
    # a few distinct codewords, from hopeless to clean, repeated to the batch size
    lam = np.concatenate([oracle.near_miss_llr(RATE, N, 1, mu, 3 + i)[0]
                          for i, mu in enumerate((1.0, 3.6, 4.2, 30.0))]).astype(np.float64)
    want = oracle.sum_product(lam, C.csr(RATE, N), N, iters=12)
    pick = np.arange(nblk) % len(lam)
    tab = ldpc.sp_tables(C.csr(RATE, N), N)
    x = torch.from_numpy(np.ascontiguousarray(lam[pick])).cuda()
    whole = ldpc.sp_decode(tab, x, iters=12)
    steps, shed = ldpc.sp_decode_deadline(tab, x, iters=12)
    assert shed == 0
    for got in (whole, steps):
        for k, w in zip(("bits", "conv", "its", "bad"), want):
            assert np.array_equal(got[k].cpu().numpy().astype(np.int64),
                                  np.asarray(w)[pick].astype(np.int64)), k

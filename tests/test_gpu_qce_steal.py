"""More codewords than resident clusters: clusters take further codewords as they
finish.  Every codeword's outputs equal those of a decode of it in a small batch,
whatever mix of early and late ends; no launch loses one; a captured launch
replays."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,n,nblk,dtype", [
    ("6/15", 64800, 23, "float32"), ("8/15", 64800, 61, "float32"), ("7/15", 64800, 40, "float32"),
    ("2/15", 16200, 311, "float32"), ("11/15", 16200, 150, "float32"),
    ("8/15", 16200, 120, "float64")])
def test_steal_equals_small_batches(rate, n, nblk, dtype):
    import torch
    from atsc3_b200 import native as N
    from atsc3_b200.ldpc import QcePlan, decode_flood
    dt = torch.float64 if dtype == "float64" else torch.float32
    plan = QcePlan(rate, n, dtype=dtype)
    g = torch.Generator(device="cuda").manual_seed(nblk)
    mu = {"2/15": 0.5, "11/15": 7.0}.get(rate, 3.0)
    # from hopeless to clean, in a mixed order
    m = mu * (0.3 + 2.5 * torch.rand((nblk, 1), generator=g, device="cuda", dtype=dt))
    x = m + (2 * m).sqrt() * torch.randn((nblk, n), generator=g, device="cuda", dtype=dt)
    run = lambda y, o=None: decode_flood(plan, y, iters=30, out=o, want_hard=True)
    got = run(x)
    keys = ("bits", "conv", "its", "bad")
    for lo in range(0, nblk, 7):
        want = run(x[lo:lo + 7])
        for k in keys:
            assert torch.equal(got[k][lo:lo + 7], want[k]), (lo, k)
    assert int(got["its"].min()) < 30 == int(got["its"].max())
    out = {k: torch.zeros_like(v) for k, v in got.items()}
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(x, out)
    for _ in range(2):
        for k in keys:
            out[k].zero_()
        graph.replay()
        for k in keys:
            assert torch.equal(got[k], out[k]), k
    err = ctypes.c_int32(-1)
    N.call("atsc3_ldpc_qce_plan_error", plan.handle, ctypes.byref(err))
    assert err.value == 0

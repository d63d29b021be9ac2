"""wide=False: the plan keeps its one cluster size for every batch, in both value
types and through every entry point that builds one, and decodes what a plan
with larger sizes decodes."""
import numpy as np
import pytest

from atsc3_b200 import ldpc
from atsc3_b200 import native as N


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_wide_false_asks_for_one_size(dtype, monkeypatch):
    calls = []
    monkeypatch.setattr(N, "call", lambda name, *a: calls.append(name))
    one = {"float32": "atsc3_ldpc_qce_plan_create_one",
           "float64": "atsc3_ldpc_qce_plan_create_one_f64"}[dtype]
    ldpc.QcePlan("6/15", 16200, dtype=dtype, wide=False)
    assert calls[0] == one
    for kw in ({}, {"cluster": 3, "wide": False}):      # several sizes; a pinned one
        calls.clear()
        ldpc.QcePlan("6/15", 16200, dtype=dtype, **kw)
        assert calls[0] != one


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_one_size_decodes_alike(dtype):
    import torch
    dt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = 3 + 6 ** 0.5 * torch.randn((9, 16200), generator=g, device="cuda", dtype=dt)
    one, wide = (ldpc.QcePlan("8/15", 16200, dtype=dtype, wide=w) for w in (False, True))
    assert one.cluster == wide.cluster
    for nblk in (1, 9):
        a, b = (ldpc.decode_flood(p, x[:nblk], iters=20) for p in (one, wide))
        for k in ("bits", "conv", "its", "bad"):
            assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy()), (nblk, k)


@pytest.mark.gpu
def test_wide_reaches_the_plan(monkeypatch):
    from atsc3_b200 import codes as C
    from atsc3_b200.pipeline import FecPipeline
    made, real = [], ldpc.QcePlan
    monkeypatch.setattr(ldpc, "QcePlan",
                        lambda *a, **kw: (made.append(kw["wide"]), real(*a, **kw))[1])
    monkeypatch.setattr(ldpc, "_PLANS", {})
    tabs = C.csr("6/15", 16200)
    checks = np.split(tabs[1], tabs[0][1:-1])
    for make in (lambda **kw: ldpc.plan_for("6/15", 16200, **kw),
                 lambda **kw: ldpc.qce_plan_from_csr(tabs, 16200, **kw),
                 lambda **kw: FecPipeline(16200, "QPSK", "9/15", **kw).plan,
                 lambda **kw: ldpc.GpuMinSum(checks, 16200, **kw).plan):
        made.clear()
        plans = [make(), make(wide=False)]
        assert made == [True, False] and plans[0] is not plans[1]

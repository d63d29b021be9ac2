"""A plan with larger clusters beside its own gives the outputs of the plan
pinned to the smallest, whatever batch size chooses which."""
import pytest

from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,n,dtype", [
    ("2/15", 16200, "float32"), ("8/15", 16200, "float32"), ("13/15", 16200, "float32"),
    ("6/15", 64800, "float32"), ("7/15", 64800, "float32"), ("11/15", 64800, "float32"),
    ("8/15", 16200, "float64")])
def test_wide_plan_equals_pinned(rate, n, dtype):
    import torch
    from atsc3_b200.ldpc import QcePlan, decode_flood
    dt = torch.float64 if dtype == "float64" else torch.float32
    wide = QcePlan(rate, n, dtype=dtype)
    one = QcePlan(rate, n, cluster=wide.cluster, dtype=dtype)
    g = torch.Generator(device="cuda").manual_seed(n)
    # the zero codeword at a noise level where some blocks converge
    mu = {"2/15": 0.5, "13/15": 11.0}.get(rate, 3.0 if n == 16200 else 2.6)
    x = mu + (2 * mu) ** 0.5 * torch.randn((24, n), generator=g, device="cuda", dtype=dt)
    for nblk in (1, 6, 7, 8, 10, 15, 16, 23):
        for sem in ("kernel", "torch"):
            a, b = (decode_flood(p, x[:nblk], iters=15, semantics=sem) for p in (wide, one))
            for k in ("bits", "conv", "its", "bad"):
                assert torch.equal(a[k], b[k]), (nblk, sem, k)

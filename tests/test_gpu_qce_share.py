"""Clusters claiming the codewords of a launch through its iteration counts:
whatever the outputs held before, whatever else decodes at the same time, every
codeword's outputs equal those of a decode that has a cluster for each."""
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("bits", "conv", "its", "bad")


def _llr(torch, nblk, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    # from hopeless to clean, in a mixed order
    m = 3.0 * (0.3 + 2.5 * torch.rand((nblk, 1), generator=g, device="cuda"))
    return m + (2 * m).sqrt() * torch.randn((nblk, n), generator=g, device="cuda")


@pytest.mark.parametrize("rate,n,nblk", [
    ("6/15", 64800, 23), ("8/15", 64800, 75), ("9/15", 16200, 75), ("9/15", 16200, 501),
    ("2/15", 16200, 1000)])
def test_outputs_held_anything_two_streams(rate, n, nblk):
    import torch
    from atsc3_b200.ldpc import QcePlan, decode_flood
    plan = QcePlan(rate, n)
    run = lambda y, o=None: decode_flood(plan, y, iters=30, out=o)
    xs = [_llr(torch, nblk, n, nblk + i) for i in range(3)]
    want = []
    for x in xs:
        parts = [run(x[lo:lo + 7]) for lo in range(0, nblk, 7)]
        want.append({k: torch.cat([p[k] for p in parts]) for k in KEYS})
    streams = [torch.cuda.Stream() for _ in xs]
    for poison in (-1, -2, 0, nblk):
        outs = [{k: torch.full_like(v, poison % 256 if v.dtype == torch.uint8 else poison)
                 for k, v in w.items()} for w in want]
        torch.cuda.synchronize()
        for _ in range(2):
            for s, x, o in zip(streams, xs, outs):
                with torch.cuda.stream(s):
                    run(x, o)
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            for k in KEYS:
                assert torch.equal(o[k], w[k]), (poison, k)


def test_status_outputs_in_pinned_host_memory():
    import torch
    from atsc3_b200.ldpc import QcePlan, decode_flood
    plan = QcePlan("9/15", 16200)
    x = _llr(torch, 200, 16200, 4)
    want = decode_flood(plan, x, iters=30)
    out = {k: torch.full_like(want[k], 77, device="cpu").pin_memory() for k in ("conv", "its", "bad")}
    for _ in range(3):
        got = decode_flood(plan, x, iters=30, out=dict(out))
        torch.cuda.synchronize()
        assert torch.equal(got["bits"], want["bits"])
        for k in out:
            assert torch.equal(out[k], want[k].cpu()), k
            out[k].fill_(-1 if k != "conv" else 1)

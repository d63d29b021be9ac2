"""The weighted min-sum's entry points without padding, which only C callers
use: outputs and records of the padded forward in the documented order, gradients
against the float64 reference, capture; and the per-row sigma2 estimate alone."""
import ctypes

import numpy as np
import pytest

from atsc3_b200 import codes as C
from atsc3_b200 import native as N

RATE, CODE_N, T = "8/15", 16200, 3


def test_backward_refuses_null_tables():
    p = ctypes.c_void_p(64)                    # never dereferenced: refused first
    fn = N.lib().atsc3_wms_backward
    args = [p] * 7 + [16200, 7560, 50000, 3, 1, 2] + [p] * 9
    for k in (0, 1, 2, 3, 6, 14, 15, 16, 17, 18, 19, 20):
        bad = list(args)
        bad[k] = None
        assert fn(*bad) == -3, k


def _forward(torch, code, x, a, b):
    nblk = x.shape[0]
    st = torch.cuda.current_stream().cuda_stream
    rec = torch.zeros((T, nblk, code.nc, 16), dtype=torch.uint8, device="cuda")
    out = torch.zeros_like(x)
    N.call("atsc3_wms_forward", *code.ptrs(), code.n, code.nc, code.ne, code.nbucket, nblk, T,
           x.data_ptr(), a.data_ptr(), b.data_ptr(), 0, rec.data_ptr(), out.data_ptr(), st)
    return rec, out


def _case(torch, nblk):
    from atsc3_b200.learned import WmsCode
    from test_gpu_wms import _case as llrs
    lam, cw = llrs(seed=nblk, nb=nblk, n=CODE_N)
    code = WmsCode(RATE, CODE_N)
    rng = np.random.default_rng(nblk)
    p = [(0.7 + 0.2 * rng.random((T, code.nbucket))).astype(np.float32),
         (0.1 * rng.random((T, code.nbucket))).astype(np.float32)]
    return code, torch.from_numpy(lam), torch.from_numpy(cw), p


@pytest.mark.gpu
@pytest.mark.parametrize("nblk", [1, 3, 33])
def test_forward_records_and_backward(nblk):
    import torch
    from atsc3_b200.learned import bce_loss, reference_f64
    code, lam, cw, p = _case(torch, nblk)
    x = lam.cuda()
    a, b = (torch.from_numpy(v).cuda() for v in p)
    st = torch.cuda.current_stream().cuda_stream
    rec, out = _forward(torch, code, x, a, b)
    # the padded forward's records (iters, nc, nbp) are the same values
    nbp = (nblk + 3) // 4 * 4
    rec2 = torch.zeros((T, code.nc, nbp, 16), dtype=torch.uint8, device="cuda")
    out2 = torch.zeros_like(x)
    work = torch.empty(nbp * (2 * code.n + code.ne), dtype=torch.float32, device="cuda")
    csr = code.ptrs(("cptr", "cidx", "vptr", "vedge", "cbucket"))
    N.call("atsc3_wms_forward_work", *csr, code.n, code.nc, code.ne, code.nbucket, nblk, T,
           x.data_ptr(), a.data_ptr(), b.data_ptr(), 0, rec2.data_ptr(), out2.data_ptr(),
           work.data_ptr(), st)
    assert torch.equal(out, out2)
    assert torch.equal(rec, rec2[:, :, :nblk].transpose(1, 2))
    # gradients: of the float64 reference by autograd.  dL/dllr is the sum of
    # dL/dtot^(t) over t = 0 .. T; the call over iterations t+1 .. T gives one each
    p64 = [torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in p]
    x64 = lam.double().requires_grad_(True)
    bce_loss(reference_f64(x64, *p64, RATE, CODE_N), cw.double()).backward()
    o = out.clone().requires_grad_(True)
    bce_loss(o, cw.cuda()).backward()
    total = o.grad.clone()
    for t in reversed(range(T)):
        g = o.grad.clone()
        ga, gb = torch.zeros_like(a), torch.zeros_like(b)
        work = torch.empty(nblk * (code.n + 2 * code.ne), dtype=torch.float32, device="cuda")
        N.call("atsc3_wms_backward", *code.ptrs(), code.n, code.nc, code.ne, code.nbucket, nblk,
               T - t, x.data_ptr(), a[t].data_ptr(), b[t].data_ptr(), rec[t].data_ptr(),
               g.data_ptr(), ga.data_ptr(), gb.data_ptr(), work.data_ptr(), st)
        total += g
    for g, gr in ((ga, p64[0].grad), (gb, p64[1].grad)):       # of all T iterations
        assert float((g.cpu().double() - gr).abs().max() / gr.abs().max()) < 1e-3
    # a check whose two smallest values round alike may choose the other one:
    # single entries differ then, so 1 in 1000 may be off
    off = (total.cpu().double() - x64.grad).abs() > 1e-3 * x64.grad.abs().max()
    assert off.double().mean() < 1e-3


@pytest.mark.gpu
def test_forward_under_capture():
    import torch
    code, lam, _, p = _case(torch, 2)
    x = lam.cuda()
    a, b = (torch.from_numpy(v).cuda() for v in p)
    rec, out = _forward(torch, code, x, a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rec2, out2 = _forward(torch, code, x, a, b)
    for _ in range(2):
        rec2.zero_()
        out2.zero_()
        graph.replay()
        assert torch.equal(rec, rec2) and torch.equal(out, out2)


@pytest.mark.gpu
@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("mod,nblk,ncell", [("QPSK", 5, 1), ("64QAM", 3, 257), ("256QAM", 1, 5000),
                                            ("1024QAM", 2, 700), ("4096QAM", 2, 300)])
def test_row_sigma2(mod, nblk, ncell, f64):
    """max(mean(|z|^2 + min q), 1e-9): the terms are the kernel's own roundings,
    none negative beyond them, summed in another order, ncell + 2 roundings of the
    float64 sum and mean, and one of the float32 result."""
    import torch
    nb = C.MOD_BITS[mod]
    pts = np.array(C.alphabet(mod, "9/15"), np.complex128)
    rng = np.random.default_rng(ncell)
    z = pts[rng.integers(0, len(pts), (nblk, ncell))]
    z = z + 0.05 * (rng.standard_normal(z.shape) + 1j * rng.standard_normal(z.shape))
    z = z.astype(np.complex128 if f64 else np.complex64)
    tab = (np.concatenate([pts.real, pts.imag, np.abs(pts) ** 2]) if f64
           else np.concatenate(C.point_tables_f32(pts)).astype(np.float32)).reshape(3, -1)
    near = np.empty((nblk, ncell))
    for k in range(nblk):
        zr, zi = z[k].real[:, None], z[k].imag[:, None]
        q = (zr * tab[0] + zi * tab[1]) * tab.dtype.type(-2) + tab[2]
        near[k] = z[k].real * z[k].real + z[k].imag * z[k].imag + q.min(1)
    want = np.maximum(near.mean(1), 1e-9)
    zt, pt = torch.from_numpy(z).cuda(), torch.from_numpy(tab.ravel()).cuda()
    got = torch.zeros(nblk, dtype=torch.float64 if f64 else torch.float32, device="cuda")
    N.call("atsc3_demap_row_sigma2_f64" if f64 else "atsc3_demap_row_sigma2",
           torch.view_as_real(zt).data_ptr(), ncell, nblk, ncell, pt.data_ptr(), nb,
           got.data_ptr(), torch.cuda.current_stream().cuda_stream)
    tol = (ncell + 2) * 2.0 ** -53 * np.abs(near).mean(1) + (0 if f64 else 2.0 ** -24 * want)
    assert np.all(np.abs(got.cpu().numpy() - want) <= tol)

"""The demapper's three ways to the per-bit minima (general, mirrored
quadrants, grid) against the oracle, bit for bit: alphabets that have the
structure and the same with one point moved (general form), cells at the
points, midway between two of them, around them and far outside, at sizes
around a CTA's 256 cells."""
import numpy as np
import pytest

import oracle
from atsc3_b200 import codes as C
from atsc3_b200 import native as N

pytestmark = pytest.mark.gpu


def _cells(pts, n, rng):
    a, b = pts[rng.integers(0, len(pts), (2, n))]
    kind = rng.integers(0, 5, n)
    far = 10.0 ** rng.uniform(0, 4, n) * np.exp(2j * np.pi * rng.random(n))
    near = a + 0.1 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    return np.select([kind == 0, kind == 1, kind == 2, kind == 3],
                     [a, (a + b) / 2, near, far], near.real + 1j * a.imag)


@pytest.mark.parametrize("moved", [False, True])
@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("mod", ["QPSK", "16QAM", "64QAM", "256QAM", "1024QAM", "4096QAM"])
def test_demap_forms_vs_oracle(mod, f64, moved):
    import torch
    nb = C.MOD_BITS[mod]
    pts = np.array(C.alphabet(mod, "9/15"), np.complex128)
    rng = np.random.default_rng(nb + 100 * moved)
    if moved:
        pts[len(pts) // 3] += 0.01 - 0.02j
    if f64:
        tab = np.concatenate([pts.real, pts.imag, np.abs(pts) ** 2])
    else:
        tab = np.concatenate(C.point_tables_f32(pts)).astype(np.float32)
    dt = tab.dtype.type
    name = "atsc3_demap_f64" if f64 else "atsc3_demap"
    t = torch.from_numpy(tab).cuda()
    for n in (1, 255, 257, 300):
        z = _cells(pts, 2 * n, rng).reshape(2, n).astype(np.complex128 if f64 else np.complex64)
        zr, zi = z.real[..., None], z.imag[..., None]
        pr, pi, p2 = tab.reshape(3, -1)
        q = (zr * pr + zi * pi) * dt(-2) + p2
        bit = (np.arange(len(pts)) >> (nb - 1 - np.arange(nb))[:, None]) & 1
        want = np.stack([q[..., b == 1].min(-1) - q[..., b == 0].min(-1) for b in bit], -1)
        if not f64:                    # the oracle's own demapper says the same
            assert np.array_equal(want.reshape(2, -1), oracle.demap(z, pts, nb, np.ones((2, n), np.float32)))
        zt = torch.from_numpy(z).cuda()
        out = torch.empty((2, n * nb), dtype=torch.float64 if f64 else torch.float32, device="cuda")
        N.call(name, torch.view_as_real(zt).data_ptr(), n, 2, n, t.data_ptr(), nb, 0, None, 0, 1.0,
               None, out.data_ptr(), n * nb, torch.cuda.current_stream().cuda_stream)
        assert np.array_equal(out.cpu().numpy().reshape(want.shape), want)


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("mod,nblk,ncell,pad", [
    ("QPSK", 5, 1, 0), ("16QAM", 3, 255, 1), ("64QAM", 1, 257, 3), ("256QAM", 2, 5000, 0),
    ("1024QAM", 5000, 3, 0), ("4096QAM", 4, 700, 5)])
def test_demap_estimate_rows(mod, nblk, ncell, pad, f64):
    """sigma2 estimated per row: the undivided LLRs over the row's mean of
    |z|^2 + min q.  The terms are the kernel's own roundings, summed here in
    another order: (ncell + 4) roundings of the sum and the division (float64),
    or one of the float32 mean and one of the division."""
    import torch
    from atsc3_b200 import demap as DM
    nb = C.MOD_BITS[mod]
    pts = np.array(C.alphabet(mod, "9/15"), np.complex128)
    rng = np.random.default_rng(nblk)
    z = pts[rng.integers(0, len(pts), (nblk, ncell))]
    z = z + 0.05 * (rng.standard_normal(z.shape) + 1j * rng.standard_normal(z.shape))
    z = z.astype(np.complex128 if f64 else np.complex64)
    tab = (np.concatenate([pts.real, pts.imag, np.abs(pts) ** 2]) if f64
           else np.concatenate(C.point_tables_f32(pts)).astype(np.float32)).reshape(3, -1)
    near = np.empty((nblk, ncell))
    for b in range(nblk):
        zr, zi = z[b].real[:, None], z[b].imag[:, None]
        q = (zr * tab[0] + zi * tab[1]) * tab.dtype.type(-2) + tab[2]
        near[b] = z[b].real * z[b].real + z[b].imag * z[b].imag + q.min(1)
    s2 = np.maximum(near.mean(1), 1e-9)[:, None]
    fn, dt = (DM.demap_f64, torch.float64) if f64 else (DM.demap, torch.float32)
    zt = torch.from_numpy(z).cuda()
    raw = fn(zt, mod, "9/15", sigma2=1.0, deinterleave=False).cpu().numpy().astype(np.float64)
    buf = torch.zeros((nblk, ncell * nb + pad), dtype=dt, device="cuda")
    fn(zt, mod, "9/15", deinterleave=False, out=buf)
    got = buf.cpu().numpy()
    assert np.all(got[:, ncell * nb:] == 0)
    want = raw / s2
    tol = (ncell + 4) * 2.0 ** -53 if f64 else 2 * 2.0 ** -24 + ncell * 2.0 ** -53
    assert np.all(np.abs(got[:, :ncell * nb] - want) <= tol * np.abs(want))

"""Scratch of a call on a stream that the caller names: its memory goes to
nobody else while that stream has not run the call, also when a second call
writes the same outputs."""
import pytest

from atsc3_b200 import codes as C

pytestmark = pytest.mark.gpu


def _demap(torch, dtype):
    from atsc3_b200 import demap as DM
    fn = DM.demap if dtype == torch.complex64 else DM.demap_f64
    z = torch.randn((2, 2700), dtype=dtype, device="cuda")
    out = torch.empty((2, 2700 * 6), dtype=z.real.dtype, device="cuda")
    return lambda st: fn(z, "64QAM", "9/15", deinterleave=False, out=out, stream=st)


def _cpe(torch, _):
    from atsc3_b200.cpe import cpe_correct_device
    pool = torch.randn(900, dtype=torch.complex128, device="cuda")
    ptr = torch.tensor([0, 400, 900], dtype=torch.int32, device="cuda")
    region = torch.zeros(900, dtype=torch.uint8, device="cuda")
    al = torch.tensor(C.alphabet("16QAM", "9/15"), dtype=torch.complex128, device="cuda")
    out = torch.empty_like(pool)
    return lambda st: cpe_correct_device(pool, ptr, region, [al], out=out, stream=st)


def _sp(torch, _):
    from atsc3_b200 import ldpc
    tab = ldpc.sp_tables(C.csr("11/15", 16200), 16200)
    x = torch.randn((1, 16200), dtype=torch.float64, device="cuda")
    out = {}
    return lambda st: ldpc.sp_decode(tab, x, iters=2, out=out, stream=st)


@pytest.mark.parametrize("make,dtype", [(_demap, "complex64"), (_demap, "complex128"),
                                        (_cpe, None), (_sp, None)])
def test_scratch_stays_until_the_stream_has_run(make, dtype, monkeypatch):
    import ctypes
    import gc

    import torch
    from atsc3_b200 import native as N
    call = make(torch, getattr(torch, dtype) if dtype else None)
    side = torch.cuda.Stream()
    sizes, empty = [], torch.empty

    def noted(*a, **kw):
        t = empty(*a, **kw)
        sizes.append(t.nbytes)
        return t

    monkeypatch.setattr(torch, "empty", noted)
    call(0)                                     # the default stream; tables and modules loaded
    monkeypatch.setattr(torch, "empty", empty)
    # the memory that is asked for below is there before the stream is held up, so
    # that nothing waits for the device meanwhile
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = [[torch.empty(n, dtype=torch.uint8, device="cuda") for _ in range(8)] for n in sizes]
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    scratch, real = [], N.call
    monkeypatch.setattr(N, "call", lambda name, *a: (scratch.append(a[-2]), real(name, *a))[1]
                        if name.startswith(("atsc3_demap_est", "atsc3_cpe_corr", "atsc3_ldpc_sp_dec"))
                        else real(name, *a))
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000_000)        # about a second
    for handle in (side.cuda_stream, ctypes.c_void_p(side.cuda_stream)):
        call(handle)
    del held
    fresh = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(40)]
    assert not side.query() and len(scratch) == 2
    for t in fresh:
        lo, hi = t.data_ptr(), t.data_ptr() + t.numel()
        assert not any(lo <= s < hi for s in scratch)
    torch.cuda.synchronize()

"""n2b_bptt_backward takes buffers of any float alignment: every array one float past a 16-byte boundary gives the
results of aligned ones, bit for bit."""

import ctypes

import pytest
import torch

from naer2_b200 import _lib
from naer2_b200.bptt import RecurrentLIF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, R, B, T", [(32, 1, 8, 5), (96, 7, 16, 40), (1024, 20, 8, 12)])
def test_backward_over_arrays_off_the_16_byte_grid(cuda, H, R, B, T):
    layer = RecurrentLIF(n_in=4, hidden=H, readouts=R, density=0.1, checkpoint=7, seed=H, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(R)
    U = 0.35 * torch.randn(T, B, H, generator=g, device=cuda) + 0.1
    dm = torch.randn(B, R, generator=g, device=cuda)
    m, ts = layer.run_forward(U, tape=True)
    want = layer.run_backward(U, dm, ts)

    def off(t, fill=False):
        buf = torch.full((t.numel() + 1,), float("nan") if t.is_floating_point() else -1, dtype=t.dtype, device=cuda)
        v = buf[1:]
        assert v.data_ptr() % 16 == 4
        return v.copy_(t.reshape(-1)) if fill else v

    ins = [off(x, True) for x in (U, layer.w_rec.detach(), layer.w_out.detach(), dm, ts)]
    outs = [off(x) for x in want]
    d = layer.desc(B, T)
    ws = layer.workspace(d)
    lib, s = _lib.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    m2, ts2 = off(m), off(ts)
    _lib.check(lib.n2b_bptt_forward(ctypes.byref(d), *(x.data_ptr() for x in ins[:3]), 1, m2.data_ptr(), ts2.data_ptr(),
                                    ws.data_ptr(), ws.numel(), s), "n2b_bptt_forward")
    _lib.check(lib.n2b_bptt_backward(ctypes.byref(d), *(x.data_ptr() for x in ins), *(x.data_ptr() for x in outs),
                                     ws.data_ptr(), ws.numel(), s), "n2b_bptt_backward")
    assert torch.equal(m2.view_as(m), m) and torch.equal(ts2.view_as(ts), ts)
    for a, b in zip(outs, want):
        assert torch.equal(a.view_as(b), b)

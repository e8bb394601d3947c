"""The spiking forward's two kernels -- one for long sequences on few SMs' worth of groups, one for the rest
(csrc/bptt.cu, scans) -- give the same bits on either side of the lines between them: a batch's samples are those of a
small batch, a sequence's first steps are the spikes of a longer one."""

import pytest
import torch

from naer2_b200.bptt import RecurrentLIF

pytestmark = pytest.mark.gpu


def _layer(cuda, H):
    return RecurrentLIF(n_in=4, hidden=H, readouts=6, density=0.1, checkpoint=7, seed=H, device=cuda)


@pytest.mark.parametrize("H, B", [(1024, 152), (512, 152), (256, 304), (64, 8)])
@pytest.mark.parametrize("tape", [False, True])
def test_lines(cuda, H, B, tape):
    g = torch.Generator(device=cuda).manual_seed(B)
    U = 0.35 * torch.randn(26, B, H, generator=g, device=cuda) + 0.1
    layer = _layer(cuda, H)
    want, want_ts = layer.run_forward(U[:, -8:].contiguous(), tape=tape)
    spikes = layer.spikes(8, 26) if tape else None
    for T in (26, 24, 23, 1):
        m, ts = layer.run_forward(U[:T].contiguous(), tape=tape)
        if tape:
            assert layer.status(B, T) == [0, 0, 0, 0]
            assert torch.equal(layer.spikes(B, T)[:, -8:], spikes[:T])
        if T == 26:
            assert torch.equal(m[-8:], want) and torch.equal(ts[-8:], want_ts)


@pytest.mark.parametrize("H, B, T", [(256, 128, 30), (256, 152, 24), (512, 64, 24), (64, 256, 12), (256, 304, 40)])
def test_gradients_of_a_batch_are_its_samples(cuda, H, B, T):
    """dU of the last samples is the small batch's, bit for bit, wherever the adjoint's blocks are placed."""
    g = torch.Generator(device=cuda).manual_seed(T)
    U = 0.35 * torch.randn(T, B, H, generator=g, device=cuda) + 0.1
    dm = torch.randn(B, 6, generator=g, device=cuda)
    layer = _layer(cuda, H)
    _, ts = layer.run_forward(U, tape=True)
    du, _, _ = layer.run_backward(U, dm, ts)
    assert layer.status(B, T) == [0, 0, 0, 0]
    small = U[:, -8:].contiguous()
    _, ts8 = layer.run_forward(small, tape=True)
    du8, _, _ = layer.run_backward(small, dm[-8:].contiguous(), ts8)
    assert torch.equal(ts[-8:], ts8) and torch.equal(du[:, -8:], du8) and float(du8.abs().max()) > 0

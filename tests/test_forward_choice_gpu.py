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

"""The spiking forward's wait for its group's spikes gives up after n2b_bptt_desc.wait_polls polls without a hang: with
one poll (every block still arrives, every launch still ends) the error word counts the waits, for the plain and the
taped forward; with the default the results are the first run's bit for bit and every word is zero."""

import pytest
import torch

from naer2_b200.bptt import RecurrentLIF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tape", [False, True])
def test_forward_wait_gives_up(cuda, tape):
    B, T, H = 16, 200, 256
    layer = RecurrentLIF(n_in=4, hidden=H, readouts=5, density=0.2, checkpoint=7, seed=1, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(2)
    U = 0.35 * torch.randn(T, B, H, generator=g, device=cuda) + 0.1
    m, ts = layer.run_forward(U, tape=tape)
    assert layer.status(B, T) == [0, 0, 0, 0]
    layer.wait_polls = 1
    layer.run_forward(U, tape=tape)
    assert layer.status(B, T)[3] >= 1
    layer.wait_polls = 0
    m2, ts2 = layer.run_forward(U, tape=tape)
    assert layer.status(B, T) == [0, 0, 0, 0]
    assert torch.equal(m, m2) and torch.equal(ts, ts2)

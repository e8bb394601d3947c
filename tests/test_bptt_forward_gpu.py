"""The spiking forward that looks at its links' spikes first (csrc/bptt.cu, fwd_group_kernel): its sums are the
links' in their order, so its results are bit for bit those of the rows read link by link from global memory (a
wrong in_cta_max, counted), and those of the kernel for rows that do not fit shared memory (1024 hidden neurons at
30%). Rows of more than 128 and 256 links (more than one mask of a share, links past its masks), shares of unequal
length, one and 32 readouts, hidden sizes that are no power of two, more groups than one launch holds."""

import pytest
import torch

from naer2_b200.bptt import RecurrentLIF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, R, density, B, T", [(32, 1, 0.5, 8, 1), (32, 3, 0.03, 8, 20), (96, 32, 0.3, 16, 33),
                                                 (256, 7, 1.0, 8, 40), (320, 11, 0.1, 24, 50),
                                                 (512, 5, 0.6, 16, 25), (1024, 20, 0.1, 160, 30),
                                                 (1024, 17, 0.15, 8, 30), (1024, 20, 0.3, 8, 30)])
def test_the_forward_gives_the_links_sums_in_order(cuda, H, R, density, B, T):
    layer = RecurrentLIF(n_in=4, hidden=H, readouts=R, density=density, checkpoint=7, seed=H + R, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(R)
    U = 0.35 * torch.randn(T, B, H, generator=g, device=cuda) + 0.1
    m, ts = layer.run_forward(U, tape=True)
    s = layer.spikes(B, T)
    assert T == 1 or 0.005 < s.float().mean() < 0.6
    if H * H * density < 130000:  # (else the backward is refused: the outgoing rows do not fit)
        layer.run_backward(U, torch.randn(B, R, generator=g, device=cuda), ts)
    assert layer.status(B, T) == [0, 0, 0, 0]
    plain, _ = layer.run_forward(U, tape=False)
    layer.wiring.in_cta_max, layer._ws_key = 0, None
    m0, ts0 = layer.run_forward(U, tape=True)
    assert layer.status(B, T)[2] > 0
    assert torch.equal(m, m0) and torch.equal(ts, ts0) and torch.equal(s, layer.spikes(B, T))
    assert torch.equal(m, plain)

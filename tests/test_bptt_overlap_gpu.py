"""Plain forwards of one layer that overlap on the device -- with one another on two streams, with a taped forward's
backward -- give what the same calls give one after the other, bit for bit: each has scratch of its own, and without a
tape n2b_bptt_forward writes nothing of the layer's workspace but the error words."""

import ctypes

import pytest
import torch

from naer2_b200 import _lib
from naer2_b200.bptt import RecurrentLIF

pytestmark = pytest.mark.gpu


def _layer(cuda, H, B, T):
    layer = RecurrentLIF(n_in=4, hidden=H, readouts=5, density=0.2, checkpoint=7, seed=H, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(B)
    return layer, [0.35 * torch.randn(T, B, H, generator=g, device=cuda) + 0.1 * k for k in (0, 1, 2)], g


@pytest.mark.parametrize("H, B, T", [(64, 8, 400), (320, 24, 151)])
def test_plain_forwards_on_two_streams(cuda, H, B, T):
    layer, us, _ = _layer(cuda, H, B, T)
    want = [layer.run_forward(U, tape=False) for U in us]
    assert layer._ws is None and layer.status(B, T) == [0, 0, 0, 0]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(cuda) for _ in us]
    got = [[], [], []]
    for _ in range(12):  # (queued without a wait: the calls of the three streams overlap)
        for k, (s, U) in enumerate(zip(streams, us)):
            with torch.cuda.stream(s):
                got[k].append(layer.run_forward(U, tape=False))
    torch.cuda.synchronize()
    for k, (m, ts) in enumerate(want):
        for gm, gt in got[k]:
            assert torch.equal(gm, m) and torch.equal(gt, ts)


def test_plain_forwards_beside_a_backward(cuda):
    B, T, H = 16, 300, 128
    layer, us, g = _layer(cuda, H, B, T)
    dm = torch.randn(B, 5, generator=g, device=cuda)
    plain = layer.run_forward(us[1], tape=False)
    _, ts = layer.run_forward(us[0], tape=True)
    want = layer.run_backward(us[0], dm, ts)
    torch.cuda.synchronize()
    side = torch.cuda.Stream(cuda)
    for _ in range(6):
        with torch.cuda.stream(side):
            inferred = [layer.run_forward(us[1], tape=False) for _ in range(4)]
        got = layer.run_backward(us[0], dm, ts)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        for m, t in inferred:
            assert torch.equal(m, plain[0]) and torch.equal(t, plain[1])


def test_a_forward_without_a_tape_leaves_the_workspace(cuda):
    B, T, H = 8, 40, 64
    layer, us, _ = _layer(cuda, H, B, T)
    m, ts = layer.run_forward(us[0], tape=False)
    d = layer.desc(B, T)
    ws = layer.workspace(d)
    ws.fill_(0x5A)
    m2, ts2 = torch.empty_like(m), torch.empty_like(ts)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().n2b_bptt_forward(ctypes.byref(d), us[0].data_ptr(), layer.w_rec.data_ptr(),
                                            layer.w_out.data_ptr(), 0, m2.data_ptr(), ts2.data_ptr(), ws.data_ptr(),
                                            ws.numel(), s), "n2b_bptt_forward")
    assert torch.equal(m, m2) and torch.equal(ts, ts2)
    assert int((ws != 0x5A).sum()) == 4 * _lib.BPTT_ERR_WORDS


def test_a_batch_of_more_groups_than_a_grid_has_rows(cuda):
    """65,544 groups of 8 samples: the last samples are those of a small batch, bit for bit."""
    B, T, H = 8 * 65544, 2, 32
    layer = RecurrentLIF(n_in=4, hidden=H, readouts=1, density=0.5, checkpoint=7, seed=H, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(1)
    U = 0.6 + 0.5 * torch.randn(T, B, H, generator=g, device=cuda)
    m, ts = layer.run_forward(U, tape=False)
    want, want_ts = layer.run_forward(U[:, -16:].contiguous(), tape=False)
    assert torch.equal(m[-16:], want) and torch.equal(ts[-16:], want_ts)
    assert int((m != 0).sum()) > B // 4


@pytest.mark.parametrize("smooth", [False, True])
def test_captured_calls_replay(cuda, smooth):
    """A plain forward, and a taped one with its backward, captured into graphs and replayed on other currents."""
    B, T, H = 16, 60, 128
    layer, us, g = _layer(cuda, H, B, T)
    layer.smooth, layer._ws_key = smooth, None
    dm = torch.randn(B, 5, generator=g, device=cuda)
    want = []
    for U in us:
        plain = layer.run_forward(U, tape=False)
        m, ts = layer.run_forward(U, tape=True)
        want.append([*plain, m, ts, *layer.run_backward(U, dm, ts)])
    torch.cuda.synchronize()
    static = us[0].clone()
    plain_graph, graph = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(plain_graph):
        plain = layer.run_forward(static, tape=False)
    with torch.cuda.graph(graph):
        m, ts = layer.run_forward(static, tape=True)
        grads = layer.run_backward(static, dm, ts)
    for U, w in zip(us, want):
        static.copy_(U)
        plain_graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip([*plain, m, ts, *grads], w):
            assert torch.equal(a, b)

"""The spiking layer's tape in segments (RecurrentLIF.segments: the membrane every `checkpoint` steps, each segment's
surrogate derivatives recomputed), the form of layers whose every step would take more than 4 GiB, or too much of the free
memory. Its forward is the other form's bit for bit; its gradients are the same sums with the readout's part added in
another order: R + 1 <= 33 terms per step and neuron, T B terms per dw_out, fp32 rounding of a few 1e-7 each, which the
adjoint carries on with a gain below ten, so within 2e-5 (norm of the difference over the norm). Against the float64
reference it is held to the tolerances of test_bptt_gpu.py."""

import pytest
import torch

from naer2_b200 import bptt
from naer2_b200.bptt import RecurrentLIF
from naer2_b200.networks import bptt_task
from test_bptt_gpu import kernel_grads, make, reference, rel

pytestmark = pytest.mark.gpu


def _run(layer, x, y):
    with torch.no_grad():
        U = layer.current(x).contiguous()
        m, ts = layer.run_forward(U, tape=True)
        s = layer.spikes(U.shape[1], U.shape[0])
        dm = torch.softmax(m, 1) - torch.nn.functional.one_hot(y, m.shape[1]).float()
        return (m, ts, s), layer.run_backward(U, dm, ts)


@pytest.mark.parametrize("B, T, H, R, K", [(16, 60, 64, 5, 7), (8, 33, 320, 11, 33), (24, 41, 96, 32, 1),
                                           (8, 30, 1024, 20, 50), (128, 12, 64, 5, 5), (256, 23, 256, 3, 9),
                                           (160, 24, 512, 7, 24)])
def test_segments_give_the_whole_tapes_results(cuda, B, T, H, R, K):
    layer, x, y = make(cuda, B=B, T=T, H=H, R=R, K=K, seed=4, density=0.1)
    layer.segments = False
    fwd, grads = _run(layer, x, y)
    whole = layer._ws.numel()
    layer.segments = True
    fwd2, grads2 = _run(layer, x, y)
    assert layer.status(B, T) == [0, 0, 0, 0]
    if 2 * K + (T + K - 1) // K < T:  # two segments and the checkpoints against every step
        assert layer._ws.numel() < whole
    assert all(torch.equal(a, b) for a, b in zip(fwd, fwd2)) and fwd[2].float().mean() > 0.002
    for a, b in zip(grads2, grads):
        assert b.abs().max() > 0 and rel(a, b) < 2e-5


def test_checkpoint_interval_changes_nothing(cuda):
    out = []
    for K in (1, 7, 60):
        layer, x, y = make(cuda, B=16, T=60, K=K, seed=4)
        layer.segments = True
        fwd, grads = _run(layer, x, y)
        out.append(fwd + grads)
        assert layer.status(16, 60) == [0, 0, 0, 0]
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("K", [13, 80])
def test_segments_match_the_teacher_forced_fp64_reference(cuda, K):
    B, T, H = 16, 80, 64
    layer, x, y = make(cuda, B=B, T=T, H=H, K=K, seed=2)
    layer.segments = True
    m, _, grads = kernel_grads(layer, x, y)
    assert layer.status(B, T) == [0, 0, 0, 0]
    spikes = layer.spikes(B, T)
    _, ts = layer.infer(x)
    m64, _, margins, _, _, g64, _ = reference(layer, x, y, forced=spikes, forced_tstar=ts)
    assert (((margins >= 0) != spikes) <= (margins.abs() < 1e-4)).all()
    assert rel(m, m64) < 1e-5
    for g, r in zip(grads, g64):
        assert rel(g, r) < 1e-4


def test_groups_beyond_one_cooperative_launch(cuda):
    """19 groups of 8 samples: the last group runs in a second launch of each segment; its samples are those of the same 8
    run alone, bit for bit."""
    T, B, C = 30, 152, 40
    layer = RecurrentLIF(n_in=C, hidden=1024, readouts=5, density=0.1, checkpoint=11, seed=9, device=cuda)
    layer.segments = True
    rates = bptt_task.templates(classes=5, channels=C, steps=T, seed=9)
    x, y = bptt_task.sample(rates, B, seed=10, device=cuda)
    out = []
    for xb, yb in ((x, y), (x[:, B - 8:].contiguous(), y[B - 8:])):
        (m, ts, _), (du, _, _) = _run(layer, xb, yb)
        assert layer.status(xb.shape[1], T) == [0, 0, 0, 0]
        out.append((m[-8:], ts[-8:], du[:, -8:]))
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_a_recomputed_spike_that_differs_is_counted(cuda):
    layer, x, y = make(cuda, B=8, T=40, K=9, seed=5)
    layer.segments = True
    with torch.no_grad():
        U = layer.current(x).contiguous()
        m, ts = layer.run_forward(U, tape=True)
        layer.run_backward(U + 2.0, torch.ones_like(m), ts)
    assert layer.status(8, 40)[1] > 0


def test_little_free_memory_takes_the_segments(cuda, monkeypatch):
    layer, x, y = make(cuda, B=16, T=60, K=7, seed=4)
    layer.segments = True
    want = _run(layer, x, y)
    small = layer._ws.numel()
    layer.segments = None
    _run(layer, x, y)
    assert layer._ws.numel() > small
    layer._ws = layer._ws_key = None
    monkeypatch.setattr(bptt, "SMALL_TAPE", 0)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: (0, 1 << 37))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev=None: torch.cuda.memory_allocated(dev) + (1 << 16))
    got = _run(layer, x, y)
    assert layer._ws.numel() == small
    for a, b in zip(got[0] + got[1], want[0] + want[1]):
        assert torch.equal(a, b)


def test_no_memory_for_the_whole_tape_takes_the_segments(cuda, monkeypatch):
    layer, x, y = make(cuda, B=16, T=60, K=7, seed=4)
    layer.segments = True
    want = _run(layer, x, y)
    small = layer._ws.numel()
    layer.segments, layer._ws, layer._ws_key = None, None, None
    empty = torch.empty

    def refuse(*size, **kw):
        if kw.get("dtype") is torch.uint8 and size[0] > small:
            raise torch.cuda.OutOfMemoryError("refused")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", refuse)
    got = _run(layer, x, y)
    assert layer._ws.numel() == small
    for a, b in zip(got[0] + got[1], want[0] + want[1]):
        assert torch.equal(a, b)

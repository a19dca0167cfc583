"""The concatenated activations of the network, which its convolutions read in place: whoever asks
for them after a forward pass finds them, and a backward pass uses those of the last forward
pass, also when that one was replayed from a graph."""
import numpy as np
import pytest

from lbm3d_bb_b200 import unet as N

pytestmark = pytest.mark.gpu

SHAPE = (1, 8, 8, 64)


def _input(seed):
    import torch

    g = torch.Generator().manual_seed(seed)
    return torch.randn((*SHAPE, N.IN_CH), generator=g).to(torch.bfloat16).cuda()


def _concatenation(low, skip):
    import torch

    for axis in (1, 2, 3):
        low = low.repeat_interleave(2, axis)
    return torch.cat([low, skip], -1)


@pytest.mark.parametrize("engine", ["auto", "mma"])
def test_concatenated_activations_are_those_of_the_last_forward(gpu, engine):
    import torch

    prev = N.set_conv_engine(engine)
    try:
        net = N.UNet3D(16, seed=1)
        for seed in (3, 4):
            net.forward(_input(seed))
            torch.cuda.synchronize()
            for cat, low, skip in (("c2", "b3", "s2"), ("c1", "a5", "s1")):
                want = _concatenation(net.A[low], net.A[skip])
                for got in (net.A[cat], net.A.get(cat), dict(net.A)[cat], dict(net.A.items())[cat]):
                    assert torch.equal(got, want), (seed, cat)
    finally:
        N.set_conv_engine(prev)


def _gradients(net, dout):
    import torch

    net.zero_grad()
    net.backward(dout)
    torch.cuda.synchronize()
    return {k: v.cpu().numpy().astype(np.float64) for k, v in net.G.items()}


def test_backward_after_a_replayed_forward(gpu):
    """Weight gradients are FP32 sums whose order changes from run to run (atomics): 1e-5 of
    their norm; with the concatenation of another input they differ by its whole norm."""
    import torch

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        net = N.UNet3D(16, seed=2, stream=stream)
        x = _input(10)
        dout = torch.randn((*SHAPE, N.OUT_CH), device="cuda").to(torch.bfloat16)
        net.forward(x)
        _gradients(net, dout)
        graph = torch.cuda.CUDAGraph()
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            net.forward(x)
        for seed in (11, 12, 13):
            x.copy_(_input(seed))
            graph.replay()
            got = _gradients(net, dout)
            net.forward(x)
            want = _gradients(net, dout)
            for k in want:
                assert np.linalg.norm(got[k] - want[k]) <= 1e-5 * np.linalg.norm(want[k]) + 1e-12, (seed, k)

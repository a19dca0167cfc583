"""Chained launches of the time loop (the next kernel is placed while the last one drains): the
same populations, bit for bit, from a non-blocking stream, from the legacy stream, with a host
wait after every launch, and from a captured graph replayed."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16dev"])
def test_captured_steps_equal_plain_steps(gpu, storage):
    import torch

    stream = torch.cuda.Stream()
    a = cases.sphere_channel(Domain, storage=storage, stream=stream)
    b = cases.sphere_channel(Domain, storage=storage)
    try:
        for d in (a, b):
            d.step(2)
            d.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            a.step(4)
        with torch.cuda.stream(stream):
            graph.replay()
        b.step(4)
        assert np.array_equal(a.populations(), b.populations())
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("mode", ["config", "reference"])
def test_moving_body_steps_do_not_depend_on_the_gaps_between_launches(gpu, mode):
    import torch

    from tests.test_gpu_parity import _ref_pose
    from tests.test_gpu_d3q27 import _case

    def make(**kw):
        return cases.moving_sphere_trt(Domain, **kw) if mode == "config" else _case(Domain, {"storage": "fp32", **kw})

    def pose(d, n):
        return cases.sphere_pose(d, n) if mode == "config" else _ref_pose(n)

    runs = [make(), make(stream=torch.cuda.Stream()), make()]
    try:
        for n in range(1, 30):
            for k, d in enumerate(runs):
                d.update_body(*pose(d, n))
                d.step(1)
                if k == 2:
                    d.synchronize()
        f = [d.populations() for d in runs]
        assert np.array_equal(f[0], f[1]) and np.array_equal(f[0], f[2])
    finally:
        for d in runs:
            d.close()

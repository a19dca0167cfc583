"""The halo-tile convolution (nn_conv3d_fwd, tcgen05) at the sizes where its tiling can go
wrong: planes along R that do not divide the box, a P axis shorter than, equal to and longer
than its 16 rows, y and z in either role, one and several 16-channel slices, weights that stay
in shared memory and weights that stream, more tiles than SMs, and unaligned tensors (which
take the warp tiles).

Tolerance: FP32 accumulation of exact BF16 products and one rounding to BF16, at most 2^-9 of
each value, hence of the 2-norm; 2^-12 of the norm on top covers the FP32 sums."""
import numpy as np
import pytest

from lbm3d_bb_b200 import unet as N
from oracle import unet_ref as U
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -9 + 2.0 ** -12


def _bf16(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda().bfloat16()


def _run(shape, cin, cout, relu, with_bias=True, shift=0):
    """Convolution of seeded data; `shift` elements of misalignment of the input tensor."""
    import torch

    rng = np.random.default_rng(sum(shape) * 100 + cin + cout)
    x = U.to_bf16(rng.standard_normal(shape + (cin,)))
    w = U.to_bf16(rng.standard_normal((27, cout, cin)) / np.sqrt(27 * cin))
    b = rng.standard_normal(cout).astype(np.float32) * 0.1 if with_bias else np.zeros(cout, np.float32)
    flat = torch.zeros(x.size + 8, dtype=torch.bfloat16, device="cuda")
    xd = flat[shift:shift + x.size].view(shape + (cin,))
    xd.copy_(_bf16(x))
    y = torch.full(shape + (cout,), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops = N.Ops()
    ops.conv(xd, _bf16(w), torch.from_numpy(b).cuda() if with_bias else None, y, shape, cin, cout, relu)
    N.tc_status()
    ref = U.conv(x, w, b)
    return y.float().cpu().numpy().astype(np.float64), np.maximum(ref, 0) if relu else ref


@pytest.mark.parametrize("shape,cin,cout", [
    ((1, 1, 1, 16), 16, 16),      # one tile, every neighbour outside
    ((1, 16, 16, 16), 16, 16),    # exactly one row of P
    ((1, 17, 15, 32), 16, 32),    # y short of P, z one past it
    ((1, 15, 17, 32), 32, 16),    # the other way round
    ((1, 3, 33, 16), 48, 16),     # three slices, P with a remainder of one
    ((2, 33, 3, 16), 16, 48),     # z is the longer axis: it takes the role of P
    ((1, 9, 20, 48), 64, 64),     # weights stream with the slices
    ((1, 5, 18, 16), 96, 32),     # six slices, weights resident
    ((1, 7, 19, 32), 32, 96),     # two output planes per MMA
    ((3, 40, 37, 64), 16, 16),    # more tiles than SMs: both accumulators and stages in turn
    ((2, 24, 40, 64), 96, 32),    # the same with slices
    ((1, 6, 250, 16), 16, 64),
])
def test_halo_conv(gpu, shape, cin, cout):
    got, ref = _run(shape, cin, cout, relu=(cin != 16))
    assert np.isfinite(got).all()
    assert rel_l2(got, ref) <= TOL


def test_halo_conv_without_bias(gpu):
    got, ref = _run((1, 6, 18, 32), 32, 32, relu=False, with_bias=False)
    assert rel_l2(got, ref) <= TOL


@pytest.mark.parametrize("cout", [16, 32])
def test_unaligned_input_takes_the_warp_tiles(gpu, cout):
    got, ref = _run((1, 4, 5, 32), 16, cout, relu=True, shift=2)  # 4-byte aligned only
    assert rel_l2(got, ref) <= TOL


@pytest.mark.parametrize("shape,cin,cout", [
    ((1, 1, 1, 16), 16, 16),     # one voxel row: every tap but the x ones outside
    ((1, 2, 3, 20), 16, 32),     # x not a multiple of the 16-voxel K step
    ((2, 5, 17, 32), 32, 32),    # planes of two samples side by side, y past a tile
    ((1, 9, 4, 48), 48, 16),     # three input slices
    ((1, 17, 6, 16), 96, 64),    # several input slices and output blocks
    ((3, 40, 37, 64), 16, 16),   # several tiles per block, z and y remainders
    ((2, 24, 40, 64), 64, 64),
])
def test_weight_gradient_tiles(gpu, shape, cin, cout):
    """FP32 sums of exact BF16 products, added onto what dw holds (tolerance of the layer tests)."""
    import torch

    rng = np.random.default_rng(sum(shape) + cin + cout)
    x = U.to_bf16(rng.standard_normal(shape + (cin,)))
    dy = U.to_bf16(rng.standard_normal(shape + (cout,)))
    start = rng.standard_normal((27, cout, cin)).astype(np.float32)
    _, ref, _ = U.conv_bwd(x, np.zeros((27, cout, cin)), dy)
    dw = torch.from_numpy(start).cuda()
    N.Ops().bwd_weight(_bf16(x), _bf16(dy), dw, shape, cin, cout)
    N.tc_status()
    assert rel_l2(dw.cpu().numpy(), start + ref) <= 1e-5

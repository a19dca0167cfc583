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


@pytest.mark.parametrize("c", [16, 32, 48, 4])
@pytest.mark.parametrize("shift", [0, 2])
def test_elementwise_forms(gpu, c, shift):
    """Grouped and one-element forms of the elementwise kernels (4 channels and misaligned
    tensors take the latter) on a box with a ragged row: copies and maxima exactly, sums to the
    BF16 rounding of the stored result (2^-9) or FP32 summation (1e-5)."""
    import torch

    ops = N.Ops()
    shape = (3, 2, 4, 22)
    coarse = (3, 1, 2, 11)
    rng = np.random.default_rng(c + shift)

    def dev(a):
        flat = torch.zeros(a.size + 8, dtype=torch.bfloat16, device="cuda")
        t = flat[shift:shift + a.size].view(a.shape)
        t.copy_(_bf16(a))
        return t

    def host(t):
        return t.float().cpu().numpy().astype(np.float64)

    x, y, dp = (U.to_bf16(rng.standard_normal(s + (c,))) for s in (shape, shape, coarse))
    p = dev(np.zeros(coarse + (c,)))
    ops.pool(dev(x), p, shape, c)
    assert rel_l2(host(p), U.pool(x)) <= 2.0 ** -8
    for acc in (False, True):
        g = dev(x)
        ops.pool_bwd(dev(dp), g, shape, c, acc)
        assert rel_l2(host(g), U.pool_bwd(dp) + (x if acc else 0)) <= 2.0 ** -8
    cat = dev(np.zeros(shape + (2 * c,)))
    ops.up_cat(dev(dp), dev(x), cat, shape, c, c)
    assert np.array_equal(host(cat), np.concatenate([U.up(dp), x], axis=-1))
    dcat = np.concatenate([y, x], axis=-1)
    dlow, dskip = dev(np.zeros(coarse + (c,))), dev(np.zeros(shape + (c,)))
    ops.up_cat_bwd(dev(dcat), dlow, dskip, shape, c, c)
    assert rel_l2(host(dlow), U.up_bwd(y)) <= 2.0 ** -8
    assert np.array_equal(host(dskip), x)
    g = dev(x)
    ops.relu_bwd(g, dev(y))
    assert np.array_equal(host(g), x * (y > 0))
    db = torch.ones(c, device="cuda")
    ops.bias_grad(dev(x), db, int(np.prod(shape)), c)
    assert rel_l2(host(db), 1 + x.reshape(-1, c).sum(0)) <= 1e-5


@pytest.mark.parametrize("cpad,ct", [(16, 4), (16, 3), (8, 4)])
def test_masked_loss_forms(gpu, cpad, ct):
    import torch

    vox = 70001  # a ragged last block, several voxels per thread of the grid at most
    rng = np.random.default_rng(cpad + ct)
    out, t = U.to_bf16(rng.standard_normal((vox, cpad))), rng.standard_normal((vox, ct)).astype(np.float32)
    mask, cw = (rng.random(vox) > 0.3).astype(np.uint8), (0.5 + rng.random(ct)).astype(np.float32)
    count = float(mask.sum())
    od = _bf16(out)
    dout = torch.full((vox, cpad), 7.0, dtype=torch.bfloat16, device="cuda")
    loss = torch.ones(1, dtype=torch.float64, device="cuda")
    L, dev = N.lib(), lambda a: torch.from_numpy(a).cuda()
    td, md, cd = dev(t), dev(mask), dev(cw)
    assert L.nn_mse(od.data_ptr(), td.data_ptr(), md.data_ptr(), cd.data_ptr(), dout.data_ptr(), loss.data_ptr(), vox,
                    cpad, ct, count, None) == 0
    d = (out[:, :ct].astype(np.float32) - t).astype(np.float64) * mask[:, None]
    ref = np.zeros((vox, cpad))
    ref[:, :ct] = 2 * cw * d / count
    assert abs(float(loss) - 1 - (cw * d * d).sum() / count) <= 1e-12 * vox
    assert rel_l2(dout.float().cpu().numpy(), ref) <= 2.0 ** -8


@pytest.mark.parametrize("replaced", [None, "W", "G"])
def test_optimiser_on_the_flat_buffers(gpu, replaced):
    """One launch over the flat buffers and one per tensor (taken when a tensor was replaced by the
    caller): the same bits."""
    import torch

    nets = [N.UNet3D(16, seed=3) for _ in range(2)]
    key = "d2b.w"
    if replaced:
        getattr(nets[0], replaced)[key] = getattr(nets[0], replaced)[key].clone()
    else:  # the per-tensor form as the reference
        nets[1].M[key] = nets[1].M[key].clone()
    for step in range(3):
        for net in nets:
            net.zero_grad()
            assert all(float(g.abs().max()) == 0 for g in net.G.values())
            gen = torch.Generator(device="cuda").manual_seed(step)
            for k in sorted(net.G):
                net.G[k].copy_(torch.randn(net.G[k].shape, device="cuda", generator=gen))
            net.adam_step(lr=1e-2)
    for k in nets[0].W:
        assert torch.equal(nets[0].W[k], nets[1].W[k])
    for k in nets[0].Wb:
        assert torch.equal(nets[0].Wb[k], nets[1].Wb[k])
        assert torch.equal(nets[0].Wb[k], nets[0].W[k + ".w"].bfloat16())


@pytest.mark.parametrize("shape,cu,cs,cout", [((1, 2, 2, 16), 32, 16, 16), ((2, 6, 18, 32), 64, 32, 32),
                                              ((1, 34, 4, 16), 32, 16, 32), ((2, 20, 34, 64), 32, 16, 16)])
def test_convolution_of_an_upsampled_concatenation(gpu, shape, cu, cs, cout):
    """The same bits as nn_up2_concat followed by nn_conv3d_fwd; refused by the other engines."""
    import torch

    ops = N.Ops()
    rng = np.random.default_rng(sum(shape) + cu)
    n, d, h, w = shape
    low, skip = (_bf16(rng.standard_normal(s)) for s in ((n, d // 2, h // 2, w // 2, cu), shape + (cs,)))
    wt, b = _bf16(rng.standard_normal((27, cout, cu + cs)) / 20), torch.from_numpy(rng.standard_normal(cout).astype(np.float32)).cuda()
    cat, y0, y1 = (torch.empty(shape + (c,), dtype=torch.bfloat16, device="cuda") for c in (cu + cs, cout, cout))
    ops.up_cat(low, skip, cat, shape, cu, cs)
    ops.conv(cat, wt, b, y0, shape, cu + cs, cout, True)
    assert ops.conv_up_cat(low, skip, wt, b, y1, shape, cu, cs, cout, True)
    N.tc_status()
    assert torch.equal(y0, y1)
    for engine in ("mma", "tcgen05-tma"):
        prev = N.set_conv_engine(engine)
        try:
            assert not ops.conv_up_cat(low, skip, wt, b, y1, shape, cu, cs, cout, True)
        finally:
            N.set_conv_engine(prev)

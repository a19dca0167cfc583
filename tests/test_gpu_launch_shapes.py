"""Block shapes that a program sets (lbm_set_launch, LBM3D_BLOCK) and the kernels that serve them: a
refused launch is an error of that call and of no later one, boxes with very many rows run, and a
set shape is the shape of the step."""
import re

import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from lbm3d_bb_b200._capi import LbmError
from tests import cases
from tests.kernel_names import launched

pytestmark = pytest.mark.gpu

CHANNEL = ("inlet", "pressure", "wall", "wall", "wall", "wall")


def _tall(storage="fp64"):
    """Rows of four cells; more rows than a grid has blocks along y."""
    d = Domain(4, 70000, 3, storage=storage, omega_p=1.3, accel=(1e-5, 2e-5, 0.0))
    rng = np.random.default_rng(8)
    d.init_equilibrium(u=0.02 * rng.standard_normal(d.N), w=0.02 * rng.standard_normal(d.N))
    return d


def test_a_refused_launch_is_no_later_calls_error(gpu):
    import torch

    a, b = _tall(), _tall()
    try:
        shape = a.launch()
        a.set_launch(32, 1)  # 70000 blocks along y
        with pytest.raises(LbmError, match="invalid"):
            a.step(1)
        assert torch.ones(3, device="cuda").add_(1).sum().item() == 6.0
        with pytest.raises(LbmError, match="invalid"):
            a.step(1)
        b.macros()
        a.set_launch(*shape)
        for d in (a, b):
            d.step(3)
        assert np.array_equal(a.populations(), b.populations())
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("storage", ["fp32", "fp16dev"])
def test_more_rows_than_a_grid_has_blocks(gpu, storage, monkeypatch):
    """With blocks of two rows a box of 65600 rows is initialised, stepped and exported, whatever
    kernels serve it: the same state as with the one-cell kernel."""
    import torch

    out = []
    for pair in (None, "0"):
        if pair is not None:
            monkeypatch.setenv("LBM3D_PAIR", pair)
        d = Domain(256, 65600, 3, storage=storage, omega_p=1.3, accel=(1e-5, 2e-5, -1e-5))
        d.set_launch(128, 2)
        d.add_spheres(np.array([[40.0, 30.0, 1.0, 3.0], [255.6, 65598.9, 1.5, 4.0], [90.0, 65540.0, 1.0, 5.0]]))
        d.init_equilibrium()
        d.step(3)
        m = torch.empty((4, d.N), dtype=torch.float32, device="cuda")
        d.macros_into(*m)
        out.append(m)
        torch.cuda.synchronize()
        d.close()
    assert (out[0][1:] != 0).any()
    tol = 1e-6 if storage == "fp32" else 2e-4  # a rounding of an FP16 deviation of order 0.1
    assert (out[0] - out[1]).abs().max().item() <= tol


def _step_kernels(d, steps=2):
    """Names of the step kernels that `steps` steps launch (even and odd phase)."""
    return {re.search(r"\b(aa_\w+_kernel)\b", n).group(1) for n in launched(lambda: d.step(steps))}


def test_a_set_shape_selects_the_one_cell_kernel(gpu):
    """Of boxes whose step has a kernel with a shape of its own; the library's shape gives it back."""
    d = Domain(160, 96, 96, storage="fp32", faces=CHANNEL, omega_p=1.3, face_u=[(0.03, 0.0, 0.0)] + [(0.0, 0.0, 0.0)] * 5)
    d.add_sphere((40.0, 48.0, 48.0), 9.0)
    d.init_equilibrium()
    try:
        own = d.launch()
        assert _step_kernels(d) == {"aa_rows_kernel"}
        for shape in ((32, 8), (160, 1)):
            assert shape != own
            d.set_launch(*shape)
            assert d.launch() == shape and _step_kernels(d) == {"aa_step_kernel"}
        d.set_launch(*own)
        assert _step_kernels(d) == {"aa_rows_kernel"}
    finally:
        d.close()


def test_block_variable_selects_the_one_cell_kernel(gpu, monkeypatch):
    for block, pair, kernel in (("32,8", None, "aa_step_kernel"), ("32,8", "1", "aa_rows_kernel"), (None, None, "aa_rows_kernel")):
        for name, value in (("LBM3D_BLOCK", block), ("LBM3D_PAIR", pair)):
            if value is None:
                monkeypatch.delenv(name, raising=False)
            else:
                monkeypatch.setenv(name, value)
        d = Domain(160, 96, 96, storage="fp32", faces=CHANNEL, omega_p=1.3)
        d.init_equilibrium()
        try:
            assert _step_kernels(d) == {kernel}
        finally:
            d.close()


def test_the_tuner_times_the_librarys_own_shape(gpu, tmp_path, monkeypatch):
    """Rows that fit no whole warps: the padded row is the library's shape and a candidate; when it
    is the fastest, the kernel that goes with it stays."""
    from lbm3d_bb_b200 import autotune

    monkeypatch.setenv("LBM3D_TUNE_CACHE", str(tmp_path / "shapes.json"))
    for nx in (70, 160, 96, 34):
        d = Domain(nx, 8, 8, storage="fp32")
        assert d.launch() in autotune.candidates(nx)
        d.close()
    d = Domain(160, 96, 96, storage="fp32", faces=CHANNEL, omega_p=1.3)
    d.init_equilibrium()
    own = d.launch()
    try:
        got = autotune.tune(d, timer=lambda: 0.0 if d.launch() == own else 1.0)
        assert got == own and _step_kernels(d) == {"aa_rows_kernel"}
    finally:
        d.close()


@pytest.mark.parametrize("pair,kernel", [(None, "aa_step_kernel"), ("0", "aa_step_kernel"), ("1", "aa_rows_kernel")])
def test_pair_variable_holds_with_a_moving_body(gpu, monkeypatch, pair, kernel):
    if pair is not None:
        monkeypatch.setenv("LBM3D_PAIR", pair)
    d = cases.moving_sphere_trt(Domain, storage="fp32")
    try:
        d.update_body(*cases.sphere_pose(d, 1))
        assert _step_kernels(d) == {kernel}
    finally:
        d.close()


@pytest.mark.parametrize("shape,faces,storage,kernel", [
    ((614, 614, 4), "channel", "fp32", "aa_step_kernel"),     # half of the rows on a z end
    ((614, 614, 4), "channel", "fp16dev", "aa_step_kernel"),
    ((614, 614, 4), "periodic", "fp32", "aa_rows_kernel"),
    ((354, 354, 12), "channel", "fp32", "aa_step_kernel"),    # a sixth
    ((354, 354, 12), "channel", "fp16dev", "aa_rows_kernel"),
    ((1200, 1200, 1), "channel", "fp32", "aa_step_kernel"),   # all of them
    ((252, 252, 24), "channel", "fp32", "aa_rows_kernel"),
    ((4, 600, 600), "channel", "fp16dev", "aa_step_kernel"),  # rows of a few cells
    ((12, 400, 360), "channel", "fp16dev", "aa_rows_kernel"),
    ((4, 1500, 1000), "channel", "fp16dev", "aa_rows_kernel"),
])
def test_boxes_of_end_rows_or_short_rows_keep_one_cell_per_thread(gpu, shape, faces, storage, kernel):
    d = Domain(*shape, storage=storage, faces=CHANNEL if faces == "channel" else ("periodic",) * 6, omega_p=1.3)
    d.init_equilibrium()
    try:
        assert _step_kernels(d) == {kernel}
    finally:
        d.close()


@pytest.mark.parametrize("radius,faces,storage,kernel,move", [
    (8.0, "periodic", "fp32", "aa_rows_kernel", None), (38.0, "periodic", "fp32", "aa_step_kernel", False),
    (8.0, "channel", "fp32", "aa_step_kernel", True), (38.0, "channel", "fp32", "aa_step_kernel", True),
    (8.0, "channel", "fp16dev", "aa_step_kernel", True), (38.0, "channel", "fp16dev", "aa_step_kernel", False)])
def test_kernels_of_large_moving_bodies(gpu, radius, faces, storage, kernel, move):
    """A body that fills the box keeps the general path for its links, but where the fast one wins."""
    d = Domain(114, 114, 114, storage=storage, faces=CHANNEL if faces == "channel" else ("periodic",) * 6, omega_p=1.3)
    d.add_sphere((57.0, 57.0, 57.0), radius, moving=True)
    d.init_equilibrium()
    try:
        names = launched(lambda: d.step(2))
        assert all(kernel in name for name in names), names
        if move is not None:  # the last template argument
            assert all(re.search(r"(true|false)>\(", name).group(1) == str(move).lower() for name in names), names
    finally:
        d.close()


@pytest.mark.parametrize("shape,block", [((161, 2, 40), (64, 2)), ((161, 5, 40), (64, 2)), ((161, 6, 40), (64, 2)),
                                         ((161, 12, 40), (32, 4)), ((1000, 1, 3), None), ((384, 3, 9), (128, 1)), ((300, 200, 3), (32, 4))])
def test_blocks_have_no_more_rows_than_boxes_fill(gpu, shape, block):
    if shape[1] < 2:
        with pytest.raises(LbmError):
            Domain(*shape, storage="fp64", faces=CHANNEL)
        return
    d = Domain(*shape, storage="fp64", faces=CHANNEL)
    try:
        assert d.launch() == block
    finally:
        d.close()


def _export_kernels(d):
    import torch

    m = torch.empty((4, (d.N + 7) // 8 * 8), device="cuda")
    names = launched(lambda: d.macros_into(*[m[k, :d.N] for k in range(4)]))
    return {k for k in ("aa_export_kernel", "aa_export_pair_kernel") for n in names if k in n}


@pytest.mark.parametrize("shape,faces,storage,pairs", [
    ((64, 128, 128), "channel", "fp16dev", False),   # a face in every warp
    ((64, 128, 128), "periodic", "fp16dev", True),
    ((34, 150, 100), "channel", "fp16dev", True),    # idle lanes in the other kernel
    ((512, 64, 64), "channel", "fp32", True),
    ((256, 80, 80), "channel", "fp64", False),
    ((256, 80, 80), "periodic", "fp64", True),
    ((600, 600, 1), "periodic", "fp64", False),      # every row on an end
])
def test_export_after_an_odd_number_of_steps(gpu, shape, faces, storage, pairs):
    d = Domain(*shape, storage=storage, faces=CHANNEL if faces == "channel" else ("periodic",) * 6, omega_p=1.3)
    d.init_equilibrium()
    d.step(1)
    try:
        assert _export_kernels(d) == {"aa_export_pair_kernel" if pairs else "aa_export_kernel"}
    finally:
        d.close()

"""Two cells per thread on rows of any even length and any faces (aa_rows_kernel; LBM3D_PAIR=1
takes it at every size) against the FP64 oracle: the shortest rows, rows whose pairs straddle
warps and blocks, every face kind on the x faces, periodic and walled y and z, bodies that
touch the faces, body forces, BGK and TRT; and against the one-cell kernel (LBM3D_PAIR=0)
with a moving body and in FP16-deviation storage.

Tolerance of FP32 against FP64: a population is rounded about ten times per step (2^-24 each),
so 1e-6 per step at most, in fact its square root."""
import os

import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from oracle.oracle import OracleDomain
from tests import cases
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu

FACES = {
    "periodic": ("periodic",) * 6,
    "outflow": ("inlet", "outflow", "wall", "wall", "wall", "wall"),
    "pressure": ("inlet", "pressure", "periodic", "periodic", "wall", "wall"),
    "walls_x": ("wall", "wall", "periodic", "periodic", "periodic", "periodic"),
    "periodic_x": ("periodic", "periodic", "wall", "wall", "inlet", "pressure"),
}


def _pair(value, fn):
    old = os.environ.get("LBM3D_PAIR")
    os.environ["LBM3D_PAIR"] = value
    try:
        return fn()
    finally:
        if old is None:
            del os.environ["LBM3D_PAIR"]
        else:
            os.environ["LBM3D_PAIR"] = old


def _case(cls, shape, faces, coll, accel=(0.0, 0.0, 0.0), **kw):
    nx, ny, nz = shape
    fu = [(0.03, 0.0, 0.0), (0.0, 0.0, 0.0)] + [(0.01, 0.0, 0.0)] * 2 + [(0.0, 0.0, 0.02), (0.0, 0.0, 0.0)]
    d = cls(nx, ny, nz, collision=coll, faces=FACES[faces], omega_p=1.0 / 0.7, omega_m=1.0 / (0.5 + 0.1875 / 0.2),
            face_u=fu, accel=accel, **kw)
    # one sphere cut by the low x and y faces (or the wrap), one inside
    if min(nx, ny, nz) >= 6:
        d.add_spheres(np.array([[0.7, 1.2, nz / 2, 2.3], [nx - 1.5, ny / 2, nz / 2, 1.9]]))
    rng = np.random.default_rng(nx * 100 + ny)
    u = 0.02 * rng.standard_normal((3, nx * ny * nz))
    d.init_equilibrium(u=u[0], v=u[1], w=u[2])
    return d


@pytest.mark.parametrize("coll", ["BGK", "TRT"])
@pytest.mark.parametrize("faces", sorted(FACES))
@pytest.mark.parametrize("shape", [(4, 5, 4), (6, 7, 6), (34, 9, 7), (130, 6, 6), (258, 7, 8)])
def test_rows_fp32_vs_oracle(gpu, oracle_lib, shape, faces, coll):
    steps = 5
    accel = (1e-5, 0.0, 0.0) if faces == "walls_x" else (2e-5, -1e-5, 3e-5) if faces == "periodic" else (0.0, 0.0, 0.0)
    g = _pair("1", lambda: _case(Domain, shape, faces, coll, accel, storage="fp32"))
    o = _case(OracleDomain, shape, faces, coll, accel, precision="fp64")
    try:
        for n in range(steps):
            g.step(1)
            o.step(1)
            assert rel_l2(g.populations(), o.populations()) <= 1e-6 * (n + 1), n
        fg, fo = g.force_history(1, steps), o.force_history(1, steps)
        assert np.linalg.norm(fg - fo) <= 1e-5 * np.linalg.norm(fo) + 1e-6
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("nx", [36, 66])
def test_rows_moving_body_vs_one_cell(gpu, nx):
    """Nodes are covered and uncovered on the way.  The wall moves faster than the lattice's
    speed of sound, so the flow itself diverges and rounding grows with it (FP32 against the
    oracle: 1e-6 after four steps, 5e-5 after six, with either kernel and with the oracle in
    FP32): the one-cell kernel is the reference."""
    kw = dict(nx=nx, ny=20, nz=18, r=3.3, amp=5.0, period=40.0, storage="fp32")
    g, o = (_pair(v, lambda: cases.moving_sphere_trt(Domain, **kw)) for v in ("1", "0"))
    try:
        for n in range(1, 13):
            for d in (g, o):
                d.update_body(*cases.sphere_pose(d, n))
                d.step(1)
            assert rel_l2(g.populations(), o.populations()) <= 1e-6 * (n + 1), n
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("coll", ["BGK", "TRT"])
@pytest.mark.parametrize("faces", sorted(FACES))
def test_rows_fp16dev_vs_one_cell(gpu, faces, coll):
    """The same per-cell arithmetic: what differs is at most a last-bit FP32 difference before
    the rounding to FP16 (2^-11 of a deviation of order 0.05)."""
    runs = [_pair(v, lambda: _case(Domain, (66, 9, 8), faces, coll, storage="fp16dev")) for v in ("1", "0")]
    try:
        for d in runs:
            d.step(6)
        a, b = (d.populations() for d in runs)
        assert rel_l2(a, b) <= 1e-4
    finally:
        for d in runs:
            d.close()


def test_odd_rows_take_the_one_cell_kernel(gpu, oracle_lib):
    g = _pair("1", lambda: _case(Domain, (35, 8, 7), "outflow", "BGK", storage="fp32"))
    o = _case(OracleDomain, (35, 8, 7), "outflow", "BGK", precision="fp64")
    try:
        for d in (g, o):
            d.step(4)
        assert rel_l2(g.populations(), o.populations()) <= 4e-6
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("shape,center", [((24, 16, 18), (0.7, 8.1, 17.2)), ((17, 40, 19), (45.0, 39.0, -30.4)),
                                          ((70, 9, 10), (35.2, 4.4, 5.1))])
def test_body_flags_across_wraps(gpu, oracle_lib, shape, center):
    """A moving sphere's flags and links, bit for bit: boxes that wrap, that start periods away
    from the origin, that are as long as the axis, that need several tiles."""
    from lbm3d_bb_b200 import abi

    runs = []
    for cls, kw in ((Domain, dict(storage="fp32")), (OracleDomain, dict(precision="fp64"))):
        d = cls(*shape, collision="BGK", faces=("periodic",) * 6, omega_p=1.2, **kw)
        d.add_spheres(np.array([[shape[0] / 2, 3.0, 4.0, 2.2]]))
        d.add_body(abi.make_body(abi.BODY_SPHERE, center, radius=4.3, moving=True))
        d.init_equilibrium()
        runs.append(d)
    try:
        for n in range(6):
            c = tuple(v + 0.45 * n for v in center)
            for d in runs:
                d.update_body(abi.make_pose(center=c), abi.make_pose(center=c))
            (fa, ba), (fb, bb) = (d.flags() for d in runs)
            assert np.array_equal(fa, fb) and np.array_equal(ba, bb), n
            for x, y in zip(runs[0].links(), runs[1].links()):
                assert np.array_equal(x, y), n
            for d in runs:
                d.step(1)
        assert rel_l2(runs[0].populations(), runs[1].populations()) <= 6e-6
    finally:
        for d in runs:
            d.close()

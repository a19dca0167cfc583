"""Flags, boundary flags and links of a moving body in reference mode, bit for bit against the
oracle: the box is periodic along z for the body, so a body may lie across the z ends or be given
periods away from the box, but the nodes on the two sides of the wrap are not neighbours; a static
body in the moving one's way keeps its nodes."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain, abi
from oracle.oracle import OracleDomain

pytestmark = pytest.mark.gpu

ROT = (0.8, -0.6, 0.0, 0.6, 0.8, 0.0, 0.0, 0.0, 1.0)


def _body(kind, center):
    if kind == "sphere":
        return abi.make_body(abi.BODY_SPHERE, center, radius=6.0, moving=True)
    return abi.make_body(abi.BODY_ELLIPSOID, center, semi=(3.0, 5.5, 6.5), rot=ROT, moving=True)


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("kind", ["sphere", "ellipsoid"])
@pytest.mark.parametrize("nz,z0", [(40, 9.0), (40, 37.0), (40, 20.0), (33, 0.4), (16, 15.6), (41, 41.0 * 3 + 2.0),
                                   (37, -37.0 * 2 + 35.5), (8, 4.0)])
def test_reference_mode_flags_across_the_z_ends(gpu, oracle_lib, nz, z0, kind, q):
    runs = []
    for cls, kw in ((Domain, dict(storage="fp32")), (OracleDomain, dict(precision="fp32"))):
        d = cls(30, 26, nz, mode="reference", collision="BGK", omega_p=1.2, u_inf=(0.02, 0.0, 0.0), q=q, **kw)
        d.add_body(abi.make_body(abi.BODY_SPHERE, (13.0, 12.0, 1.5), radius=2.0))
        d.add_body(_body(kind, (14.2, 13.1, z0)))
        d.init_equilibrium()
        runs.append(d)
    g, o = runs
    try:
        for n in range(6):
            pose = abi.make_pose(center=(14.2 - 0.3 * n, 13.1, z0 + 1.7 * n), rot=ROT)
            for d in runs:
                d.update_body(pose, pose)
            for a, b in zip((*g.flags(), *g.links()), (*o.flags(), *o.links())):
                assert np.array_equal(a, b), n
            assert g.flags()[0].sum() > 0
            for d in runs:
                d.step(1)
    finally:
        for d in runs:
            d.close()


@pytest.mark.parametrize("mode,q", [("config", 19), ("reference", 19), ("reference", 27)])
@pytest.mark.parametrize("radius,launches", [(13.0, 1), (24.0, 2)])
def test_boxes_of_one_and_of_two_launches(gpu, oracle_lib, mode, q, radius, launches):
    """A large body's flags come from two kernels, a small one's from one: the same rules."""
    kw = dict(mode="reference", u_inf=(0.02, 0.0, 0.0), q=q) if mode == "reference" else dict(faces=("inlet", "outflow", "wall", "wall", "periodic", "periodic"))
    runs = []
    for cls, precision in ((Domain, dict(storage="fp32")), (OracleDomain, dict(precision="fp32"))):
        d = cls(74, 66, 58, collision="BGK", omega_p=1.2, **kw, **precision)
        d.add_body(abi.make_body(abi.BODY_SPHERE, (13.0, 12.0, 1.5), radius=4.0))
        d.add_body(abi.make_body(abi.BODY_SPHERE, (33.2, 31.0, 50.3), radius=radius, moving=True))
        d.init_equilibrium()
        runs.append(d)
    g, o = runs
    try:
        for n in range(1, 4):
            pose = abi.make_pose(center=(33.2 - 0.4 * n, 31.0 + 0.3 * n, 50.3 + 1.1 * n))
            before = g.launch_count
            for d in runs:
                d.update_body(pose, pose)
                d.step(1)
            assert g.launch_count - before == launches + 1, n
            for a, b in zip((*g.flags(), *g.links()), (*o.flags(), *o.links())):
                assert np.array_equal(a, b), n
    finally:
        for d in runs:
            d.close()

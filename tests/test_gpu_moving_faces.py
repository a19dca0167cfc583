"""A moving body one node away from a face: the nodes between them take the face's value of the
populations that leave the box and the moving wall's value of those that leave the body, each made
of the same post-collision state.  Every face of the box, every kind of face, an edge of two
faces; FP64 (where the only difference to the oracle is the order of a few sums: 1e-12 of the
field) and FP32 (a population is rounded about ten times per step, 2^-24 each: 1e-6 per step)
against the FP64 oracle after every step, odd and even."""
import math

import numpy as np
import pytest

from lbm3d_bb_b200 import Domain, abi
from oracle.oracle import OracleDomain
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu

SHAPE = (26, 22, 20)
R = 4.6
KINDS = ("outflow", "pressure", "wall", "inlet")


def _center(faces_near):
    """One node between the body and each of these faces (a node lies at index + 0.5)."""
    c = [SHAPE[0] / 2 + 0.2, SHAPE[1] / 2 - 0.1, SHAPE[2] / 2 + 0.3]
    for f in faces_near:
        a, high = f // 2, f % 2
        c[a] = SHAPE[a] - 1.5 - R + 0.15 if high else 1.5 + R - 0.15
    return c


def _make(cls, faces, near, coll, **kw):
    u = [(0.04, 0.01, -0.02)] * 6
    d = cls(*SHAPE, collision=coll, faces=faces, face_u=u, omega_p=1.0 / 0.7, omega_m=1.0 / (0.5 + 0.1875 / 0.2), **kw)
    d.add_body(abi.make_body(abi.BODY_SPHERE, _center(near), radius=R, moving=True))
    rng = np.random.default_rng(5)
    v = 0.02 * rng.standard_normal((3, d.N))
    d.init_equilibrium(u=v[0], v=v[1], w=v[2])
    return d


def _pose(near, n):
    """The body shakes by a fraction of a cell (its solid nodes stay the same on most steps) and
    turns; normal and tangential wall speeds of the order of 0.05."""
    w = 2.0 * math.pi / 9.0
    c = _center(near)
    s = 0.07 * math.sin(w * n)
    v = 0.07 * w * math.cos(w * n)
    return abi.make_pose(center=[x + s for x in c], vel=(v, v, v), omega=(0.004, -0.003, 0.005))


def _compare(faces, near, coll, storage):
    g = _make(Domain, faces, near, coll, storage=storage)
    o = _make(OracleDomain, faces, near, coll, precision="fp64")
    tol = 1e-12 if storage == "fp64" else 1e-6
    try:
        for n in range(1, 13):
            for d in (g, o):
                d.update_body(_pose(near, n - 1.0), _pose(near, n - 0.5))
                d.step(1)
            assert rel_l2(g.populations(), o.populations()) <= tol * (n + 1), n
        fg, fo = g.force_history(1, 12), o.force_history(1, 12)
        assert np.linalg.norm(fg - fo) <= 100 * tol * np.linalg.norm(fo) + 1e-10
    finally:
        g.close()
        o.close()


@pytest.mark.parametrize("storage,coll", [("fp64", "BGK"), ("fp64", "TRT"), ("fp32", "TRT")])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("face", range(6))
def test_body_beside_a_face(gpu, oracle_lib, face, kind, storage, coll):
    faces = ["wall"] * 6
    faces[face ^ 1] = "inlet"
    faces[face] = kind
    _compare(tuple(faces), (face,), coll, storage)


@pytest.mark.parametrize("near", [(1, 2), (0, 5), (3, 4), (1, 3, 5)])
def test_body_beside_an_edge(gpu, oracle_lib, near):
    faces = ["wall"] * 6
    for f in near:
        faces[f] = "outflow"
    _compare(tuple(faces), near, "TRT", "fp64")

"""The force on a moving body beside a node whose populations are lost: the components that are NaN
or infinite are those of the oracle, also for a node that touches the body with one link only."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain, abi
from oracle.oracle import OracleDomain
from tests import cases

pytestmark = pytest.mark.gpu

SHAPE = (30, 22, 20)


def _make(cls, f=None, **kw):
    d = cls(*SHAPE, collision="BGK", faces=cases.INLET_CHANNEL, omega_p=1.3, face_u=cases.face_u_inlet(0.03), **kw)
    d.add_body(abi.make_body(abi.BODY_SPHERE, (12.1, 11.0, 9.8), radius=4.6, moving=True))
    d.init_equilibrium()
    if f is not None:
        with np.errstate(all="ignore"):
            d.set_populations(f)
    return d


@pytest.mark.parametrize("steps", [1, 2])
def test_force_of_a_lost_node(gpu, oracle_lib, steps):
    d = _make(Domain, storage="fp64")
    ptr, lidx, dirs = d.links()
    d.close()
    links = np.diff(ptr) if len(ptr) == np.prod(SHAPE) + 1 else np.bincount(lidx - 1, minlength=int(np.prod(SHAPE)))
    single = np.flatnonzero(links == 1)
    assert single.size > 0
    pose = abi.make_pose(center=(12.1, 11.0, 9.8), vel=(0.01, 0.02, -0.015), omega=(0.001, 0.0, 0.002))
    for node in (int(single[0]), int(single[-1]), int(np.argmax(links))):
        f = np.repeat(np.array([1 / 18] * 6 + [1 / 36] * 12 + [1 / 3])[:, None], int(np.prod(SHAPE)), 1)
        f[18, node] = np.inf
        out = []
        for cls, kw in ((Domain, dict(storage="fp64")), (OracleDomain, dict(precision="fp64"))):
            d = _make(cls, f, **kw)
            for _ in range(steps):
                d.update_body(pose, pose)
                d.step(1)
            out.append(d.force(steps))
            d.close()
        g, o = out
        assert np.array_equal(np.isnan(g), np.isnan(o)) and np.array_equal(np.isinf(g), np.isinf(o)), (node, g, o)
        assert np.isnan(o).any()

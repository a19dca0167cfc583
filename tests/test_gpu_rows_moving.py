"""Two cells per thread (aa_rows_kernel) where boxes take it by themselves and a body moves or the
box is a z-slab, against the one-cell kernel (LBM3D_PAIR=0): the same arithmetic per cell, so FP32
differs by a last bit before each store at most (2^-24, about ten per step: 1e-6 per step), FP16
deviations by the rounding of one (2^-11 of a deviation of order 0.05)."""
import re

import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from lbm3d_bb_b200.slab import SlabDomain, SlabGroup
from tests import cases
from tests.cases import rel_l2
from tests.kernel_names import launched

pytestmark = pytest.mark.gpu


def _kernels(run):
    return {re.search(r"\b(aa_\w+_kernel)\b", n).group(1) for n in launched(run)}


def _channel(shape, storage, coll):
    nx, ny, nz = shape
    om_m = 1.0 / (0.5 + 0.1875 / (1.0 / 1.4 - 0.5)) if coll == "TRT" else None
    d = Domain(nx, ny, nz, collision=coll, storage=storage, faces=cases.INLET_CHANNEL, omega_p=1.4, omega_m=om_m,
               face_u=cases.face_u_inlet(0.03))
    from lbm3d_bb_b200 import abi

    d.add_body(abi.make_body(abi.BODY_SPHERE, (nx / 3.0, ny / 2.0, nz / 2.0), radius=9.3, moving=True))
    d.init_equilibrium()
    d._motion = (nx / 3.0, ny / 2.0, nz / 2.0, 2.0, 150.0)  # wall speed 0.08
    return d


@pytest.mark.parametrize("shape,storage,coll", [((250, 160, 152), "fp32", "BGK"), ((256, 154, 156), "fp32", "TRT"),
                                                ((162, 112, 112), "fp16dev", "BGK"), ((252, 156, 154), "fp16dev", "TRT")])
def test_moving_body_in_a_large_channel(gpu, monkeypatch, shape, storage, coll):
    fields, forces, names = [], [], []
    for pair, kernel in ((None, "aa_rows_kernel"), ("0", "aa_step_kernel")):
        if pair is not None:
            monkeypatch.setenv("LBM3D_PAIR", pair)
        d = _channel(shape, storage, coll)

        for n in range(1, 13):
            d.update_body(*cases.sphere_pose(d, n))
            d.step(1)
        fields.append(d.populations(np.float32))
        forces.append(d.force_history(1, 12))
        names.append((_kernels(lambda: d.step(2)), {kernel}))
        d.close()
    tol = 1e-6 * 12 if storage == "fp32" else 1e-4
    assert rel_l2(fields[0], fields[1]) <= tol
    assert np.linalg.norm(forces[0] - forces[1]) <= 100 * tol * np.linalg.norm(forces[1])
    assert all(got == want for got, want in names), names


@pytest.mark.parametrize("faces", [cases.PERIODIC, ("inlet", "pressure", "wall", "wall", "wall", "wall"),
                                   ("periodic", "periodic", "periodic", "periodic", "wall", "wall")])
@pytest.mark.parametrize("storage", ["fp32", "fp16dev"])
@pytest.mark.parametrize("parts", [2, 3])
def test_slabs_of_even_rows(gpu, monkeypatch, parts, storage, faces):
    """Slabs on the rows kernel against the undivided box on the one-cell kernel."""
    nx, ny, nz, steps = 26, 14, 31, 7
    spheres = np.array([[6.3, 7.1, 10.2, 4.2], [15.5, 9.4, 15.1, 3.6], [19.2, 4.8, 20.7, 3.9], [25.6, 12.2, 0.6, 3.4]])
    kw = dict(collision="TRT", storage=storage, faces=faces, omega_p=1.0 / 0.7, omega_m=1.0 / (0.5 + 0.1875 / 0.2),
              face_u=[(0.04, 0.0, 0.0)] + [(0.0, 0.0, 0.0)] * 5,
              accel=(1e-5, 0.0, 0.0) if faces[0] == "periodic" else (0.0, 0.0, 0.0))
    monkeypatch.setenv("LBM3D_PAIR", "1")
    slabs = [SlabDomain(nx, ny, nz, parts, r, **kw) for r in range(parts)]
    monkeypatch.setenv("LBM3D_PAIR", "0")
    full = Domain(nx, ny, nz, **kw)
    try:
        for d in (*slabs, full):
            d.add_spheres(spheres)
            d.init_equilibrium()
        g = SlabGroup(slabs)
        g.step(steps)
        full.step(steps)
        got = np.concatenate([s.populations() for s in slabs], axis=1)
        assert rel_l2(got, full.populations().reshape(19, nz, ny, nx)) <= (1e-6 * steps if storage == "fp32" else 1e-4)
        assert _kernels(lambda: g.step(2)) == {"aa_rows_kernel"}
        assert _kernels(lambda: full.step(2)) == {"aa_step_kernel"}
    finally:
        for d in (*slabs, full):
            d.close()

"""Moments exported two nodes at a time (lbm_get_macros into aligned device arrays) against the
one-node kernel (taken when an output array is not on a two-element word): the same values from
the same populations, in the plain layout (even step counts) and the swapped one (odd), for
rows of even and odd length, faces, wraps and solids on the box's edges, all storages and both
output types; and the force history across the end of its ring."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain

pytestmark = pytest.mark.gpu

CHANNEL = ("inlet", "pressure", "wall", "wall", "wall", "wall")


def _domain(shape, faces, storage, **kw):
    nx, ny, nz = shape
    d = Domain(nx, ny, nz, storage=storage, faces=faces, omega_p=1.3, accel=(1e-5, 2e-5, -1e-5) if faces[0] == "periodic" else (0, 0, 0),
               face_u=[(0.04, 0.0, 0.0)] + [(0.0, 0.0, 0.0)] * 5, **kw)
    d.add_spheres(np.array([[0.6, 1.1, nz / 2, 1.7], [nx / 2, ny - 1.2, nz - 0.9, 1.6]]))
    rng = np.random.default_rng(nx + ny)
    d.init_equilibrium(u=0.03 * rng.standard_normal(d.N), v=0.03 * rng.standard_normal(d.N))
    return d


@pytest.mark.parametrize("storage", ["fp32", "fp64", "fp16dev"])
@pytest.mark.parametrize("faces", [("periodic",) * 6, CHANNEL])
@pytest.mark.parametrize("shape", [(4, 5, 4), (6, 4, 3), (35, 6, 5), (130, 7, 6), (514, 3, 3)])
def test_pair_export_equals_node_export(gpu, shape, faces, storage):
    import torch

    d = _domain(shape, faces, storage)
    try:
        for _ in range(3):
            for dt in (torch.float32, torch.float64):
                a = torch.full((4, d.N + 2), -7.0, dtype=dt, device="cuda")
                b = torch.full((4, d.N + 3), -7.0, dtype=dt, device="cuda")
                base = a.view(-1)[: 4 * (d.N + d.N % 2)].view(4, -1)  # rows on two-element words
                d.macros_into(*[base[k, : d.N] for k in range(4)])
                d.macros_into(*[b[k, 1 + (k * (d.N + 3)) % 2:][: d.N] for k in range(4)])  # none of them
                got = [base[k, : d.N].cpu().numpy() for k in range(4)]
                ref = [b[k, 1 + (k * (d.N + 3)) % 2:][: d.N].cpu().numpy() for k in range(4)]
                for g, r in zip(got, ref):
                    assert np.array_equal(g, r)
                assert np.abs(got[1]).max() > 0
            d.step(1)
    finally:
        d.close()


def test_force_history_across_the_ring_end(gpu):
    d = _domain((24, 12, 12), CHANNEL, "fp64", force_history=5)
    try:
        one = []
        for n in range(1, 10):
            d.step(1)
            one.append(d.force(n))
        for first, count in ((5, 5), (6, 3), (9, 1), (7, 0)):
            assert np.array_equal(d.force_history(first, count), np.array(one[first - 1:first - 1 + count]).reshape(-1, 6))
        with pytest.raises(Exception):
            d.force_history(4, 5)
    finally:
        d.close()

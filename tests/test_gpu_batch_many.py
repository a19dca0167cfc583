"""Batches with so many work items that boxes without faces take the kernel with more warps and
fewer registers per SM (read from the kernel's name): the same domains stepped one by one.
Tolerances as for other batches: the two group cells into warps differently."""
import re

import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from lbm3d_bb_b200.batch import Batch
from tests import cases
from tests.cases import rel_l2
from tests.kernel_names import launched

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-13, "fp32": 1e-6, "fp16dev": 1e-4}


def _domain(k, storage, coll, faces):
    d = Domain(16, 16, 16, collision=coll, storage=storage, faces=faces, omega_p=1.4, omega_m=1.1 if coll == "TRT" else None,
               face_u=cases.face_u_inlet(0.03), accel=(1e-5, 0.0, 0.0) if faces[0] == "periodic" else (0.0, 0.0, 0.0))
    d.add_sphere((5.0 + 0.01 * k, 8.0, 7.5), 2.6)
    d.init_equilibrium()
    return d


@pytest.mark.parametrize("faces", [cases.PERIODIC, cases.INLET_CHANNEL], ids=["periodic", "channel"])
@pytest.mark.parametrize("storage,coll,few,many", [("fp16dev", "BGK", 5, 8), ("fp16dev", "TRT", 5, 8), ("fp32", "BGK", 5, 5),
                                                   ("fp32", "TRT", 5, 6), ("fp64", "BGK", 3, 3), ("fp64", "TRT", 3, 4)])
def test_register_budget_follows_the_work(gpu, storage, coll, few, many, faces):
    for count, blocks in ((4, few), (313, many if faces == cases.PERIODIC else few)):  # 32 items each
        domains = [_domain(k, storage, coll, faces) for k in range(count)]
        try:
            with Batch(domains) as b:
                b.step(3)
                b.synchronize()
            for k in (0, count - 1):
                one = _domain(k, storage, coll, faces)
                one.step(3)
                a, c = domains[k].populations(), one.populations()
                fa, fc = domains[k].force_history(1, 3), one.force_history(1, 3)
                one.close()
                assert rel_l2(a, c) <= TOL[storage]
                assert np.linalg.norm(fa[:, :3] - fc[:, :3]) <= 10 * TOL[storage] * np.linalg.norm(fc[:, :3]) + 1e-12
            with Batch(domains) as b:
                names = launched(lambda: b.step(2), "aa_batch_kernel")
            assert {int(re.search(r", (\d+)>\(", n).group(1)) for n in names} == {blocks}, names
        finally:
            for d in domains:
                d.close()

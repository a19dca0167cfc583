"""Block shapes that a program sets (lbm_set_launch): a refused launch is an error of that call and
of no later one."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from lbm3d_bb_b200._capi import LbmError

pytestmark = pytest.mark.gpu


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

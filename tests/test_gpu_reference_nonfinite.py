"""Populations that are not finite, or whose sums are not, in reference mode: the same values,
infinities and NaN as the oracle, bit for bit, in the moments and in the populations of the steps
that follow (a diverging run shows the same nodes as lost)."""
import numpy as np
import pytest

from lbm3d_bb_b200 import Domain
from oracle.oracle import OracleDomain

pytestmark = pytest.mark.gpu

SHAPE = (20, 12, 9)


def _populations(q, precision):
    """A gentle flow with single nodes replaced, far enough apart to stay apart for three steps."""
    rng = np.random.default_rng(4)
    nx, ny, nz = SHAPE
    f = 1.0 / q + 0.01 * rng.standard_normal((q, nz, ny, nx))
    f = f.astype(np.float32).astype(np.float64)
    big = 3e38 if precision == "fp32" else 1.5e308
    rest = q - 1
    f[0, 2, 5, 2] = np.inf  # enters one momentum
    f[rest, 6, 5, 6] = np.inf  # enters none
    f[7, 2, 5, 10] = -np.inf
    f[4, 6, 5, 14] = np.nan
    f[0, 2, 5, 17], f[1, 2, 5, 17] = big, -big  # momentum overflows, density does not
    f[0, 6, 1, 2], f[1, 6, 1, 2] = big, big  # density overflows, momentum does not
    f[:, 6, 9, 10] = 0.0  # no density
    f[2, 2, 1, 14], f[3, 2, 1, 14] = big / 4, big / 8  # a large velocity whose square overflows
    return f.reshape(q, -1)


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("coll", ["BGK", "TRT"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_non_finite_values_spread_as_in_the_oracle(gpu, oracle_lib, precision, coll, q):
    kw = dict(mode="reference", collision=coll, omega_p=1.25, omega_m=1.1, u_inf=(0.02, 0.0, 0.0), q=q)
    g = Domain(*SHAPE, storage=precision, **kw)
    o = OracleDomain(*SHAPE, precision=precision, **kw)
    dt = np.float32 if precision == "fp32" else np.float64
    try:
        with np.errstate(all="ignore"):
            for d in (g, o):
                d.set_populations(_populations(q, precision))
            for n in range(4):
                for a, b in zip(g.macros(dt), o.macros(dt)):
                    assert np.array_equal(a, b, equal_nan=True), n
                a, b = g.populations(dt), o.populations(dt)
                assert np.array_equal(a, b, equal_nan=True), n
                assert n > 0 or not np.isfinite(b).all()
                for d in (g, o):
                    d.step(1)
    finally:
        g.close()
        o.close()

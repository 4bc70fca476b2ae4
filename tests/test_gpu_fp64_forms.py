"""FP64 kernels with fewer operations against the oracle's statements: the same
values, over sizes, boundary types and operands where a form could go wrong."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e-60, 1e-160, 1e20, 1e70, 1e100, 0.0])
def test_weno_weights_over_the_range_of_their_divisors(ctx, orc, scale):
    """The weights' quotients have a fast form in the middle of the range and the
    operator's outside; v / 3 and v / 6 are exact fused forms.  Infinite and NaN
    inputs give NaN on both sides."""
    rng = np.random.default_rng(3)
    n = 3000
    v = [rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-6, 3, n) * scale for _ in range(5)]
    for a in v[:2]:
        a[:5] = 0.0
    v[2][7], v[4][8], v[0][9], v[3][10] = np.nan, np.inf, -np.inf, np.nan
    v = [np.asfortranarray(a.reshape(30, 10, 10)) for a in v]
    ref = np.zeros((30, 10, 10), order="F")
    with np.errstate(all="ignore"):
        orc.call("dFdx_Weno5", ref, *v, ref.size)
    out = ht.zeros(30, 10, 10)
    api.dFdx_Weno5(ctx, out, *[ht.from_numpy(a) for a in v])
    np.testing.assert_array_equal(ht.to_numpy(out), ref)

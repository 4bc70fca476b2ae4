"""Lines of a march sweep cut into short segments (few lines) against whole ones
(many lines): a line's result does not depend on the cut, bit for bit."""
import numpy as np
import pytest
import torch

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [9, 17, 31, 63, 64, 95, 200])
@pytest.mark.parametrize("form", ["f32", "mixed"])
@pytest.mark.parametrize("variant", [abi.WENO_V1, abi.WENO_V2_REF])
def test_segments_do_not_change_a_line(ctx, axis, n, form, variant):
    rng = np.random.default_rng(n)
    few, many = [3, 5, 4], [3, 5, 4]
    few[axis] = many[axis] = n
    if axis == 0:
        many = [n, 200, 200]  # rows
    else:
        many[3 - axis] = 1300  # y lines need planes, z lines rows
    period = [few[a] for a in range(3)]
    T = rng.uniform(0, 1, few)
    V = rng.uniform(-1, 1, [m + (a == axis) for a, m in enumerate(few)])
    dt = torch.float32 if form == "f32" else torch.float64
    out = []
    for size in (few, many):
        idx = np.ix_(*[np.arange(m) % p for m, p in zip(size, period)])
        vidx = np.ix_(*[np.arange(m + 1) if a == axis else np.arange(m) % p
                        for a, (m, p) in enumerate(zip(size, period))])
        Td = ht.zeros(*[m + 2 for m in size], dtype=dt)
        Td[1:-1, 1:-1, 1:-1] = torch.from_numpy(T[idx]).to(device="cuda", dtype=dt)
        Vd = [ht.zeros(*[m + (a == b) for b, m in enumerate(size)], dtype=dt) for a in range(3)]
        Vd[axis].copy_(torch.from_numpy(V[vidx]).to(device="cuda", dtype=dt))
        torch.cuda.synchronize()
        args = (ctx, Td, *Vd, 0.3 / n, *[float(m) for m in few], [0, 1, 1, 0, 0, 1], [0.0, 0.2, 1.0, 0.0, 0.0, 0.5], variant)
        if form == "f32":
            api.weno5_advect_f32(*args)
        else:
            api.weno5_advect(*args, abi.MIXED)
        ctx.synchronize()
        out.append(Td[1:few[0] + 1, 1:few[1] + 1, 1:few[2] + 1].cpu().numpy())
    np.testing.assert_array_equal(*out)
    assert np.abs(out[0] - T.astype(out[0].dtype)).max() > 0

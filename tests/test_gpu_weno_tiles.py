"""Mixed WENO5 stages with a periodic axis: 32 x 8 tiles (many cells, rows that fill
them) against runs of cells (few cells), on the same lines, bit for bit."""
import numpy as np
import pytest
import torch

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi

pytestmark = pytest.mark.gpu


# rows of five whole tiles and of three but for one cell; rows and planes that leave
# the last tiles partly empty; 2^19 cells and more in the larger grid
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("nx", [95, 160])
@pytest.mark.parametrize("variant", [abi.WENO_V1, abi.WENO_V2_REF])
def test_tiles_do_not_change_a_line(ctx, axis, nx, variant):
    few, many = {0: ((nx, 9, 7), (nx, 91, 64)), 1: ((nx, 30, 7), (nx, 30, 190)), 2: ((nx, 7, 30), (nx, 189, 30))}[axis]
    rng = np.random.default_rng(nx + axis)
    T = rng.uniform(0, 1, few)
    V = rng.uniform(-1, 1, [m + (a == axis) for a, m in enumerate(few)])
    bc = [2 if f // 2 == axis else 0 for f in range(6)]
    out = []
    for size in (few, many):
        idx = np.ix_(*[np.arange(m) % p for m, p in zip(size, few)])
        vidx = np.ix_(*[np.arange(m + 1) if a == axis else np.arange(m) % p for a, (m, p) in enumerate(zip(size, few))])
        Td = ht.zeros(*[m + 2 for m in size])
        Td[1:-1, 1:-1, 1:-1] = torch.from_numpy(T[idx]).cuda()
        Vd = [ht.zeros(*[m + (a == b) for b, m in enumerate(size)]) for a in range(3)]
        Vd[axis].copy_(torch.from_numpy(V[vidx]).cuda())
        torch.cuda.synchronize()
        api.weno5_advect(ctx, Td, *Vd, 0.3 / few[axis], *[float(m) for m in few], bc, [0.0] * 6, variant, abi.MIXED)
        out.append(ht.to_numpy(Td)[1:-1, 1:-1, 1:-1])
    np.testing.assert_array_equal(out[1], out[0][np.ix_(*[np.arange(m) % p for m, p in zip(many, few)])])
    assert np.abs(out[0] - T).max() > 0

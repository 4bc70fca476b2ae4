"""Which runs of an ensemble's iterations go in one launch per wave of members: short
runs and small ensembles, for which that is the slower way, are left to the batched
kernel.  Either way gives the same values."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi, hrl

pytestmark = pytest.mark.gpu


def step(ctx, sizes, nitout, nitmax):
    mem = []
    for q, n in enumerate(sizes):
        T, P, ktv, kfv = hrl.initial_fields(*n, seed=q, amp=1e-2)
        mem.append(api.Member(ht.from_numpy(T), ht.from_numpy(P), ht.from_numpy(ktv), ht.from_numpy(kfv),
                              ht.zeros(n[0] + 1, n[1], n[2]), ht.zeros(n[0], n[1] + 1, n[2]),
                              ht.zeros(n[0], n[1], n[2] + 1), hrl.params(*n, Ra=300.0, tol=1e-30, nitout=nitout,
                                                                         nitmax=nitmax)))
    before = ctx.launches
    api.ensemble_step(ctx, mem, abi.MIXED)
    return ctx.launches - before, [ht.to_numpy(getattr(m, f)) for m in mem for f in ("Tc_ex", "Pc_ex", "Vx", "Vy", "Vz")]


# two iterations between checks of a member, of many small ones and of waves of large
# ones; runs that end with the solve; long runs of one member that a launch per
# iteration serves as well, of a small one and of several; thin and long members
@pytest.mark.parametrize("sizes,nitout,nitmax,runs", [
    ([(63, 63, 63)], 4, 60, False), ([(31, 31, 31)] * 22, 5, 60, False), ([(95, 95, 95)] * 3, 6, 60, False),
    ([(63, 63, 63)], 1000, 900, False), ([(20, 17, 16)], 1000, 900, True), ([(63, 63, 63)] * 4, 100, 250, True),
    ([(95, 90, 95), (33, 29, 31)], 100, 250, True), ([(16, 16, 600)] * 2, 4, 40, False), ([(60, 60, 3), (300, 11, 20)], 3, 20, False)])
def test_runs_that_pay(ctx, sizes, nitout, nitmax, runs):
    got, a = step(ctx, sizes, nitout, nitmax)
    try:
        ctx.set_tuning(abi.TUNE_TEMPORAL, 0)
        plain, b = step(ctx, sizes, nitout, nitmax)
    finally:
        ctx.set_tuning(abi.TUNE_TEMPORAL, 1)
    assert (got < plain) == runs
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)

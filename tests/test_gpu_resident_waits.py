"""The bounded waits of resident runs (k_mixed_resident): which block the wait test
mutes, in a solve and in an ensemble, and what the context does afterwards."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi, hrl

pytestmark = pytest.mark.gpu
TYPES, VALS = (0, 1, 1, 0, 1, 0), (0.0, 0.3, 1.0, 0.0, -0.2, 0.0)


def solve(ctx, n, niter):
    nx, ny, nz = n
    rng = np.random.default_rng(7)
    f = lambda *s: ht.from_numpy(np.asfortranarray(rng.uniform(0.5, 1.5, s)))
    X, R = f(nx + 2, ny + 2, nz + 2), f(nx, ny, nz)
    k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
    api.dyrel_solve_dimless(ctx, X, R, *k, 30.0, 1.0 / nx, 0.9 / ny, 1.2 / nz, TYPES, VALS,
                            abi.DyrelParams.reference(nitout=20), ht.zeros(nx, ny, nz), ht.zeros(nx, ny, nz), abi.MIXED,
                            n_iter_fixed=niter)


def three_members():
    mem = []
    for q, n in enumerate([(40, 30, 12), (31, 33, 20), (20, 20, 5)]):  # three, four blocks and one
        T, P, ktv, kfv = hrl.initial_fields(*n, seed=q, amp=1e-2)
        mem.append(api.Member(ht.from_numpy(T), ht.from_numpy(P), ht.from_numpy(ktv), ht.from_numpy(kfv),
                              ht.zeros(n[0] + 1, n[1], n[2]), ht.zeros(n[0], n[1] + 1, n[2]),
                              ht.zeros(n[0], n[1], n[2] + 1), hrl.params(*n, Ra=300.0, nitout=50, nitmax=200)))
    return mem


@pytest.mark.parametrize("block", [2, 4])
def test_a_silent_block_of_an_ensemble(ctx, block):
    """A block of two members never publishes, or the last one of a member that alone
    has that many: every member reports the timeout, and the next step is a clean one."""
    ctx.set_tuning(abi.TUNE_WAIT_TEST, block)
    try:
        mem = three_members()
        with pytest.raises(api.Ht3dError) as e:
            api.ensemble_step(ctx, mem, abi.MIXED)
        assert e.value.status == abi.ERR_TIMEOUT and all(m.status == abi.ERR_TIMEOUT for m in mem)
        a = three_members()
        api.ensemble_step(ctx, a, abi.MIXED)
        ctx.set_tuning(abi.TUNE_TEMPORAL, 0)
        b = three_members()
        api.ensemble_step(ctx, b, abi.MIXED)
    finally:
        ctx.set_tuning(abi.TUNE_WAIT_TEST, 0)
        ctx.set_tuning(abi.TUNE_TEMPORAL, 1)
    for x, y in zip(a, b):
        for f in ("Tc_ex", "Pc_ex", "Vx", "Vy", "Vz"):
            np.testing.assert_array_equal(ht.to_numpy(getattr(x, f)), ht.to_numpy(getattr(y, f)))


def test_the_wait_test_stays_armed_where_no_block_waits(ctx):
    """A grid of one block has nobody to be silent to; the next one with several has."""
    try:
        ctx.set_tuning(abi.TUNE_WAIT_TEST, 1)
        solve(ctx, (6, 5, 1), 30)
        with pytest.raises(api.Ht3dError) as e:
            solve(ctx, (40, 30, 12), 30)
        assert e.value.status == abi.ERR_TIMEOUT
    finally:
        ctx.set_tuning(abi.TUNE_WAIT_TEST, 0)

"""Runs of mixed inner iterations kept on the chip (k_mixed_resident) against one
k_mixed_inner launch per iteration: the same cell arithmetic in another place,
so every result is the same value."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi, hrl

pytestmark = pytest.mark.gpu


def solve(ctx, n, types, vals, niter, seed=7):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    f = lambda *s: ht.from_numpy(np.asfortranarray(rng.uniform(0.5, 1.5, s)))
    X, R = f(nx + 2, ny + 2, nz + 2), f(nx, ny, nz)
    k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
    F, F0 = ht.zeros(nx, ny, nz), ht.zeros(nx, ny, nz)
    st = api.dyrel_solve_dimless(ctx, X, R, *k, 30.0, 1.0 / nx, 0.9 / ny, 1.2 / nz, types, vals,
                                 abi.DyrelParams.reference(nitout=20), F, F0, abi.MIXED, n_iter_fixed=niter)
    out = [ht.to_numpy(t) for t in (X, F, F0)]
    return out, (st.nF_abs, st.lambda_min, st.iters)


# one cell; rows of 4 m - 1 .. 4 m + 2 cells; columns of 1, 2, 3, 5 and 7 planes
# (the last one partly outside the grid), blocks of whole rows of cells, one and
# two CTAs per SM, a last row block that is nearly empty
SIZES = [(1, 1, 1), (1, 2, 3), (3, 1, 9), (4, 5, 2), (5, 40, 6), (33, 29, 31), (63, 63, 63), (64, 33, 150), (66, 65, 30),
         (79, 79, 79), (80, 73, 71), (127, 60, 61), (95, 95, 95), (111, 97, 113), (127, 119, 131), (300, 11, 20)]
BCS = [((0, 1, 1, 0, 1, 0), (0.0, 0.3, 1.0, 0.0, -0.2, 0.0)), ((1, 0, 0, 1, 0, 1), (0.5, 0.0, 0.0, 0.2, 0.0, 1.0))]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("niter", [45, 38])
def test_runs_on_the_chip_equal_single_iterations(ctx, n, bc, niter):
    ctx.set_tuning(abi.TUNE_MIXED_REFRESH, 16)
    try:
        l0 = ctx.launches
        a = solve(ctx, n, *BCS[bc], niter)
        l1 = ctx.launches
        ctx.set_tuning(abi.TUNE_TEMPORAL, 0)
        b = solve(ctx, n, *BCS[bc], niter)
        assert l1 - l0 < ctx.launches - l1  # runs took one launch each
    finally:
        ctx.set_tuning(abi.TUNE_TEMPORAL, 1)
        ctx.set_tuning(abi.TUNE_MIXED_REFRESH, 512)
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)
    assert a[1] == b[1]


def test_a_silent_block_ends_the_wait_and_the_context_recovers(ctx):
    """HT3D_TUNE_WAIT_TEST: one block never publishes its faces; its neighbours'
    bounded waits run out, the solve reports HT3D_ERR_TIMEOUT, and the next solve
    of the same context is a normal one."""
    n = (40, 30, 12)
    try:
        ctx.set_tuning(abi.TUNE_WAIT_TEST, 2)
        with pytest.raises(api.Ht3dError) as e:
            solve(ctx, n, *BCS[0], 30)
        assert e.value.status == abi.ERR_TIMEOUT
        a = solve(ctx, n, *BCS[0], 30)
        ctx.set_tuning(abi.TUNE_TEMPORAL, 0)
        b = solve(ctx, n, *BCS[0], 30)
    finally:
        ctx.set_tuning(abi.TUNE_WAIT_TEST, 0)
        ctx.set_tuning(abi.TUNE_TEMPORAL, 1)
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)


def test_ensemble_waves_equal_members_stepped_alone(ctx):
    """Members that need several launches (waves) per run, with columns of both
    heights, each equal to its own ht3d_step_hrl with single iterations."""
    sizes = [(95, 90, 95), (40, 95, 94), (31, 33, 47), (95, 95, 93), (50, 31, 36), (111, 97, 113)]
    mem = []
    for q, n in enumerate(sizes):
        T, P, ktv, kfv = hrl.initial_fields(*n, seed=q, amp=1e-2)
        mk = lambda: api.Member(ht.from_numpy(T), ht.from_numpy(P), ht.from_numpy(ktv), ht.from_numpy(kfv),
                                ht.zeros(n[0] + 1, n[1], n[2]), ht.zeros(n[0], n[1] + 1, n[2]),
                                ht.zeros(n[0], n[1], n[2] + 1), hrl.params(*n, Ra=300.0 + 100 * q, nitout=100,
                                                                           nitmax=300))
        mem.append((mk(), mk()))
    api.ensemble_step(ctx, [a for a, _ in mem], abi.MIXED)
    try:
        ctx.set_tuning(abi.TUNE_TEMPORAL, 0)
        for _, m in mem:
            m.st_thermal, m.st_darcy = api.step_hrl(ctx, m.Tc_ex, m.Pc_ex, m.ktv, m.kfv, m.Vx, m.Vy, m.Vz, m.params,
                                                    abi.MIXED)
    finally:
        ctx.set_tuning(abi.TUNE_TEMPORAL, 1)
    for a, b in mem:
        for f in ("Tc_ex", "Pc_ex", "Vx", "Vy", "Vz"):
            np.testing.assert_array_equal(ht.to_numpy(getattr(a, f)), ht.to_numpy(getattr(b, f)))
        assert a.st_thermal.iters == b.st_thermal.iters and a.st_darcy.lambda_min == b.st_darcy.lambda_min

"""FP64 kernels with fewer operations against the oracle's statements: the same
values, over sizes, boundary types and operands where a form could go wrong."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi, v18

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


# one cell; a lane's second cell missing; a wall on a tile's edge (nx = 63, 64,
# 65); two and three tiles; rows and planes that end inside a block and a chunk
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 1), (3, 1, 4), (31, 9, 5), (62, 4, 7), (63, 8, 3), (64, 5, 6), (65, 17, 2),
                               (66, 3, 9), (127, 4, 3), (128, 9, 2), (129, 5, 4), (200, 7, 3), (140, 96, 80)])
@pytest.mark.parametrize("cX", [0.0, 25.0])
@pytest.mark.parametrize("types", [(0, 0, 1, 1, 0, 0), (1, 0, 0, 1, 1, 0), (0, 1, 1, 0, 0, 1)])
def test_fp64_iteration_equals_the_oracle(ctx, orc, n, cX, types):
    nx, ny, nz = n
    rng = np.random.default_rng(11)
    f = lambda *s: np.asfortranarray(rng.uniform(0.2, 1.7, s))
    X, R = f(nx + 2, ny + 2, nz + 2), f(nx, ny, nz) - 1.0
    k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
    vals = (0.3, -0.1, 1.0, 0.0, 0.5, 0.2)
    d = (1.0 / nx, 0.9 / ny, 1.1 / nz)
    prm = abi.DyrelParams.reference(nitout=5)
    Xo, F, F0 = X.copy(order="F"), orc.zeros(*n), orc.zeros(*n)
    s, sto = orc.dyrel_solve_dimless(Xo, R, *k, cX, *d, types, vals, prm, F, F0, n_iter_fixed=13)
    Xd, Fd, F0d = ht.from_numpy(X), ht.zeros(*n), ht.zeros(*n)
    std = api.dyrel_solve_dimless(ctx, Xd, ht.from_numpy(R), *[ht.from_numpy(a) for a in k], cX, *d, types, vals, prm, Fd,
                                  F0d, abi.FP64, n_iter_fixed=13)
    g = ht.to_numpy(Xd)
    idx = np.indices(g.shape)
    edge = sum(((idx[a] == 0) | (idx[a] == g.shape[a] - 1)).astype(int) for a in range(3))
    np.testing.assert_array_equal(g[edge <= 1], Xo[edge <= 1])
    np.testing.assert_array_equal(ht.to_numpy(Fd), F)
    np.testing.assert_array_equal(ht.to_numpy(F0d), F0)
    assert (std.nF_abs, std.lambda_min, std.lambda_max) == (sto.nF_abs, sto.lambda_min, sto.lambda_max)


@pytest.mark.parametrize("n_iter", [1, 3, 4, 7])
def test_fp64_iterate_with_and_without_reciprocals(ctx, n_iter):
    """ht3d_dyrel_iterate forms the quotient from a stored reciprocal from four
    iterations on, and in the kernel below; both equal the per-cell layout."""
    n = (70, 13, 9)
    nx, ny, nz = n
    out = []
    for variant in (0, abi.DYREL_CELL):
        ctx.set_tuning(abi.TUNE_DYREL_VARIANT, variant)
        rng = np.random.default_rng(5)
        f = lambda *s: ht.from_numpy(np.asfortranarray(rng.uniform(0.5, 1.5, s)))
        X, R, PC, F0 = f(nx + 2, ny + 2, nz + 2), f(*n), f(*n), f(*n)
        PC *= 4e4
        k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
        ctx.call("ht3d_dyrel_iterate", X.data_ptr(), R.data_ptr(), *[a.data_ptr() for a in k], PC.data_ptr(),
                 F0.data_ptr(), 3.0, 1.0 / nx, 1.0 / ny, 1.0 / nz, abi.int6(0, 1, 1, 0, 0, 1),
                 abi.dbl6(0, .5, 1, 0, 0, .2), 0.9, 0.02, 0.01, n_iter, *n)
        out.append((ht.to_numpy(X), ht.to_numpy(F0)))
    ctx.set_tuning(abi.TUNE_DYREL_VARIANT, 0)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


# an SM's share of the blocks held down by shared memory and not; one cell per thread
# in blocks of 128 and 256, two (odd nx) in blocks of 64 and of 256, at every size class
@pytest.mark.parametrize("n", [(40, 31, 30), (48, 48, 24), (40, 38, 46), (48, 48, 48), (63, 63, 63), (79, 70, 74),
                               (80, 80, 80)])
def test_fp64_iteration_at_the_shapes_of_its_rule(ctx, orc, n):
    nx, ny, nz = n
    rng = np.random.default_rng(17)
    f = lambda *s: np.asfortranarray(rng.uniform(0.2, 1.7, s))
    X, R = f(nx + 2, ny + 2, nz + 2), f(nx, ny, nz) - 1.0
    k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
    d, types, vals = (1.0 / nx, 0.9 / ny, 1.1 / nz), (0, 1, 1, 0, 0, 1), (0.3, -0.1, 1.0, 0.0, 0.5, 0.2)
    prm = abi.DyrelParams.reference(nitout=4)
    Xo, F, F0 = X.copy(order="F"), orc.zeros(*n), orc.zeros(*n)
    s, sto = orc.dyrel_solve_dimless(Xo, R, *k, 25.0, *d, types, vals, prm, F, F0, n_iter_fixed=9)
    Xd, Fd, F0d = ht.from_numpy(X), ht.zeros(*n), ht.zeros(*n)
    std = api.dyrel_solve_dimless(ctx, Xd, ht.from_numpy(R), *[ht.from_numpy(a) for a in k], 25.0, *d, types, vals, prm,
                                  Fd, F0d, abi.FP64, n_iter_fixed=9)
    inner = (slice(1, -1),) * 3
    np.testing.assert_array_equal(ht.to_numpy(Xd)[inner], Xo[inner])
    np.testing.assert_array_equal(ht.to_numpy(Fd), F)
    np.testing.assert_array_equal(ht.to_numpy(F0d), F0)
    assert (std.nF_abs, std.lambda_min, std.lambda_max) == (sto.nF_abs, sto.lambda_min, sto.lambda_max)


@pytest.mark.parametrize("n", [(40, 31, 30), (48, 48, 24), (40, 38, 46), (56, 56, 28), (63, 63, 31)])
def test_dimensional_iteration_with_the_shared_blocks_held_down(ctx, orc, n):
    """Twelve iterations of each system against the oracle's: the bounds of the
    dimensional step (1e-12 of the largest value), at shares of 2 to 5 blocks
    and with more blocks than run at once."""
    nx, ny, nz = n
    b = v18.box(*n, seed=3, nitout=6, nitmax=12)
    V = [np.zeros(s, order="F") for s in ((nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1))]
    T, P = b["T"].copy(order="F"), b["P"].copy(order="F")
    Td, Pd = ht.from_numpy(T), ht.from_numpy(P)
    Vd = [ht.zeros(*v.shape) for v in V]
    a = [b[q] for q in ("phc", "phv", "wN", "kmul")]
    p_o, p_d = b["params"], v18.box(*n, seed=3, nitout=6, nitmax=12)["params"]
    p_o.it = p_d.it = 2
    _, st_t, st_p = orc.step_v18(T, P, *a, *V, p_o)
    gt, gp = api.step_v18(ctx, Td, Pd, *[ht.from_numpy(x) for x in a], *Vd, p_d)
    assert (gt.iters, gp.iters) == (st_t.iters, st_p.iters)
    inner = (slice(1, -1),) * 3
    for d, o in ((ht.to_numpy(Td)[inner], T[inner]), (ht.to_numpy(Pd)[inner], P[inner])):
        assert np.abs(d - o).max() <= 1e-12 * np.abs(o).max()
    for d, o in zip(Vd, V):
        assert np.abs(ht.to_numpy(d) - o).max() <= 1e-12 * np.abs(o).max()


# runs of 128 and of 256 cells that end inside a row and a plane; the smallest grid;
# one inflow side everywhere, two at some points of each warp, two at every point
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 43, 4), (33, 17, 9), (129, 3, 5), (48, 48, 24), (67, 61, 33)])
@pytest.mark.parametrize("flow", ["one", "rough", "spread"])
@pytest.mark.parametrize("variant", [abi.WENO_V1, abi.WENO_V2_REF])
def test_fused_sweep_with_two_inflow_sides(ctx, orc, n, flow, variant):
    nx, ny, nz = n
    rng = np.random.default_rng(29)
    T = np.asfortranarray(rng.uniform(0, 1, (nx + 2, ny + 2, nz + 2)))
    V = [rng.uniform(-1, 1, [m + (a == b) for b, m in enumerate(n)]) for a in range(3)]
    if flow == "one":
        V = [abs(v) for v in V]
    elif flow == "spread":  # every other face flows backwards: a cell has two inflow sides or none
        V = [abs(v) * (1 - 2 * (np.indices(v.shape)[a] % 2 == 0)) for a, v in enumerate(V)]
    V = [np.asfortranarray(v) for v in V]
    h, dt, types, vals = [float(m) for m in n], 0.2 / max(n), [0, 0, 1, 1, 2, 2], [0, 0, 1.0, 0.3, 0, 0]
    To = T.copy(order="F")
    if variant == abi.WENO_V1:
        orc.call("AdvectWithWeno5_v1", To, *V, dt, *h, orc.int6(*types), orc.dbl6(*vals), *n)
    else:
        orc.call("AdvectWithWeno5_v2", To, *V, dt, *h, orc.int6(*types), orc.dbl6(*vals), 1, *n)
    Td = ht.from_numpy(T)
    api.weno5_advect(ctx, Td, *[ht.from_numpy(v) for v in V], dt, *h, types, vals, variant, abi.FP64)
    inner = (slice(1, -1),) * 3
    np.testing.assert_array_equal(ht.to_numpy(Td)[inner], To[inner])


def test_quotients_have_the_operators_bits(ctx):
    """Init_vel_dim divides a flux by a mean of four equal densities: every pair of
    signed zeros, ends of the fast form's range, subnormal, infinite and NaN
    operands and some in between, compared bit by bit with the host's quotient."""
    rng = np.random.default_rng(31)
    ends = [0.0, 5e-324, 2.0 ** -1022, 2.0 ** -1000, np.nextafter(2.0 ** -400, 0), 2.0 ** -400, 0.1, 1.0, 3.0,
            np.nextafter(2.0 ** 400, 0), 2.0 ** 400, 2.0 ** 1000, np.inf, np.nan]
    v = np.array([s * e for e in ends for s in (1, -1)] + list(rng.uniform(-2, 2, 60) * 10.0 ** rng.uniform(-90, 90, 60)))
    a, b = (m.ravel() for m in np.meshgrid(v, v))
    n = a.size - 1
    qx, rfv = np.zeros((n + 1, 1, 1), order="F"), np.zeros((n + 1, 2, 2), order="F")
    qx[:, 0, 0] = a
    rfv[:] = b[:, None, None]
    V = [ht.zeros(n + 1, 1, 1), ht.zeros(n, 2, 1), ht.zeros(n, 1, 2)]
    api.Init_vel_dim(ctx, *V, ht.from_numpy(qx), ht.zeros(n, 2, 1), ht.zeros(n, 1, 2), ht.from_numpy(rfv))
    with np.errstate(all="ignore"):
        ref = a / ((b + b + b + b) * 0.25)
    got = ht.to_numpy(V[0])[:, 0, 0]
    num = ~np.isnan(ref)
    np.testing.assert_array_equal(np.isnan(got), ~num)
    np.testing.assert_array_equal(got[num].view(np.int64), ref[num].view(np.int64))


# more planes than a grid has blocks in z, a cell and three in each; warps past a thin
# plane in blocks of 128 and 256, also where the grid has many cells
@pytest.mark.parametrize("n", [(1, 1, 100000), (3, 1, 66000), (5, 7, 40), (13, 11, 50), (20, 13, 2100)])
def test_fp64_iteration_on_columns_of_many_planes(ctx, n):
    """ht3d_dyrel_iterate and ht3d_dyrel_iterate_noalloc take such columns, an even
    number of iterations of them, and equal the per-cell layout."""
    nx, ny, nz = n
    out = []
    for form in ("cell", "default", "noalloc"):
        ctx.set_tuning(abi.TUNE_DYREL_VARIANT, abi.DYREL_CELL if form == "cell" else 0)
        rng = np.random.default_rng(37)
        f = lambda *s: ht.from_numpy(np.asfortranarray(rng.uniform(0.5, 1.5, s)))
        X, R, PC, F0 = f(nx + 2, ny + 2, nz + 2), f(*n), f(*n), f(*n)
        k = [f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)]
        args = (X.data_ptr(), R.data_ptr(), *[a.data_ptr() for a in k], PC.data_ptr(), F0.data_ptr(), 3.0, 1.0, 1.0, 1.0,
                abi.int6(0, 1, 1, 0, 0, 1), abi.dbl6(0, .5, 1, 0, 0, .2), 0.9, 0.02, 0.01, 2, *n)
        if form == "noalloc":
            assert ctx.lib.ht3d_dyrel_iterate_noalloc(*args, ctx.stream) == abi.OK
            ctx.synchronize()
        else:
            ctx.call("ht3d_dyrel_iterate", *args)
        out.append((ht.to_numpy(X), ht.to_numpy(F0)))
    ctx.set_tuning(abi.TUNE_DYREL_VARIANT, 0)
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)

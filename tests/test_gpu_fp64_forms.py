"""FP64 kernels with fewer operations against the oracle's statements: the same
values, over sizes, boundary types and operands where a form could go wrong."""
import numpy as np
import pytest

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi

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

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


def sweep_lines(T, V, dt, h, types, vals):
    """The FP32 sweep's scheme along the first axis, in 64 bits: its weights have the
    floor 1e-18 + 1e-6 max d^2 (the FP64 sweep's has 1e-99)."""
    def weno(v1, v2, v3, v4, v5):
        p = [v1 / 3 - 7 / 6 * v2 + 11 / 6 * v3, -v2 / 6 + 5 / 6 * v3 + v4 / 3, v3 / 3 + 5 / 6 * v4 - v5 / 6]
        e = 1e-18 + 1e-6 * np.max(np.square([v1, v2, v3, v4, v5]), axis=0)
        s = [13 / 12 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2 + e,
             13 / 12 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2 + e,
             13 / 12 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2 + e]
        w = [c / x ** 2 for c, x in zip((0.1, 0.6, 0.3), s)]
        return sum(a * b for a, b in zip(w, p)) / sum(w)

    def stage(x):
        n = len(x)
        left = [2 * vals[0] - x[q] if types[0] else x[q] for q in (2, 1, 0)]
        right = [2 * vals[1] - x[q] if types[1] else x[q] for q in (n - 1, n - 2, n - 3)]
        d = h * np.diff(np.concatenate([left, x, right]), axis=0)
        d = [d[q:q + n] for q in range(6)]
        return x - dt * (np.maximum(V[1:], 0) * weno(*d[:5]) + np.minimum(V[:-1], 0) * weno(*d[:0:-1]))

    return 0.5 * stage(stage(T)) + 0.5 * T


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 10, 15, 16, 23])
@pytest.mark.parametrize("flow", ["one", "other", "both", "none"])
@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e6])
def test_paired_stages_at_a_lines_ends(ctx, axis, n, flow, scale):
    """The FP32 march runs both stages in one step up to a line's last four cells:
    short lines against the scheme in 64 bits, 2e-5 of the largest value (the
    bound of an FP32 sweep), for each direction of the flow."""
    rng = np.random.default_rng(n + 100 * axis)
    size = [4, 6, 5]
    size[axis] = n
    T = rng.uniform(0, scale, size)
    V = rng.uniform(-1, 1, [m + (a == axis) for a, m in enumerate(size)])
    V = {"one": abs(V), "other": -abs(V), "both": V, "none": 0 * V}[flow]
    types, vals = [0, 1, 1, 0, 0, 1], [0.0, 0.2 * scale, scale, 0.0, 0.0, 0.5 * scale]
    Td = ht.zeros(*[m + 2 for m in size], dtype=torch.float32)
    Td[1:-1, 1:-1, 1:-1] = torch.from_numpy(T).to(device="cuda", dtype=torch.float32)
    Vd = [ht.zeros(*[m + (a == b) for b, m in enumerate(size)], dtype=torch.float32) for a in range(3)]
    Vd[axis].copy_(torch.from_numpy(V).to(device="cuda", dtype=torch.float32))
    torch.cuda.synchronize()
    api.weno5_advect_f32(ctx, Td, *Vd, 0.3 / n, *[float(m) for m in size], types, vals, abi.WENO_V1)
    ctx.synchronize()
    ref = np.moveaxis(sweep_lines(np.moveaxis(T, axis, 0), np.moveaxis(V, axis, 0), 0.3 / n, float(n),
                                  types[2 * axis:2 * axis + 2], vals[2 * axis:2 * axis + 2]), 0, axis)
    assert np.abs(Td[1:-1, 1:-1, 1:-1].cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_bad_cell_stays_downstream(ctx, axis, bad):
    """Both sides are evaluated, and the side that the flow does not come from is
    taken as 0 whatever it is: a stage carries a bad cell two cells upstream."""
    size, p = [5, 5, 5], 30
    size[axis] = 60
    out = []
    for poison in (False, True):
        rng = np.random.default_rng(2)
        T = ht.zeros(*[m + 2 for m in size], dtype=torch.float32)
        T[1:-1, 1:-1, 1:-1] = torch.from_numpy(rng.uniform(0, 1, size)).to(device="cuda", dtype=torch.float32)
        if poison:
            T[1:-1, 1:-1, 1:-1].select(axis, p)[:] = float(bad)
        V = [ht.zeros(*[m + (a == b) for b, m in enumerate(size)], dtype=torch.float32) for a in range(3)]
        V[axis] += 0.5
        torch.cuda.synchronize()
        api.weno5_advect_f32(ctx, T, *V, 0.005, *[float(m) for m in size], [0] * 6, [0.0] * 6, abi.WENO_V1)
        ctx.synchronize()
        out.append(T[1:-1, 1:-1, 1:-1].cpu().movedim(axis, 0))
    assert torch.equal(out[0][:p - 4], out[1][:p - 4])
    assert bool(torch.isfinite(out[0]).all()) and not bool(torch.isfinite(out[1][p:p + 3]).any())

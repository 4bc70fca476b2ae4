"""Performance cases of the ht3d framework: what its users run, through its public entry points.

A case is a dict of plain values; its "kind" is the call it stands for:

  step      one time step of the dimensionless porous-convection model (api.step_hrl): thermal DYREL
            solve, Darcy DYREL solve, velocity, WENO5 advection, adaptive dt; FP64 or mixed precision
  ensemble  one time step of an ensemble of independent models of different sizes (api.ensemble_step)
  v18       one transient time step of the dimensional model on the synthetic box (api.step_v18)
  solve     a DYREL solve of a bounded number of pseudo-iterations on its own (api.dyrel_solve_dimless)
  sweep     a stand-alone WENO5 advection (api.weno5_advect, api.weno5_advect_f32)
  post      the twelve output diagnostics of a time step (api.postprocess_fields)
  kernels   a driver that calls the reference-shaped kernels one by one: the property kernels and one
            thermal and one Darcy pseudo-iteration of the dimensional model

The in-place calls start every pass from the same fields: a pass first copies the state that the step
starts from into the arrays that the call updates, as a program does that keeps the last time level.
"""
import ctypes
import math

import torch

from hydrothermal3d_gb300 import abi, api, hrl, post, sweep, v18

PRECISION = {"fp64": abi.FP64, "mixed": abi.MIXED}
VARIANT = {"v1": abi.WENO_V1, "v2ref": abi.WENO_V2_REF, "v2fixed": abi.WENO_V2_FIXED}
SWEEP_BC, SWEEP_VAL = [0, 0, 1, 1, 0, 0], [0.0, 0.0, 0.0, 0.0, 0.0, 0.0]
SOLVE_BC, SOLVE_VAL = (0, 0, 0, 0, 0, 0), (0.0, 0.0, 0.0, 0.0, 0.0, 0.0)


def _case(kind, n, name=None, **more):
    c = dict(kind=kind, nx=int(n[0]), ny=int(n[1]), nz=int(n[2]), **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coarse trial run on an odd box with a random permeability: latency and launches count
        _case("step", (33, 29, 31), "step_mixed_33x29x31", precision="mixed", perm="lognormal"),
        # the 63^3 model that the reference runs on a workstation, in both precisions
        _case("step", (63, 63, 63), "step_mixed_63", precision="mixed", perm="uniform"),
        _case("step", (63, 63, 63), "step_fp64_63", precision="fp64", perm="uniform"),
        # a medium production grid whose sides are no multiples of any tile
        _case("step", (127, 119, 131), "step_mixed_127x119x131", precision="mixed", perm="lognormal"),
        # the benchmark's headline grid
        _case("step", (255, 255, 255), "step_mixed_255", precision="mixed", perm="uniform"),
        # a parameter study: 64 members of 31 to 95 cells a side
        dict(name="ensemble_64", kind="ensemble", members=64, smallest=31, largest=95),
        # the dimensional model (plain FP64 throughout), a transient step with its advection sub-steps
        _case("v18", (48, 48, 24), "v18_step_48x48x24"),
        # the largest grid: the heterogeneous medium with a fault slab, a bounded number of iterations
        _case("solve", (511, 511, 511), "solve_mixed_511", precision="mixed", iters=600),
        # stand-alone advection: the large FP32 sweep, and the FP64 sweep of the dimensional model
        _case("sweep", (511, 511, 511), "sweep_f32_511", precision="f32", variant="v1", periodic=False),
        _case("sweep", (127, 127, 127), "sweep_fp64_127", precision="fp64", variant="v2ref", periodic=False),
        # the output step of a large run
        _case("post", (255, 255, 127), "post_255x255x127"),
        # a driver written against the reference's kernels
        _case("kernels", (127, 95, 63), "kernels_127x95x63"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo, hi):
    """Three sides around one size drawn over its logarithm, within [lo, hi]."""
    n = _log(rng, lo, hi)
    return [max(lo, min(hi, round(n * rng.uniform(0.75, 1.3)))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "ensemble", "v18", "solve", "solve", "sweep", "sweep", "post",
                       "kernels"])
    if kind == "step":
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        return _case(kind, _box(rng, 24, 255 if precision == "mixed" else 95), precision=precision,
                     perm=rng.choice(["uniform", "lognormal"]))
    if kind == "ensemble":
        return dict(kind=kind, members=round(_log(rng, 4, 64)), smallest=31, largest=rng.randint(47, 95))
    if kind == "v18":
        return _case(kind, (rng.randint(24, 56), rng.randint(24, 56), rng.randint(12, 28)))
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        return _case(kind, _box(rng, 48, 480) if precision == "mixed" else _box(rng, 31, 160), precision=precision,
                     iters=rng.randint(150, 600))
    if kind == "sweep":
        precision = rng.choice(["f32", "mixed", "fp64"])
        return _case(kind, _box(rng, 31, 480 if precision == "f32" else 255), precision=precision,
                     variant=rng.choice(["v1", "v2ref", "v2fixed"]), periodic=rng.random() < 0.25)
    return _case(kind, _box(rng, 31, 255 if kind == "post" else 191))


def _sides(case):
    return case["nx"], case["ny"], case["nz"]


# ------------------------------------------------------------------ preparation
_HANDLE = {}


def _handle():
    """The program's context and the stream that it and torch share."""
    if not _HANDLE:
        s = torch.cuda.Stream()
        _HANDLE["stream"], _HANDLE["ctx"] = s, api.Context(device=0, stream=s.cuda_stream)
    return _HANDLE["ctx"], _HANDLE["stream"]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _hrl_fields(n, gen, perm, slab=False):
    """T (linear in y, perturbed), P = 0, ktv = 1 and kfv of the porous-convection model."""
    nx, ny, nz = n
    T, P = api.zeros(nx + 2, ny + 2, nz + 2), api.zeros(nx + 2, ny + 2, nz + 2)
    y = (torch.arange(ny + 2, dtype=torch.float64, device="cuda") - 0.5) / ny
    T.copy_((1.0 - y)[None, :, None].expand(nx + 2, ny + 2, nz + 2))
    T[1:-1, 1:-1, 1:-1] += (torch.rand((nz, ny, nx), generator=gen, dtype=torch.float64, device="cuda") * 2e-3
                            - 1e-3).permute(2, 1, 0)
    ktv, kfv = api.ones(nx + 1, ny + 1, nz + 1), api.ones(nx + 1, ny + 1, nz + 1)
    if perm == "lognormal":
        kfv.copy_(hrl.lognormal_torch((nx + 1, ny + 1, nz + 1), seed=int(torch.randint(1 << 30, (1,), generator=gen,
                                                                                       device="cuda"))))
    if slab:  # three cells of ten times the permeability at mid-x
        kfv[nx // 2 - 1:nx // 2 + 3] *= 10.0
    return T, P, ktv, kfv


def _faces_of_vertices(kv):
    """Face conductivities: the mean of a face's four vertices."""
    return (((kv[:, :-1, :-1] + kv[:, 1:, :-1]) + (kv[:, :-1, 1:] + kv[:, 1:, 1:])) * 0.25,
            ((kv[:-1, :, :-1] + kv[1:, :, :-1]) + (kv[:-1, :, 1:] + kv[1:, :, 1:])) * 0.25,
            ((kv[:-1, :-1, :] + kv[1:, :-1, :]) + (kv[:-1, 1:, :] + kv[1:, 1:, :])) * 0.25)


def _columns(t):
    """The tensor in the framework's column-major layout."""
    return api.zeros(*t.shape, dtype=t.dtype).copy_(t)


def _clone_params(p):
    q = type(p)()
    ctypes.memmove(ctypes.byref(q), ctypes.byref(p), ctypes.sizeof(p))
    return q


def prepare(case, seed):
    ctx, stream = _handle()
    with torch.cuda.stream(stream):
        s = _PREPARE[case["kind"]](case, seed)
    s.update(case=case, ctx=ctx, stream=stream)
    stream.synchronize()
    return s


def _prepare_step(case, seed):
    n = _sides(case)
    T, P, ktv, kfv = _hrl_fields(n, _generator(seed), case["perm"])
    nx, ny, nz = n
    return dict(T0=T, P0=P, T=_columns(T), P=_columns(P), ktv=ktv, kfv=kfv, p0=hrl.params(*n, dt_max=1e-3),
                V=[api.zeros(nx + 1, ny, nz), api.zeros(nx, ny + 1, nz), api.zeros(nx, ny, nz + 1)])


def _member_sides(case):
    """The members' grids: they belong to the case, whatever the seed of the fields."""
    g = torch.Generator().manual_seed(1000003 * case["members"] + case["largest"])
    return torch.randint(case["smallest"], case["largest"] + 1, (case["members"], 3), generator=g).tolist()


def _prepare_ensemble(case, seed):
    gen = _generator(seed)
    sides = _member_sides(case)
    u = torch.rand(case["members"], generator=gen, device="cuda").tolist()
    ex = [(a + 2) * (b + 2) * (c + 2) for a, b, c in sides]
    fl = {"T0": ex, "P0": ex, "T": ex, "P": ex, "Vx": [(a + 1) * b * c for a, b, c in sides],
          "Vy": [a * (b + 1) * c for a, b, c in sides], "Vz": [a * b * (c + 1) for a, b, c in sides]}
    flat = {k: torch.zeros(sum(v), dtype=torch.float64, device="cuda") for k, v in fl.items()}
    part = {k: torch.split(flat[k], v) for k, v in fl.items()}
    members, p0 = [], []
    for m, n in enumerate(sides):
        nx, ny, nz = n
        view = lambda k, a, b, c: part[k][m].view(c, b, a).permute(2, 1, 0)  # noqa: E731
        T, P, ktv, kfv = _hrl_fields(n, gen, "lognormal")
        view("T0", nx + 2, ny + 2, nz + 2).copy_(T)
        p0.append(hrl.params(*n, Ra=100.0 * 50.0 ** u[m], dt_max=1e-3))
        members.append(api.Member(view("T", nx + 2, ny + 2, nz + 2), view("P", nx + 2, ny + 2, nz + 2), ktv, kfv,
                                  view("Vx", nx + 1, ny, nz), view("Vy", nx, ny + 1, nz), view("Vz", nx, ny, nz + 1),
                                  _clone_params(p0[-1])))
    return dict(flat=flat, members=members, p0=p0)


def _v18_box(case, seed):
    b = v18.box(*_sides(case), seed=seed)
    b["params"].it = 2
    return b


def _prepare_v18(case, seed):
    nx, ny, nz = _sides(case)
    b = _v18_box(case, seed)
    d = {k: api.from_numpy(b[k]) for k in ("T", "P", "phc", "phv", "wN", "kmul")}
    return dict(T0=d["T"], P0=d["P"], T=_columns(d["T"]), P=_columns(d["P"]), fixed=[d["phc"], d["phv"], d["wN"],
                                                                                    d["kmul"]], p0=b["params"],
                V=[api.zeros(nx + 1, ny, nz), api.zeros(nx, ny + 1, nz), api.zeros(nx, ny, nz + 1)])


def _prepare_solve(case, seed):
    """The Darcy solve of the model's fault-slab medium: buoyancy of the initial temperature as its right-hand side."""
    n = _sides(case)
    T, P, _, kfv = _hrl_fields(n, _generator(seed), "lognormal", slab=True)
    k = [_columns(f) for f in _faces_of_vertices(kfv)]
    del kfv
    q = k[1] * ((T[1:-1, :-1, 1:-1] + T[1:-1, 1:, 1:-1]) * 0.5)
    q[:, 0] = 0.0
    q[:, -1] = 0.0
    return dict(X0=P, X=_columns(P), R=_columns(torch.diff(q, dim=1) * (1000.0 * n[1])), k=k, F=api.zeros(*n),
                F0=api.zeros(*n), prm=abi.DyrelParams.reference())


def _prepare_sweep(case, seed):
    n = _sides(case)
    dt = torch.float32 if case["precision"] == "f32" else torch.float64
    V = sweep.curl_velocity(*n, seed=seed, dtype=dt)
    c = torch.rand(3, generator=_generator(seed), device="cuda").tolist()
    T0 = sweep.blob(*n, centre=tuple(0.3 + 0.4 * v for v in c), dtype=dt)
    return dict(T0=T0, T=_columns(T0), V=V, dt=sweep.cfl_dt(*n), bc=_sweep_bc(case))


def _sweep_bc(case):
    return [2, 2] + SWEEP_BC[2:] if case["periodic"] else SWEEP_BC


def _prepare_post(case, seed):
    n = _sides(case)
    return dict(d=post.device_case(*n, seed=seed), o=post.outputs(*n))


def _prepare_kernels(case, seed):
    n = nx, ny, nz = _sides(case)
    b = _v18_box(case, seed)
    d = {k: api.from_numpy(b[k]) for k in ("T", "P", "phc", "phv", "wN", "kmul")}
    z = api.zeros
    w = {k: z(*n) for k in ("rC", "G", "D", "F", "F0", "Fp", "F0p", "prf", "prf0", "drdp", "kc", "Gp")}
    w.update({k: z(nx + 1, ny + 1, nz + 1) for k in ("ktv", "kfv", "rfv")})
    for f in ("k", "q", "h", "u", "V"):
        w[f] = [z(nx + 1, ny, nz), z(nx, ny + 1, nz), z(nx, ny, nz + 1)]
    inner = (slice(1, -1),) * 3
    return dict(T0=d["T"], P0=d["P"], T=_columns(d["T"]), P=_columns(d["P"]), Told=_columns(d["T"][inner]),
                Pold=_columns(d["P"][inner]), d=d, w=w, p=b["params"])


_PREPARE = dict(step=_prepare_step, ensemble=_prepare_ensemble, v18=_prepare_v18, solve=_prepare_solve,
                sweep=_prepare_sweep, post=_prepare_post, kernels=_prepare_kernels)


# ------------------------------------------------------------------ one pass
def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_step(s):
    p = _clone_params(s["p0"])
    with torch.cuda.stream(s["stream"]):
        s["T"].copy_(s["T0"])
        s["P"].copy_(s["P0"])
    a, b = api.step_hrl(s["ctx"], s["T"], s["P"], s["ktv"], s["kfv"], *s["V"], p, PRECISION[s["case"]["precision"]])
    return dict(T=s["T"], P=s["P"], V=s["V"], dt=p.dt, iters=[a.iters, b.iters])


def _run_ensemble(s):
    f = s["flat"]
    with torch.cuda.stream(s["stream"]):
        f["T"].copy_(f["T0"])
        f["P"].copy_(f["P0"])
    for m, p in zip(s["members"], s["p0"]):
        m.params.dt = p.dt
    api.ensemble_step(s["ctx"], s["members"])
    return dict(T=f["T"], P=f["P"], V=[f["Vx"], f["Vy"], f["Vz"]],
                dt=torch.tensor([m.params.dt for m in s["members"]], dtype=torch.float64),
                iters=torch.tensor([[m.st_thermal.iters, m.st_darcy.iters] for m in s["members"]]))


def _run_v18(s):
    p = _clone_params(s["p0"])
    with torch.cuda.stream(s["stream"]):
        s["T"].copy_(s["T0"])
        s["P"].copy_(s["P0"])
    a, b = api.step_v18(s["ctx"], s["T"], s["P"], *s["fixed"], *s["V"], p)
    return dict(T=s["T"], P=s["P"], V=s["V"], counts=[a.iters, b.iters, p.n_adv])


def _run_solve(s):
    c = s["case"]
    with torch.cuda.stream(s["stream"]):
        s["X"].copy_(s["X0"])
    api.dyrel_solve_dimless(s["ctx"], s["X"], s["R"], *s["k"], 0.0, 1.0 / c["nx"], 1.0 / c["ny"], 1.0 / c["nz"],
                            SOLVE_BC, SOLVE_VAL, s["prm"], s["F"], s["F0"], PRECISION[c["precision"]],
                            n_iter_fixed=c["iters"])
    return dict(X=s["X"], F=s["F"], F0=s["F0"])


def _run_sweep(s):
    c = s["case"]
    with torch.cuda.stream(s["stream"]):
        s["T"].copy_(s["T0"])
    args = (s["ctx"], s["T"], *s["V"], s["dt"], float(c["nx"]), float(c["ny"]), float(c["nz"]), s["bc"], SWEEP_VAL,
            VARIANT[c["variant"]])
    if c["precision"] == "f32":
        api.weno5_advect_f32(*args)
    else:
        api.weno5_advect(*args, PRECISION[c["precision"]])
    return s["T"]


def _run_post(s):
    post.run_fused(s["ctx"], s["d"], s["o"])
    return s["o"]


def _run_kernels(s):
    ctx, w, d, p = s["ctx"], s["w"], s["d"], s["p"]
    T, P = s["T"], s["P"]
    _dx, _dy, _dz, _dt = 1.0 / p.dx, 1.0 / p.dy, 1.0 / p.dz, 1.0 / p.dt
    with torch.cuda.stream(s["stream"]):
        T.copy_(s["T0"])
        P.copy_(s["P0"])
        w["F0"].zero_()
        w["F0p"].zero_()
    # heat: properties, preconditioner, one pseudo-iteration
    api.ComputeThermalConductivity(ctx, w["ktv"], T, d["phv"], p.phi_i, p.sc_kt, p.sc_T)
    api.SmoothConductivityV2C(ctx, w["kc"], w["ktv"])
    api.SmoothConductivityC2V(ctx, w["ktv"], w["kc"])
    api.InitConductivity(ctx, *w["k"], w["ktv"])
    api.ComputeRhoCeffective(ctx, w["rC"], T, P, d["phc"], p.phi_i, p.sc_T, p.sc_sigma, p.sc_C, p.sc_rho)
    api.GershgorinPoisson(ctx, w["G"], w["D"], w["rC"], *w["k"], 1.0, p.dt, p.dx, p.dy, p.dz)
    lmax = api.maximum_g(ctx, w["G"])
    h1, h2, dtau = _dyrel_scalars(lmax)
    api.SetTemperatureBCs(ctx, T, w["k"][1], d["wN"], d["phc"], p.qyS, _dy, 0.0, 0.0, p.Ttop)
    api.ComputeFlux(ctx, *w["q"], *w["k"], T, _dx, _dy, _dz)
    api.ResidualTemperatureLinearised(ctx, w["F"], T, s["Told"], w["rC"], d["phc"], w["D"], *w["q"], p.Qt, 1.0, _dt,
                                      _dx, _dy, _dz)
    api.DYRELUpdate(ctx, w["F0"], T, w["F"], h1, h2, dtau)
    # pore fluid: the same
    api.ComputeHydroConductivity(ctx, w["kfv"], T, P, d["phv"], p.ymin, p.dy, p.k_fact, p.delta, p.sc_sigma, p.sc_T,
                                 p.sc_L, p.sc_t, p.sc_eta, 1, d["kmul"])
    api.ComputeFluidDensity(ctx, w["rfv"], T, P, d["phv"], p.sc_sigma, p.sc_T, p.sc_rho)
    api.InitConductivity(ctx, *w["h"], w["kfv"])
    api.PhiRhofOld(ctx, w["prf0"], s["Told"], s["Pold"], d["phc"], p.phi_i, p.sc_rho, p.sc_T, p.sc_sigma)
    api.PhiRhof(ctx, w["prf"], T, P, d["phc"], p.phi_i, p.sc_rho, p.sc_T, p.sc_sigma)
    api.PhiDrhodP(ctx, w["drdp"], T, P, d["phc"], p.phi_i, p.sc_rho, p.sc_T, p.sc_sigma)
    api.GershgorinPoisson(ctx, w["Gp"], w["D"], w["drdp"], *w["h"], 1.0, p.dt, p.dx, p.dy, p.dz)
    lmax = api.maximum_g(ctx, w["Gp"])
    h1, h2, dtau = _dyrel_scalars(lmax)
    api.SetPressureBCs_dim(ctx, P, d["wN"], d["phc"], p.Pbot, p.Ptop)
    api.ComputeDarcyFlux(ctx, *w["u"], w["rfv"], *w["h"], P, p.g, _dx, _dy, _dz)
    api.ResidualFluidPressure(ctx, w["Fp"], d["phc"], w["prf"], w["prf0"], w["D"], *w["u"], 1.0, _dt, _dx, _dy, _dz)
    api.DYRELUpdate(ctx, w["F0p"], P, w["Fp"], h1, h2, dtau)
    api.Init_vel_dim(ctx, *w["V"], *w["u"], w["rfv"])
    return dict(T=T, P=P, F=w["F"], Fp=w["Fp"], ktv=w["ktv"], kfv=w["kfv"], rC=w["rC"], G=w["G"], Gp=w["Gp"], q=w["q"],
                u=w["u"], V=w["V"], rfv=w["rfv"], prf=w["prf"], drdp=w["drdp"])


_RUN = dict(step=_run_step, ensemble=_run_ensemble, v18=_run_v18, solve=_run_solve, sweep=_run_sweep, post=_run_post,
            kernels=_run_kernels)


# ------------------------------------------------------------------ the least work of a pass
def work(case):
    """Inputs read once and outputs written once; flops of the arithmetic that the method asks for: about 35 per
    cell and pseudo-iteration of the dimensionless operator (85 of the Darcy one with its density polynomial), 430
    per cell of a WENO5 sweep.  The solves check their residual every 1000 iterations: a thermal solve takes 1000
    and a Darcy solve at least 2000 (dimensional: 5000), which is what is counted."""
    kind = case["kind"]
    N = sum(a * b * c for a, b, c in (_member_sides(case) if kind == "ensemble" else [_sides(case)]))
    if kind in ("step", "ensemble"):  # T, P updated; ktv, kfv read; V written
        return dict(bytes=9 * 8 * N, flops=N * (3000 * 35 + 430))
    if kind == "v18":  # T, P updated; phases and kmul read; V written
        return dict(bytes=10 * 8 * N, flops=N * (1000 * 35 + 5000 * 85 + 100 * 430))
    if kind == "solve":  # X updated; R, k read; F, F0 written
        return dict(bytes=8 * 8 * N, flops=N * case["iters"] * 35)
    if kind == "sweep":  # T updated; V read
        return dict(bytes=5 * (4 if case["precision"] == "f32" else 8) * N, flops=N * 430)
    if kind == "post":
        return dict(bytes=post.bytes_fused(*_sides(case)), flops=N * 120)
    return dict(bytes=33 * 8 * N, flops=N * 600)


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
def exact(case, seed):
    s = prepare(case, seed)
    with torch.cuda.stream(s["stream"]):
        r = _EXACT[case["kind"]](case, seed, s)
    s["stream"].synchronize()
    return r


IN = (slice(1, -1),) * 3


def _axis(t, a, lo, hi):
    """t[lo:hi] along axis a (hi None: to the end)."""
    i = [slice(None)] * 3
    i[a] = slice(lo, hi)
    return t[tuple(i)]


def _ghost(t, a, end):
    """(ghost plane, the inner plane next to it) of a ghosted field, over the inner cells of the other axes."""
    i, j = [slice(1, -1)] * 3, [slice(1, -1)] * 3
    i[a], j[a] = (slice(0, 1), slice(1, 2)) if end == 0 else (slice(-1, None), slice(-2, -1))
    return t[tuple(i)], t[tuple(j)]


def _fill_faces(X, types, vals):
    for f in range(6):
        g, v = _ghost(X, f // 2, f % 2)
        g.copy_(2.0 * vals[f] - v if types[f] == 1 else v)


def _across(X, a):
    """Differences of a ghosted field across the faces of axis a."""
    i = [slice(1, -1)] * 3
    i[a] = slice(None)
    return torch.diff(X[tuple(i)], dim=a)


def _div(q, h):
    return sum(torch.diff(q[a], dim=a) * h[a] for a in range(3))


def _gershgorin(k, h, c):
    """(diagonal, sum of magnitudes over the diagonal) of c + div(k grad)."""
    s = sum((_axis(k[a], a, 0, -1) + _axis(k[a], a, 1, None)) * h[a] ** 2 for a in range(3))
    return s + c, (s + (s + c).abs()) / (s + c)


def _dyrel_scalars(lmax, lmin=None, cfl=0.99, cfact=0.5, ratio=500.0):
    dtau = 2.0 / math.sqrt(lmax) * cfl
    c = 2.0 * math.sqrt(lmax / ratio if lmin is None else lmin) * cfact
    return (2 - c * dtau) / (2 + c * dtau), 2 * dtau / (2 + c * dtau), dtau


def _dyrel(X, fill, residual, PC, lmax, prm, fixed=0):
    """The damped iteration with its checks; X is updated; (F, F0, iterations)."""
    F, F0 = torch.zeros_like(PC), torch.zeros_like(PC)
    h1, h2, dtau = _dyrel_scalars(lmax)
    N, first = PC.numel(), None
    for it in range(1, (fixed or prm.nitmax) + 1):
        old = F
        fill(X)
        F = residual(X) / PC
        F0 = F0 * h1 + h2 * F
        X[IN] -= dtau * F0
        if it % prm.nitout and it > 2:
            continue
        norm = float((F * PC).abs().sum()) / N / math.sqrt(N) * prm.norm_scale
        first = norm if first is None else first
        if it > 1:
            d = dtau * F0
            h1, h2, dtau = _dyrel_scalars(lmax, abs(float((d * (F - old)).sum())) / float((d * d).sum()))
        if not fixed and (norm < prm.tol_abs or norm / first < prm.tol_rel):
            break
    return F, F0, it


def _diffusion(X, R, k, cX, h, types, vals, prm, fixed=0):
    PC, G = _gershgorin(k, h, cX)

    def residual(X):
        return R + cX * X[IN] + _div([-k[a] * (_across(X, a) * h[a]) for a in range(3)], h)

    return _dyrel(X, lambda X: _fill_faces(X, types, vals), residual, PC, float(G.max()), prm, fixed)


def _weno_side(v):
    v1, v2, v3, v4, v5 = v
    p1 = v1 / 3 - 7 / 6 * v2 + 11 / 6 * v3
    p2 = -v2 / 6 + 5 / 6 * v3 + v4 / 3
    p3 = v3 / 3 + 5 / 6 * v4 - v5 / 6
    big = v1 * v1
    for x in (v2, v3, v4, v5):
        big = torch.maximum(big, x * x)
    e = 1e-99 + 1e-6 * big
    s1 = 13 / 12 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    s2 = 13 / 12 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    s3 = 13 / 12 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    w1, w2, w3 = 0.1 / (s1 + e) ** 2, 0.6 / (s2 + e) ** 2, 0.3 / (s3 + e) ** 2
    return (w1 * p1 + w2 * p2 + w3 * p3) / (w1 + w2 + w3)


def _weno_rhs(T, a, V, h, types, vals, quirk):
    """V dT/da of the inner cells T."""
    lo, hi = types[2 * a], types[2 * a + 1]
    n = T.shape[a]
    if lo == 2:
        left, right = _axis(T, a, n - 3, None), _axis(T, a, 0, 3)
    else:
        left, right = torch.flip(_axis(T, a, 0, 3), (a,)), torch.flip(_axis(T, a, n - 3, None), (a,))
        left = 2 * vals[2 * a] - left if lo == 1 else left
        right = 2 * vals[2 * a + 1] - right if hi == 1 else right
    x = torch.cat([left, T, right], a)
    d = h * torch.diff(x, dim=a)
    g = [d.narrow(a, o, n) for o in range(6)]
    m5 = h * (x.narrow(a, 5, n) - x.narrow(a, 2, n)) if quirk else g[4]
    Vm, Vp = _axis(V, a, 0, -1).clamp(max=0.0), _axis(V, a, 1, None).clamp(min=0.0)
    return Vp * _weno_side([g[0], g[1], g[2], g[3], m5]) + Vm * _weno_side([g[5], g[4], g[3], g[2], g[1]])


def _weno(T_ex, V, dt, h, types, vals, quirk):
    T = T_ex[IN].clone()
    for a in range(3):
        t = T - dt * _weno_rhs(T, a, V[a], h[a], types, vals, quirk)
        T = 0.5 * (t - dt * _weno_rhs(t, a, V[a], h[a], types, vals, quirk)) + 0.5 * T
    T_ex[IN] = T


def _step(T, P, ktv, kfv, p):
    h, dt = (1 / p.dx, 1 / p.dy, 1 / p.dz), p.dt
    k = _faces_of_vertices(ktv)
    _, _, a = _diffusion(T, -1 / dt * T[IN], k, 1 / dt, h, list(p.thermal_bc), list(p.thermal_val), p.thermal)
    k = _faces_of_vertices(kfv)
    Ty = (T[1:-1, :-1, 1:-1] + T[1:-1, 1:, 1:-1]) * 0.5
    if p.kill_ns:
        Ty[:, 0] = 0
        Ty[:, -1] = 0
    _, _, b = _diffusion(P, p.Ra * h[1] * torch.diff(k[1] * Ty, dim=1), k, 0.0, h, list(p.darcy_bc),
                         list(p.darcy_val), p.darcy)
    V = [-k[i] * (_across(P, i) * h[i] - (p.Ra * Ty if i == 1 else 0.0)) for i in range(3)]
    _weno(T, V, dt, h, list(p.weno_bc), list(p.weno_val), False)
    dt = p.dt_fact / 6.1 * min(p.dx, p.dy, p.dz) / max(float(v.abs().max()) for v in V)
    return V, min(dt, p.dt_max) if p.dt_max > 0 else dt, [a, b]


def _exact_step(case, seed, s):
    V, dt, its = _step(s["T0"], s["P0"], s["ktv"], s["kfv"], s["p0"])
    return dict(T=s["T0"], P=s["P0"], V=V, dt=dt, iters=its)


def _exact_ensemble(case, seed, s):
    if case["members"] > 16:
        return None  # members one after the other: over 20 seconds
    r = []
    for m, p in zip(s["members"], s["p0"]):
        T, P = m.Tc_ex.clone(), m.Pc_ex.clone()
        r.append((T, P) + _step(T, P, m.ktv, m.kfv, p))
    flat = lambda ts: torch.cat([t.permute(2, 1, 0).reshape(-1) for t in ts])  # noqa: E731
    return dict(T=flat([x[0] for x in r]), P=flat([x[1] for x in r]), V=[flat([x[2][a] for x in r]) for a in range(3)],
                dt=torch.tensor([x[3] for x in r], dtype=torch.float64), iters=torch.tensor([x[4] for x in r]))


def _exact_solve(case, seed, s):
    h = (float(case["nx"]), float(case["ny"]), float(case["nz"]))
    F, F0, _ = _diffusion(s["X0"], s["R"], s["k"], 0.0, h, SOLVE_BC, SOLVE_VAL, s["prm"], case["iters"])
    return dict(X=s["X0"], F=F, F0=F0)


def _exact_sweep(case, seed, s):
    T = s["T0"].double()
    _weno(T, [v.double() for v in s["V"]], s["dt"], (case["nx"], case["ny"], case["nz"]), s["bc"], SWEEP_VAL,
          case["variant"] == "v2ref")
    return T


# material laws of the dimensional model (T in K unless said otherwise, p in Pa)
def _phi(ph, phi0):
    return phi0 * (1.0 + 2.0 * (ph == 2.0).double())


def _rhof(T, p):  # T in C
    return (1006 + 7.424e-7 * p - 0.3922 * T - 4.441e-15 * p ** 2 + 4.547e-9 * p * T - 0.003774 * T ** 2
            + 1.451e-23 * p ** 3 - 1.793e-17 * p ** 2 * T + 7.485e-12 * p * T ** 2 + 2.955e-6 * T ** 3
            - 1.463e-32 * p ** 4 + 1.361e-26 * p ** 3 * T + 4.018e-21 * p ** 2 * T ** 2 - 7.372e-15 * p * T ** 3
            + 5.698e-11 * T ** 4)


def _drhodp(T, p):  # T in C
    return (-7.372e-15 * T ** 3 + 8.036e-21 * T ** 2 * p + 7.485e-12 * T ** 2 + 4.083e-26 * T * p ** 2
            - 3.586e-17 * T * p + 4.547e-9 * T - 5.852e-32 * p ** 3 + 4.353e-23 * p ** 2 - 8.882e-15 * p + 7.424e-7)


def _kT(T, phi):
    return (1 - phi) * (3.1138 - 0.0023 * T) + phi * (-0.069 + 0.0012 * T)


def _mu(T):
    return 2.414e-5 * torch.pow(10.0, 247.8 / (T - 140.0))


def _exact_post(case, seed, s):
    d, q = s["d"], post.PARAMS
    ph = d["phc"][IN]
    air = ph == 1.0
    T, P, phi = d["T"][IN] * q["scale_T"], d["P"][IN] * q["scale_sigma"], _phi(ph, q["phi0"])
    V = [0.5 * (_axis(d[v], a, 0, -1) + _axis(d[v], a, 1, None)) * q["scale_V"]
         for a, v in enumerate(("Vx", "Vy", "Vz"))]
    y = q["ymin"] + torch.arange(case["ny"], dtype=torch.float64, device="cuda") * q["dy"] + q["dy"] / 2
    kf = (5e-16 * torch.exp(y / q["delta"]))[None, :, None]
    rho, keff = _rhof(T - 273.15, P), _kT(T, phi)
    nan = lambda t: torch.where(air, math.nan, t)  # noqa: E731
    keep = lambda t: torch.where(air, 0.0, t)  # noqa: E731  (air cells stay as they were)
    speed = torch.sqrt(V[0] ** 2 + V[1] ** 2 + V[2] ** 2)
    return dict(phase=nan(ph), pressure=nan(P), temperature=nan(T), vx=nan(V[0]), vy=keep(V[1]), vz=keep(V[2]),
                k_thermal=nan(keff), heat_capacity=keep(0.5915 * T + 636.14),
                permeability=nan(kf * (1.0 + (q["k_fact"] - 1.0) * (ph == 2.0).double())), density=nan(rho),
                viscosity=nan(_mu(T)), peclet=nan(q["scale_L"] * rho * (1000 + 7.5 * T) * speed / keff))


def _at_vertices(A):
    """Mean of a ghosted field's eight cells around each vertex."""
    for a in range(3):
        A = 0.5 * (_axis(A, a, 0, -1) + _axis(A, a, 1, None))
    return A


def _smooth(kv):
    c = _at_vertices(kv)
    kv[IN] = _at_vertices(c)


def _rhoC(T, P, ph, p):
    phi, T, P = _phi(ph, p.phi_i), T * p.sc_T, P * p.sc_sigma
    rho = phi * _rhof(T - 273.15, P) + (1 - phi) * 2800 * (1 - 0.000024 * (T - 293))
    return rho * (phi * (1000 + 7.5 * T) + (1 - phi) * (0.5915 * T + 636.14)) / p.sc_rho / p.sc_C


def _hydro(T, P, kmul, p, mode):
    Tv, Pv = (_at_vertices(T) * p.sc_T).clamp(min=293.15), _at_vertices(P) * p.sc_sigma
    y = p.ymin + torch.arange(T.shape[1] - 1, dtype=torch.float64, device="cuda") * p.dy
    kF = (5e-16 * torch.exp(y / p.delta))[None, :, None] * kmul
    if mode == 1:
        return _rhof(Tv - 273.15, Pv) * kF / _mu(Tv) / p.sc_t
    return kF / _mu(Tv) / (p.sc_L ** 2 / p.sc_eta)


def _density(T, P, p):
    return _rhof(_at_vertices(T) * p.sc_T - 273.15, _at_vertices(P) * p.sc_sigma) / p.sc_rho


def _prf(T, P, ph, p, law=_rhof, scale=1.0):
    return _phi(ph, p.phi_i) * law(T * p.sc_T - 273.15, P * p.sc_sigma) / (p.sc_rho / scale)


def _box_faces(X, p, ky=None):
    """Boundary cells of the box: air above, mirrored sides, the basal flux (heat) or no gradient (pressure) below."""
    for a, end in ((0, 0), (0, 1), (1, 0), (2, 0), (2, 1)):
        g, v = _ghost(X, a, end)
        g.copy_(v + p.qyS * p.dy / ky[:, :1] if a == 1 and ky is not None else v)
    if ky is not None:  # the x rule of the temperature reaches the edges at the front
        X[0, 1:-1, -1], X[-1, 1:-1, -1] = X[1, 1:-1, -1], X[-2, 1:-1, -1]
    X[:, -1] = p.Ttop if ky is not None else p.Ptop


def _darcy_flux(P, k, rfy, p, h):
    return [-k[a] * (_across(P, a) * h[a] - (p.g * rfy if a == 1 else 0.0)) for a in range(3)]


def _exact_v18(case, seed, s):
    p, T, P = s["p0"], s["T0"], s["P0"]
    ph, kmul = s["fixed"][0][IN], s["fixed"][3]
    h, _dt = (1 / p.dx, 1 / p.dy, 1 / p.dz), 1 / p.dt
    T0, P0 = T[IN].clone(), P[IN].clone()
    kv = _kT(_at_vertices(T) * p.sc_T, p.phi_i) / p.sc_kt
    _smooth(kv)
    k = _faces_of_vertices(kv)
    rC = _rhoC(T[IN], P[IN], ph, p)
    PC, G = _gershgorin(k, h, rC * _dt)

    def heat(X):
        return rC * _dt * (X[IN] - T0) + _div([-k[a] * (_across(X, a) * h[a]) for a in range(3)], h)

    _, _, a = _dyrel(T, lambda X: _box_faces(X, p, k[1]), heat, PC, float(G.max()), p.thermal_dyrel)
    kv = _hydro(T, P, kmul, p, 1)
    _smooth(kv)
    u = _faces_of_vertices(kv)
    PC, G = _gershgorin(u, h, _prf(T[IN], P[IN], ph, p, _drhodp, p.sc_sigma) * _dt)
    prf0, rfy = _prf(T0, P0, ph, p), _faces_of_vertices(_density(T, P, p))[1]

    def mass(X):
        return _dt * (_prf(T[IN], X[IN], ph, p) - prf0) + _div(_darcy_flux(X, u, rfy, p, h), h)

    _, _, b = _dyrel(P, lambda X: _box_faces(X, p), mass, PC, float(G.max()), p.darcy_dyrel)
    kv = _hydro(T, P, kmul, p, 2)
    _smooth(kv)
    V = _darcy_flux(P, _faces_of_vertices(kv), _faces_of_vertices(_density(T, P, p))[1], p, h)
    dt_adv = p.C_adv / 6.1 * min(p.dx, p.dy, p.dz) / max(float(v.abs().max()) for v in V)
    n_adv = math.ceil(p.dt / dt_adv)
    for _ in range(n_adv):
        _weno(T, V, p.dt / n_adv, h, [0, 0, 1, 1, 0, 0], [0, 0, p.Tbot, p.Ttop, 0, 0], True)
    return dict(T=T, P=P, V=V, counts=[a, b, n_adv])


def _exact_kernels(case, seed, s):
    p, T, P = s["p"], s["T0"], s["P0"]
    ph, h, _dt = s["d"]["phc"][IN], (1 / p.dx, 1 / p.dy, 1 / p.dz), 1 / p.dt
    T0, P0 = T[IN].clone(), P[IN].clone()
    ktv = _kT(_at_vertices(T) * p.sc_T, p.phi_i) / p.sc_kt
    _smooth(ktv)
    k = _faces_of_vertices(ktv)
    rC = _rhoC(T[IN], P[IN], ph, p)
    D, G = _gershgorin(k, h, rC * _dt)
    _, h2, dtau = _dyrel_scalars(float(G.max()))
    _box_faces(T, p, k[1])
    q = [-k[a] * (_across(T, a) * h[a]) for a in range(3)]
    F = (rC * _dt * (T[IN] - T0) + _div(q, h)) / D
    T[IN] -= dtau * h2 * F
    kfv, rfv = _hydro(T, P, s["d"]["kmul"], p, 1), _density(T, P, p)
    u = _faces_of_vertices(kfv)
    prf0, prf, drdp = _prf(T0, P0, ph, p), _prf(T[IN], P[IN], ph, p), _prf(T[IN], P[IN], ph, p, _drhodp, p.sc_sigma)
    D, Gp = _gershgorin(u, h, drdp * _dt)
    _, h2, dtau = _dyrel_scalars(float(Gp.max()))
    _box_faces(P, p)
    rf = _faces_of_vertices(rfv)
    u = _darcy_flux(P, u, rf[1], p, h)
    Fp = (_dt * (prf - prf0) + _div(u, h)) / D
    P[IN] -= dtau * h2 * Fp
    return dict(T=T, P=P, F=F, Fp=Fp, ktv=ktv, kfv=kfv, rC=rC, G=G, Gp=Gp, q=q, u=u, V=[u[a] / rf[a] for a in range(3)],
                rfv=rfv, prf=prf, drdp=drdp)


_EXACT = dict(step=_exact_step, ensemble=_exact_ensemble, v18=_exact_v18, solve=_exact_solve, sweep=_exact_sweep,
              post=_exact_post, kernels=_exact_kernels)

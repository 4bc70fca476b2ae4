"""Work memory that a call can do without: calls run where it is not to be had, in
a stream capture among others, with the same results."""
import numpy as np
import pytest
import torch

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi, v18

pytestmark = pytest.mark.gpu
TYPES, VALS = (0, 1, 1, 0, 0, 1), (0.0, 0.5, 1.0, 0.0, 0.0, 0.2)


@pytest.fixture
def fresh(gpu_stream):
    """A context of the test's own, with no work memory yet."""
    c = ht.Context(device=0, stream=gpu_stream.cuda_stream)
    yield c
    c.close()


class leaving:
    """Takes the device's memory but for `free` bytes."""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.t = torch.empty(torch.cuda.mem_get_info()[0] - self.free, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        del self.t
        torch.cuda.empty_cache()


def fields(n, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = lambda a, b, c: (torch.rand((c, b, a), generator=g, dtype=torch.float64, device="cuda") + 0.5).permute(2, 1, 0)
    nx, ny, nz = n
    return dict(X=f(nx + 2, ny + 2, nz + 2), R=f(*n), k=[f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1)],
                PC=f(*n), F0=f(*n), F=ht.zeros(*n))


def iterate(ctx, d, n, n_iter):
    ctx.call("ht3d_dyrel_iterate", d["X"].data_ptr(), d["R"].data_ptr(), *[a.data_ptr() for a in d["k"]],
             d["PC"].data_ptr(), d["F0"].data_ptr(), 3.0, 1.0, 1.1, 0.9, abi.int6(*TYPES), abi.dbl6(*VALS), 0.9, 0.02, 0.01,
             n_iter, *n)
    return d["X"], d["F0"]


def solve(ctx, d, n):
    st = api.dyrel_solve_dimless(ctx, d["X"], d["R"], *d["k"], 3.0, 1.0, 1.1, 0.9, TYPES, VALS,
                                 abi.DyrelParams.reference(nitout=5), d["F"], d["F0"], abi.FP64, n_iter_fixed=13)
    assert st.iters == 13
    return d["X"], d["F"], d["F0"]


# the 16 million cells' reciprocals take 122 MB, the rest of the call's memory 125
# (an iteration) and 614 (a solve)
N = (250, 256, 250)


@pytest.mark.parametrize("call,free", [(lambda c, d: iterate(c, d, N, 8), 190 << 20), (lambda c, d: solve(c, d, N), 690 << 20)])
def test_fp64_iterations_without_room_for_reciprocals(ctx, fresh, call, free):
    ref = call(ctx, fields(N))
    iterate(fresh, fields((8, 8, 8)), (8, 8, 8), 8)  # the kernels are loaded
    d = fields(N)
    with leaving(free):
        got = call(fresh, d)
    for a, b in zip(ref, got):
        assert torch.equal(a, b)


def test_reciprocals_give_way_to_what_a_later_call_needs(fresh):
    n = N
    iterate(fresh, fields(n), n, 8)
    d = fields(n)
    V = [ht.zeros(n[0] + 1, n[1], n[2]), ht.zeros(n[0], n[1] + 1, n[2]), ht.zeros(n[0], n[1], n[2] + 1)]
    with leaving(60 << 20):
        api.weno5_advect(fresh, d["X"], *V, 1e-3, 1.0, 1.0, 1.0, [0] * 6, [0.0] * 6, abi.WENO_V1, abi.FP64)
    assert torch.equal(d["X"], fields(n)["X"])


def test_iterations_captured_after_a_shorter_call(gpu_stream):
    """A call of three iterations makes the context's memory; a longer one of the
    same grid can then be captured, and its graph stays good when a larger solve
    takes more of the memory that the context can do without."""
    n = (40, 33, 21)
    c = ht.Context(device=0, stream=gpu_stream.cuda_stream, sync=False)
    ref = [t.clone() for t in iterate(c, fields(n), n, 9)]
    c.close()
    c = ht.Context(device=0, stream=gpu_stream.cuda_stream, sync=False)
    iterate(c, fields(n), n, 3)
    d, start = fields(n), fields(n)
    gpu_stream.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=gpu_stream):
        iterate(c, d, n, 9)
    solve(c, fields((80, 80, 80)), (80, 80, 80))
    for q in ("X", "F0"):
        d[q].copy_(start[q])
    g.replay()
    gpu_stream.synchronize()
    assert torch.equal(d["X"], ref[0]) and torch.equal(d["F0"], ref[1])
    c.close()


def test_dimensional_step_takes_no_memory_beyond_its_fields(fresh):
    """Its work memory: a ghosted field and one of phase codes, the vertex and face
    conductivities and the faces' density, eight cell fields and a check's three
    terms a cell (the reciprocals and the density's temperature terms lie in fields
    that are done with); 2 MB of rounding for each of the eighteen allocations (no
    advection)."""
    n = nx, ny, nz = 128, 120, 100
    b = v18.box(*n, seed=3, nitout=2, nitmax=5)
    b["params"].it, b["params"].advection = 2, 0
    d = [ht.from_numpy(b[k]) for k in ("T", "P", "phc", "phv", "wN", "kmul")]
    V = [ht.zeros(nx + 1, ny, nz), ht.zeros(nx, ny + 1, nz), ht.zeros(nx, ny, nz + 1)]
    small = v18.box(8, 8, 8, seed=3, nitout=2, nitmax=5)
    small["params"].it, small["params"].advection = 2, 0
    c = ht.Context(device=0, stream=fresh.stream)  # loads the kernels
    api.step_v18(c, *[ht.from_numpy(small[k]) for k in ("T", "P", "phc", "phv", "wN", "kmul")], ht.zeros(9, 8, 8),
                 ht.zeros(8, 9, 8), ht.zeros(8, 8, 9), small["params"])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    api.step_v18(fresh, *d, *V, b["params"])
    used = before - torch.cuda.mem_get_info()[0]
    c.close()
    cells, ghosted, vertices = nx * ny * nz, (nx + 2) * (ny + 2) * (nz + 2), (nx + 1) * (ny + 1) * (nz + 1)
    faces = sum(v.numel() for v in V) + V[1].numel()
    assert used <= 8 * (ghosted + vertices + faces + 11 * cells) + ghosted + 18 * (2 << 20)

"""Two contexts of two threads on one GPU, each with resident runs of its own: one
context is a stream and a thread, so their cooperative grids share the chip."""
import threading

import numpy as np
import pytest
import torch

import hydrothermal3d_gb300 as ht
from hydrothermal3d_gb300 import api, abi

pytestmark = pytest.mark.gpu
TYPES, VALS = (0, 1, 1, 0, 1, 0), (0.0, 0.3, 1.0, 0.0, -0.2, 0.0)


def fields(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    f = lambda *s: ht.from_numpy(np.asfortranarray(rng.uniform(0.5, 1.5, s)))
    return [f(nx + 2, ny + 2, nz + 2), f(nx, ny, nz), f(nx + 1, ny, nz), f(nx, ny + 1, nz), f(nx, ny, nz + 1),
            ht.zeros(nx, ny, nz), ht.zeros(nx, ny, nz)]


def solve(ctx, n, d):
    X, R, kx, ky, kz, F, F0 = d
    st = api.dyrel_solve_dimless(ctx, X, R, kx, ky, kz, 30.0, 1.0 / n[0], 0.9 / n[1], 1.2 / n[2], TYPES, VALS,
                                 abi.DyrelParams.reference(nitout=200), F, F0, abi.MIXED, n_iter_fixed=1000)
    assert st.iters == 1000


# grids that fill the chip (63^3: two blocks on most SMs) and one of a few blocks
@pytest.mark.parametrize("sizes", [((63, 63, 63), (63, 63, 63)), ((95, 95, 95), (40, 30, 12))])
def test_two_contexts_solve_at_once(ctx, sizes):
    rounds = 6
    data = [[fields(n, s) for _ in range(rounds + 1)] for s, n in enumerate(sizes)]
    for n, d in zip(sizes, data):
        solve(ctx, n, d[0])
    torch.cuda.synchronize()
    ctxs = [ht.Context(device=0, stream=torch.cuda.Stream().cuda_stream) for _ in sizes]
    start, failed = threading.Barrier(len(sizes)), []

    def work(c, n, d):
        try:
            start.wait(30)
            for r in range(1, rounds + 1):
                solve(c, n, d[r])
        except BaseException as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(c, n, d)) for c, n, d in zip(ctxs, sizes, data)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not failed, failed
    for d in data:
        for r in range(1, rounds + 1):
            for a, b in ((d[0][0], d[r][0]), (d[0][5], d[r][5]), (d[0][6], d[r][6])):
                assert torch.equal(a, b)

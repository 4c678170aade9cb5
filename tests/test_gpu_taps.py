"""FP64 gridding with stored tap weights (single operators and batches) against
the oracle, and against the column walk, which evaluates the polynomials.

Tolerances (relative L2): 1e-12 against the oracle and the walk.  The tap fit
deviates from the kernel by at most 1e-13 of its peak and the sums run over at
most a few hundred terms of FP64 rounding.  A batch is compared with the oracle
too, not bit for bit with a single operator: on grids that are no powers of two
the two run different cuFFT plans."""
import numpy as np
import pytest

from conftest import rel_l2
from purify_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,J,M,weighted", [
    ("kb", 1, 33, False), ("kb", 2, 2000, True), ("kb", 3, 1, False), ("kb", 6, 3001, False),
    ("kb", 7, 500, True), ("kb", 8, 4096, False), ("pswf", 6, 2500, False),
    ("gauss", 4, 31, True)])
def test_stored_taps(pg, oracle_mod, cuda, kernel, J, M, weighted):
    torch = cuda
    n = 48
    rng = np.random.default_rng(J * 1000 + M)
    u, v = synthetic.mixed_uv(M, 2 * n, 2 * n, 0.7, 0.15, seed=J)
    u[0], v[-1] = -n, n - 1e-9  # the grid's edges
    wt = rng.standard_normal(M) + 1j * rng.standard_normal(M) if weighted else None
    x, y = synthetic.sky_image(n, n, seed=J), synthetic.random_vis(M, seed=J)
    args = (u, v, None, wt, n, n, 2.0)
    kw = dict(power_iters=0, kernel=kernel, Ju=J, Jv=J, precision="fp64")
    op = pg.MeasurementOperator(*args, **kw)
    ref = oracle_mod.Operator(*args, kernel=kernel, Ju=J, Jv=J)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    f, a = op.forward(xd), op.adjoint(yd)
    assert rel_l2(f.cpu().numpy(), ref.forward(x)) < 1e-12
    assert rel_l2(a.cpu().numpy(), ref.adjoint(y)) < 1e-12
    if J <= 6:
        walk = pg.MeasurementOperator(*args, tuning={"grid_walk": 1}, **kw)
        assert rel_l2(walk.adjoint(yd).cpu().numpy(), a.cpu().numpy()) < 1e-12
    b = pg.Batch([dict(u=u, v=v, weights=wt, imsizey=n, imsizex=n)] * 2, kernel=kernel, J=J,
                 precision="fp64", tuning={"tile": 32, "degrid_threads": 64, "grid_threads": 64})
    vis, out = [torch.empty_like(yd) for _ in range(2)], [torch.empty_like(xd) for _ in range(2)]
    b.bind([xd, xd], vis, out)
    b.apply(1)
    torch.cuda.synchronize()
    for t in vis:
        assert rel_l2(t.cpu().numpy(), ref.forward(x)) < 1e-12
    for t in vis:
        t.copy_(yd)
    b.apply(2)
    torch.cuda.synchronize()
    assert rel_l2(out[1].cpu().numpy(), a.cpu().numpy()) < 1e-12


@pytest.mark.parametrize("kernel,J,n,M", [
    ("kb", 1, 48, 3000), ("kb", 2, 48, 60000), ("kb", 3, 40, 5000), ("kb", 4, 64, 40000),
    ("kb", 5, 48, 2000), ("kb", 6, 64, 30000), ("kb", 7, 48, 5000), ("kb", 8, 48, 20000),
    ("pswf", 6, 40, 9000), ("gauss", 3, 48, 7000), ("kb", 6, 48, 1)])
def test_table_and_polynomials_give_the_same_bits(pg, cuda, kernel, J, n, M):
    """tap_table = 1 leaves the table out: forward, adjoint and normal have the
    same bits either way, for single operators and for a batch."""
    torch = cuda
    u, v = synthetic.mixed_uv(M, 2 * n, 2 * n, 0.7, 0.15, seed=J)
    rng = np.random.default_rng(J)
    wt = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    kw = dict(power_iters=0, kernel=kernel, Ju=J, Jv=J, precision="fp64")
    xd = torch.from_numpy(synthetic.sky_image(n, n, seed=J)).cuda()
    yd = torch.from_numpy(synthetic.random_vis(M, seed=J)).cuda()
    got, infos = [], []
    for off in (0, 1):
        op = pg.MeasurementOperator(u, v, None, wt, n, n, 2.0, tuning={"tap_table": off}, **kw)
        infos.append(op.info())
        got.append([op.forward(xd), op.adjoint(yd), op.normal(xd)])
        b = pg.Batch([dict(u=u, v=v, weights=wt, imsizey=n, imsizex=n)] * 2, kernel=kernel, J=J,
                     precision="fp64", tuning={"tap_table": off})
        assert (b.info()["tap_table_bytes"] > 0) == (off == 0)
        assert b.tuning["tap_table"] == off
        vis, out = [torch.empty_like(yd) for _ in range(2)], [torch.empty_like(xd) for _ in range(2)]
        b.bind([xd, xd], vis, out)
        b.apply(1)
        torch.cuda.synchronize()
        got[-1] += [t.clone() for t in vis]
        for t in vis:
            t.copy_(yd)
        b.apply(2)
        torch.cuda.synchronize()
        got[-1] += out
    assert infos[0]["tap_table_bytes"] >= 16 * J * M and infos[1]["tap_table_bytes"] == 0
    assert (infos[0]["device_bytes"] - infos[1]["device_bytes"] == infos[0]["tap_table_bytes"])
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_no_table_in_single_precision_or_where_memory_is_promised(pg, cuda):
    """FP32 stores no taps; a coverage of a server whose budget is above the free
    memory stores none either, is built, and gives the same bits."""
    n, M = 48, 4000
    u, v = synthetic.mixed_uv(M, 2 * n, 2 * n, 0.7, 0.15, seed=3)
    args, kw = (u, v, None, None, n, n, 2.0), dict(power_iters=0, Ju=6, Jv=6)
    assert pg.MeasurementOperator(*args, **kw).info()["tap_table_bytes"] == 0
    y = synthetic.random_vis(M, seed=3)
    got = []
    for budget in (1 << 30, 1 << 45):
        srv = pg.Server(slots=1, hbm_budget=budget)
        cov = srv.add_coverage(*args, precision="fp64", **kw)
        got.append(srv.wait(srv.submit(cov, "adjoint", vis=y)))
        srv.close()
    assert np.array_equal(np.asarray(got[0]["x"]), np.asarray(got[1]["x"]))

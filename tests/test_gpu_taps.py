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

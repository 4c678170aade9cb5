"""The fold of the task windows: tiles narrower and wider than a chunk of 32
columns, ragged last tiles, halos of up to 7 rows, tiles with several tasks
(batches of one slot, max_per_item 1) and with none.

Tolerances (relative L2 against the FP64 oracle): FP64 1e-12, as the tap fit
deviates by at most 1e-13 of the peak and sums of a few hundred terms add
rounding of that order; FP32 2e-6, some thirty units of 6e-8 for taps,
products, sums and the FFT."""
import numpy as np
import pytest

from conftest import rel_l2
from purify_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("tile,J,per_item,ny,nx,M", [
    (8, 4, 64, 40, 52, 900), (24, 8, 1, 64, 50, 4000), (32, 4, 1, 64, 64, 20000),
    (33, 5, 64, 47, 66, 3000), (40, 6, 2, 64, 96, 3000), (48, 4, 64, 100, 72, 1),
    (64, 8, 64, 70, 64, 5000)])
def test_fold_tiles(pg, oracle_mod, cuda, precision, tile, J, per_item, ny, nx, M):
    torch = cuda
    u, v = synthetic.mixed_uv(M, 2 * nx, 2 * ny, 0.5, 0.1, seed=tile)
    u[0], v[-1] = -nx, ny - 1e-9  # the grid's edges
    y = synthetic.random_vis(M, seed=J)
    ref = oracle_mod.Operator(u, v, None, None, ny, nx, 2.0, kernel="kb", Ju=J, Jv=J)
    b = pg.Batch([dict(u=u, v=v, imsizey=ny, imsizex=nx)] * 2, kernel="kb", J=J,
                 precision=precision, tuning={"tile": tile, "max_per_item": per_item,
                                              "degrid_threads": 64, "grid_threads": 64})
    yd = torch.from_numpy(y).cuda().to(b.complex_dtype)
    out = [torch.empty(ny, nx, dtype=b.complex_dtype, device="cuda") for _ in range(2)]
    b.bind([torch.zeros_like(t) for t in out], [yd.clone(), yd.clone()], out)
    b.apply(2)
    torch.cuda.synchronize()
    want = ref.adjoint(y).reshape(ny, nx)
    assert torch.equal(out[0], out[1])
    assert rel_l2(out[0].cpu().numpy(), want) < (2e-6 if precision == "fp32" else 1e-12)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n,tile,J,per_item", [
    (112, 8, 4, 64), (120, 8, 4, 64), (117, 8, 8, 1), (112, 8, 8, 1)])
def test_few_and_many_tiles(pg, oracle_mod, cuda, precision, n, tile, J, per_item):
    """Single operators on both sides of the number of tiles from which CTAs have
    128 threads (784 and 900, and ragged ones), halos up to a tile's width."""
    torch = cuda
    M = 4000
    u, v = synthetic.mixed_uv(M, 2 * n, 2 * n, 0.5, 0.1, seed=n)
    y = synthetic.random_vis(M, seed=J)
    op = pg.MeasurementOperator(u, v, None, None, n, n, 2.0, power_iters=0, kernel="kb", Ju=J,
                                Jv=J, precision=precision,
                                tuning={"tile": tile, "max_per_item": per_item})
    ref = oracle_mod.Operator(u, v, None, None, n, n, 2.0, kernel="kb", Ju=J, Jv=J)
    got = op.adjoint(torch.from_numpy(y).to(op.complex_dtype).cuda()).cpu().numpy()
    assert rel_l2(got, ref.adjoint(y)) < (2e-6 if precision == "fp32" else 1e-12)


@pytest.mark.parametrize("n", [64, 341])
def test_wide_halos(pg, cuda, n):
    """Halos of 23 cells (the walk over any halo) on few and on many tiles, against
    the FP64 operator's G^H."""
    torch = cuda
    M = 3000
    rng = np.random.default_rng(n)
    u, v = rng.uniform(-n, n, M), rng.uniform(-n, n, M)
    y = torch.from_numpy(synthetic.random_vis(M, seed=n)).to(torch.complex64).cuda()
    out = []
    for prec, dt in (("fp32", torch.complex64), ("fp64", torch.complex128)):
        op = pg.MeasurementOperator(u, v, None, None, n, n, 2.0, power_iters=0, kernel="kb",
                                    Ju=20, Jv=20, precision=prec, tuning={"row_kernels": 1})
        g = torch.empty(4 * n * n, dtype=dt, device="cuda")
        op.grid_into(y.to(dt), g)
        out.append(g.cpu().numpy())
    assert rel_l2(out[0], out[1]) < 2e-6

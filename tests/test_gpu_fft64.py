"""FP64 row and column passes on power-of-two grids of 128 ... 2048 a side (a side of 64 takes the plan): the
operator against the same one on the strided cuFFT plan (fft_columns 1), with
images that fill their half of the grid, odd ones and single rows or columns.

Tolerance (relative L2): 1e-11 against the oracle at oversampling as low as
1.73, whose 1 / correction amplifies the tap fit's 1e-13; 1e-14 between plans.  A transform of N points has at most 11 levels
of rounding to 1.1e-16 in either implementation, which add up to about
sqrt(22) x 2 x 1.1e-16 = 1e-15 for the two dimensions."""
import numpy as np
import pytest

from conftest import rel_l2
from purify_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(32, 32), (64, 1024), (1024, 64), (128, 512), (256, 256),
                                   (512, 128)])
def test_passes_match_cufft(pg, cuda, ny, nx):
    torch = cuda
    M = 3000
    u, v = synthetic.mixed_uv(M, 2 * nx, 2 * ny, 0.5, 0.2, seed=nx)
    args = (u, v, None, None, ny, nx, 2.0)
    kw = dict(power_iters=0, kernel="kb", Ju=4, Jv=4, precision="fp64")
    own = pg.MeasurementOperator(*args, **kw)
    ref = pg.MeasurementOperator(*args, tuning={"fft_columns": 1}, **kw)
    x = torch.from_numpy(synthetic.sky_image(ny, nx, seed=1)).cuda()
    y = torch.from_numpy(synthetic.random_vis(M, seed=2)).cuda()
    f, a = own.forward(x), own.adjoint(y)
    assert rel_l2(f.cpu().numpy(), ref.forward(x).cpu().numpy()) < 1e-14
    assert rel_l2(a.cpu().numpy(), ref.adjoint(y).cpu().numpy()) < 1e-14


@pytest.mark.parametrize("ny,nx,over", [(37, 37, 1.7298), (33, 66, 1.9395), (50, 25, 2.5601),
                                        (1, 2, 64.0), (74, 74, 1.7298),
                                        (66, 132, 1.9395), (100, 50, 2.5601)])
def test_odd_images(pg, oracle_mod, cuda, ny, nx, over):
    torch = cuda
    M = 500
    Nv, Nu = int(ny * over), int(nx * over)
    assert Nv & (Nv - 1) == 0 and Nu & (Nu - 1) == 0
    rng = np.random.default_rng(ny)
    u, v = rng.uniform(-Nu / 2, Nu / 2, M), rng.uniform(-Nv / 2, Nv / 2, M)
    args = (u, v, None, None, ny, nx, over)
    kw = dict(kernel="kb", Ju=4, Jv=4)
    own = pg.MeasurementOperator(*args, power_iters=0, precision="fp64", **kw)
    ref = oracle_mod.Operator(*args, **kw)
    x, y = synthetic.sky_image(ny, nx, seed=1), synthetic.random_vis(M, seed=2)
    f = own.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    a = own.adjoint(torch.from_numpy(y).cuda()).cpu().numpy()
    assert rel_l2(f, ref.forward(x)) < 1e-11
    assert rel_l2(a, ref.adjoint(y)) < 1e-11

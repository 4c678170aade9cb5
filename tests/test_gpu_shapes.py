"""The launch shapes the planner chooses (2, 4 or 8 warps per CTA) against the
default CTAs on the same coverage (tuning threads): a few dense tiles (many
warps), a sparse wide coverage (few), every support.  G computes each
visibility on its own and G^H flushes in the order of the default's warps, so
both are bit-identical; the one-pass normal operator sums the warps' windows in
another grouping: 2e-6 (FP32) and 1e-13 (FP64) relative L2, a few roundings of
sums of up to eight windows."""
import numpy as np
import pytest

from conftest import rel_l2
from purify_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J", range(1, 9))
@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_chosen_shape_matches_default(pg, cuda, J, dense, precision):
    torch = cuda
    n, M = (64, 60000) if dense else (300, 20000)
    rng = np.random.default_rng(J)
    if dense:
        u, v = rng.normal(0, 9, M), rng.normal(0, 9, M)
    else:
        u, v = synthetic.mixed_uv(M, 2 * n, 2 * n, 0.2, 0.15, seed=J)
    a, b = (pg.MeasurementOperator(u, v, None, None, n, n, 2.0, power_iters=0, kernel="kb", Ju=J,
                                   Jv=J, precision=precision, tuning=t)
            for t in (None, {"threads": 64 if J >= 6 else 128}))
    dt = a.complex_dtype
    x = torch.from_numpy(rng.standard_normal(n * n) + 1j * rng.standard_normal(n * n)).to(dt).cuda()
    y = torch.from_numpy(rng.standard_normal(M) + 1j * rng.standard_normal(M)).to(dt).cuda()
    assert torch.equal(a.forward(x), b.forward(x))
    assert torch.equal(a.adjoint(y), b.adjoint(y))
    tol = 2e-6 if precision == "fp32" else 1e-13
    assert rel_l2(a.normal(x).cpu().numpy(), b.normal(x).cpu().numpy()) < tol


@pytest.mark.parametrize("J", [4, 6, 8])
def test_which_shape_is_chosen(pg, cuda, J):
    """A few dense tiles take more warps than the default in both directions;
    coverages whose tiles fill the chip by themselves keep it in G^H (with more it
    was 1.2 to 1.3 times as slow from J = 6)."""
    default = 2 if J >= 6 else 4

    def warps(n, M, spread, **kw):
        rng = np.random.default_rng(J)
        u, v = (rng.normal(0, spread, M) if spread else rng.uniform(-n, n, M) for _ in range(2))
        op = pg.MeasurementOperator(np.clip(u, -n, n - 1), np.clip(v, -n, n - 1), None, None, n, n,
                                    2.0, power_iters=0, kernel="kb", Ju=J, Jv=J, **kw)
        i = op.info()
        return i["degrid_warps"], i["grid_warps"], i["normal_warps"]
    g, gh, normal = warps(64, 60000, 9)
    assert g > default and gh > default and (normal > 2 if J < 6 else normal == 0)
    assert warps(400, 200000, 0)[1] == default
    assert warps(64, 60000, 9, tuning={"threads": 96})[:2] == (3, 3)

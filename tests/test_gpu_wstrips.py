"""The tensor-core row kernels (FP32 w-projection rows, supports of 9 to 32
taps, Ju != Jv) at the edges of their blocks, against the FP64 oracle.

Tolerance (relative L2): 2e-6.  Operands are split so that a product keeps
about 2^-23 of itself; with sums of a few hundred terms of random sign the
result is within a few times that, 5e-7, and a lost or misplaced tap would
show at 1e-3.  Non-finite values stay inside the footprints they belong to;
the finite rest is held to the same tolerance."""
import numpy as np
import pytest

from conftest import rel_l2
from purify_gb300 import synthetic

pytestmark = pytest.mark.gpu
TOL = 2e-6


def _w(rng, M, N, cell=1.0):
    return rng.uniform(-12, 12, M) * 60.0 * 60.0 * 180.0 / cell / N / np.pi


def _check(pg, oracle_mod, torch, args, kw, okw, ny, nx, seed):
    M = args[0].size
    rng = np.random.default_rng(seed)
    op = pg.MeasurementOperator(*args, ny, nx, 2.0, power_iters=0, precision="fp32", **kw)
    ref = oracle_mod.Operator(*args, ny, nx, 2.0, **okw)
    x = rng.standard_normal(ny * nx) + 1j * rng.standard_normal(ny * nx)
    y = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    xd = torch.from_numpy(x).to(torch.complex64).cuda()
    yd = torch.from_numpy(y).to(torch.complex64).cuda()
    f, a = op.forward(xd), op.adjoint(yd)
    assert rel_l2(f.cpu().numpy(), ref.forward(x)) < TOL
    assert rel_l2(a.cpu().numpy(), ref.adjoint(y)) < TOL
    assert torch.equal(op.normal(xd), op.adjoint(op.forward(xd)))
    assert torch.equal(op.forward(xd), f) and torch.equal(op.adjoint(yd), a)


# supports S = Jw + 3 on both sides of a change in the number of 8-cell blocks
# (S + 7 = 8 k), one visibility, a dense cell, odd and unequal sizes
@pytest.mark.parametrize("Jw,M,ny,nx,dense", [
    (1, 1, 32, 32, False), (6, 2000, 33, 50, False), (7, 3000, 48, 31, False),
    (14, 1500, 64, 40, True), (15, 700, 37, 64, False), (22, 1000, 48, 36, False),
    (29, 800, 31, 62, True)])
def test_w_rows_at_block_edges(pg, oracle_mod, cuda, Jw, M, ny, nx, dense):
    rng = np.random.default_rng(Jw)
    u, v = rng.uniform(-nx, nx, M), rng.uniform(-ny, ny, M)
    if dense:
        u[: M // 2], v[: M // 2] = 3.25 + 0.5 * rng.random(M // 2), -5.75 + 0.5 * rng.random(M // 2)
    w = _w(rng, M, 2 * nx)
    wt = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    kw = dict(kernel="kb", Ju=4, Jv=4, w_term=True, Jw=Jw)
    _check(pg, oracle_mod, cuda, (u, v, w, wt), kw, kw, ny, nx, Jw)


def test_mixed_supports_and_empty_stretches(pg, oracle_mod, cuda):
    n, M = 128, 900  # sparse: tasks are cut at gaps
    rng = np.random.default_rng(2)
    u, v = synthetic.gaussian_core_uv(M, 2 * n, 2 * n, 0.2, seed=3)
    u[:40], v[:40] = rng.uniform(-n, n, 40), rng.uniform(-n, n, 40)
    w = _w(rng, M, 2 * n)
    jw = rng.integers(1, 22, M).astype(np.int32)
    kw = dict(kernel="kb", Ju=4, Jv=4, w_term=True, jw_rows=jw)
    _check(pg, oracle_mod, cuda, (u, v, w, None), kw, kw, n, n, 5)


@pytest.mark.parametrize("kernel,Ju,Jv", [("gauss", 3, 2), ("kb", 9, 9), ("gauss", 18, 18),
                                          ("kb", 25, 25)])
def test_plain_rows(pg, oracle_mod, cuda, kernel, Ju, Jv):
    rng = np.random.default_rng(Ju)
    M, ny, nx = 600, 48, 36
    u, v = rng.uniform(-nx, nx, M), rng.uniform(-ny, ny, M)
    kw = dict(kernel=kernel, Ju=Ju, Jv=Jv)
    _check(pg, oracle_mod, cuda, (u, v, None, None), kw, kw, ny, nx, Ju)


def test_largest_support(pg, cuda):
    """G and G^H alone against the FP64 operator's: the image-plane correction
    of so wide a Gaussian amplifies the FFT's own rounding past the tolerance."""
    torch = cuda
    rng = np.random.default_rng(32)
    M, ny, nx = 600, 31, 62
    u, v = rng.uniform(-nx, nx, M), rng.uniform(-ny, ny, M)
    y = torch.from_numpy(rng.standard_normal(M) + 1j * rng.standard_normal(M)).cuda()
    g = torch.from_numpy(rng.standard_normal(4 * ny * nx) + 1j * rng.standard_normal(4 * ny * nx))
    out = {}
    for prec, dt in (("fp32", torch.complex64), ("fp64", torch.complex128)):
        op = pg.MeasurementOperator(u, v, None, None, ny, nx, 2.0, power_iters=0, kernel="gauss",
                                    Ju=32, Jv=32, precision=prec)
        gd = g.to(torch.complex64).to(dt).cuda()
        vis, grid = torch.empty(M, dtype=dt, device="cuda"), torch.empty_like(gd)
        op.degrid_into(gd, vis)
        op.grid_into(y.to(torch.complex64).to(dt), grid)
        out[prec] = vis.cpu().numpy(), grid.cpu().numpy()
    for a, b in zip(out["fp32"], out["fp64"]):
        assert rel_l2(a, b) < TOL


def test_non_finite_values_stay_in_their_footprint(pg, cuda):
    torch = cuda
    n, M, S = 64, 400, 9
    N = 2 * n
    rng = np.random.default_rng(8)
    u, v = rng.uniform(-20, 20, M), rng.uniform(-20, 20, M)
    w = _w(rng, M, N)
    op = pg.MeasurementOperator(u, v, w, None, n, n, 2.0, power_iters=0, kernel="kb", Ju=4, Jv=4,
                                w_term=True, Jw=S - 3, precision="fp32")
    y = torch.from_numpy(rng.standard_normal(M) + 1j * rng.standard_normal(M)).to(
        torch.complex64).cuda()
    grid0 = torch.empty(N * N, dtype=torch.complex64, device="cuda")
    grid1 = torch.empty_like(grid0)
    k = 7
    q = np.mod(np.floor(u[k] - S / 2) + 1 + np.arange(S), N).astype(int)
    p = np.mod(np.floor(v[k] - S / 2) + 1 + np.arange(S), N).astype(int)
    inside = np.zeros((N, N), bool)
    inside[np.ix_(p, q)] = True
    y[k] = 0
    op.grid_into(y, grid0)
    for bad in (float("inf"), float("nan")):
        y[k] = bad
        op.grid_into(y, grid1)
        g0, g1 = (t.cpu().numpy().reshape(N, N) for t in (grid0, grid1))
        assert not np.isfinite(g1[inside]).any()
        assert np.isfinite(g1[~inside]).all()
        assert rel_l2(g1[~inside], g0[~inside]) < TOL
    # G: a NaN cell reaches the visibilities whose rows hold it
    vis0 = torch.empty(M, dtype=torch.complex64, device="cuda")
    vis1 = torch.empty_like(vis0)
    op.degrid_into(grid0, vis0)
    pc, qc = 3, N - 2
    grid0[pc * N + qc] = float("nan")
    op.degrid_into(grid0, vis1)
    hit = ((np.mod(qc - np.floor(u - S / 2) - 1, N) < S) &
           (np.mod(pc - np.floor(v - S / 2) - 1, N) < S))
    assert hit.any() and not hit.all()
    f0, f1 = vis0.cpu().numpy(), vis1.cpu().numpy()
    assert not np.isfinite(f1[hit]).any() and np.isfinite(f1[~hit]).all()
    assert rel_l2(f1[~hit], f0[~hit]) < TOL


@pytest.mark.parametrize("w_rows", [True, False])
def test_grids_and_visibilities_of_any_alignment(pg, cuda, w_rows):
    """G and G^H on views one element into their buffers (8 bytes past a
    16-byte boundary): the same values are copied, so the bits are those of
    aligned buffers."""
    torch = cuda
    n, M = 48, 700
    N = 2 * n
    rng = np.random.default_rng(21)
    u, v = rng.uniform(-n, n, M), rng.uniform(-n, n, M)
    kw = (dict(kernel="kb", Ju=4, Jv=4, w_term=True, Jw=9) if w_rows else
          dict(kernel="kb", Ju=12, Jv=12))
    op = pg.MeasurementOperator(u, v, _w(rng, M, N) if w_rows else None, None, n, n, 2.0,
                                power_iters=0, precision="fp32", tuning={"row_kernels": 2}, **kw)
    assert op.info()["row_kernels"] == 2
    z = torch.from_numpy(rng.standard_normal(2 * (N * N + M))).float().cuda()
    out = []
    for shift in (0, 1):
        def buf(size):
            t = torch.zeros(size + 2, dtype=torch.complex64, device="cuda")[shift:shift + size]
            assert t.data_ptr() % 16 == 8 * shift
            return t
        g, y = buf(N * N), buf(M)
        g.copy_(torch.view_as_complex(z[:2 * N * N].view(-1, 2)))
        y.copy_(torch.view_as_complex(z[2 * N * N:].view(-1, 2)))
        vis, grid = buf(M), buf(N * N)
        op.degrid_into(g, vis)
        op.grid_into(y, grid)
        out.append((vis, grid))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("data", ["random", "positive", "constant"])
def test_g_and_gh_keep_fp32(pg, cuda, data):
    """G and G^H alone against the FP64 operator: taps of 1 on 3 x 5 cells, so
    that nothing but the values' own splits, products and sums is off.  A
    rounding of FP32 is 2.5e-8 in the mean square; a cell passes one product, one
    block sum and two or three sums outside, 5e-8 or less in all.  Tolerance
    1e-7 (relative L2): values cut to 23 bits without their low x low products
    are 1.3e-7 off on random and 2.0e-7 on constant values."""
    torch = cuda
    n, M = 64, 20000
    rng = np.random.default_rng(3)
    u, v = rng.uniform(-n, n, M), rng.uniform(-n, n, M)

    def values(size):
        if data == "random":
            z = rng.standard_normal(size) + 1j * rng.standard_normal(size)
        elif data == "positive":
            z = rng.random(size) + 1j * rng.random(size)
        else:
            z = np.full(size, 1.2345678 + 0.7654321j)
        return torch.from_numpy(z).to(torch.complex64).cuda()
    g, y = values(4 * n * n), values(M)
    out = {}
    for prec, dt in (("fp32", torch.complex64), ("fp64", torch.complex128)):
        op = pg.MeasurementOperator(u, v, None, None, n, n, 2.0, power_iters=0, kernel="box",
                                    Ju=3, Jv=5, precision=prec, tuning={"row_kernels": 2})
        assert op.info()["row_kernels"] == (2 if prec == "fp32" else 1)
        vis = torch.empty(M, dtype=dt, device="cuda")
        grid = torch.empty(4 * n * n, dtype=dt, device="cuda")
        op.degrid_into(g.to(dt), vis)
        op.grid_into(y.to(dt), grid)
        out[prec] = vis.cpu().numpy(), grid.cpu().numpy()
    for a, b in zip(out["fp32"], out["fp64"]):
        assert rel_l2(a, b) < 1e-7


def _scaled_case(pg, w_rows):
    n, M = 48, 4000
    rng = np.random.default_rng(5)
    u, v = rng.uniform(-n, n, M), rng.uniform(-n, n, M)
    kw = (dict(kernel="kb", Ju=4, Jv=4, w_term=True, Jw=9) if w_rows else
          dict(kernel="kb", Ju=12, Jv=12))
    w = _w(rng, M, 2 * n) if w_rows else None
    ops = [pg.MeasurementOperator(u, v, w, None, n, n, 2.0, power_iters=0, precision=p,
                                  tuning={"row_kernels": 2}, **kw) for p in ("fp32", "fp64")]
    assert ops[0].info()["row_kernels"] == 2
    return ops, rng, n, M, u, v


def _apply(torch, op, g, y, n, M):
    vis = torch.empty(M, dtype=op.complex_dtype, device="cuda")
    grid = torch.empty(4 * n * n, dtype=op.complex_dtype, device="cuda")
    op.degrid_into(g.to(op.complex_dtype), vis)
    op.grid_into(y.to(op.complex_dtype), grid)
    return vis, grid


@pytest.mark.parametrize("w_rows", [True, False])
def test_values_of_any_scale(pg, cuda, w_rows):
    """Powers of two scale G and G^H bit for bit: values far from 1 are brought
    to it by powers of two, and the rest of the arithmetic has no scale.  (The
    values span about 2^12, and the smallest results stay normal numbers.)"""
    torch = cuda
    (op, _), rng, n, M, _, _ = _scaled_case(pg, w_rows)
    draw = lambda size: torch.from_numpy(np.exp(2j * np.pi * rng.random(size)) *  # noqa: E731
                                         2.0 ** rng.uniform(-6, 6, size)).to(torch.complex64).cuda()
    g, y = draw(4 * n * n), draw(M)
    one = _apply(torch, op, g, y, n, M)
    for e in (-84, -70, -40, 70, 95, 110):
        got = _apply(torch, op, g * 2.0 ** e, y * 2.0 ** e, n, M)
        for a, b in zip(got, one):
            assert torch.equal(torch.view_as_real(a), torch.view_as_real(b) * 2.0 ** e), e


@pytest.mark.parametrize("w_rows", [True, False])
def test_scales_side_by_side(pg, cuda, w_rows):
    """G where one half of the grid is 2^-100 of the other: visibilities whose
    taps lie in the small half keep their own relative accuracy; and G^H of a
    few visibilities of 2^70 among ones.  Zero grids give zeros.  Tolerance of
    the file."""
    torch = cuda
    (op, ref), rng, n, M, u, v = _scaled_case(pg, w_rows)
    N, S = 2 * n, 12
    z = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    z[:, N // 2:] *= 2.0 ** -100
    y = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    y[::97] *= 2.0 ** 70
    g = torch.from_numpy(z.ravel()).to(torch.complex64).cuda()
    y = torch.from_numpy(y).to(torch.complex64).cuda()
    got, want = (_apply(torch, o, g, y, n, M) for o in (op, ref))
    q = np.mod(np.floor(u - S / 2) + 1, N)
    small = (q >= N // 2) & (q + S <= N)
    assert small.sum() > 100
    a, b = (t[0].cpu().numpy().astype(np.complex128) for t in (got, want))
    assert rel_l2(a[small] * 2.0 ** 100, b[small] * 2.0 ** 100) < TOL
    assert rel_l2(a[~small], b[~small]) < TOL
    assert rel_l2(got[1].cpu().numpy(), want[1].cpu().numpy()) < TOL
    assert _apply(torch, op, torch.zeros_like(g), y, n, M)[0].abs().max().item() == 0


@pytest.mark.parametrize("row_kernels", [1, 2, 3])
@pytest.mark.parametrize("Jw,M,ny,nx,dense,fits", [
    (1, 1, 32, 32, False, True), (5, 900, 32, 45, False, True), (6, 2000, 32, 45, False, True),
    (6, 2000, 33, 50, False, False), (13, 1500, 64, 40, True, True), (14, 1500, 64, 40, True, True),
    (21, 1000, 48, 36, False, True), (22, 700, 48, 36, True, True), (29, 800, 31, 62, True, False)])
def test_every_choice_of_kernels(pg, oracle_mod, cuda, row_kernels, Jw, M, ny, nx, dense, fits):
    """The band kernels, the tensor-core kernels and G with the one, G^H with the
    other, on both sides of each number of 8-cell blocks, also where the windows
    would not fit and past the largest support (25), where all are the band
    kernels; and the allocation-free entry point."""
    torch = cuda
    rng = np.random.default_rng(Jw)
    u, v = rng.uniform(-nx, nx, M), rng.uniform(-ny, ny, M)
    if dense:
        u[: M // 2], v[: M // 2] = 3.25 + 0.5 * rng.random(M // 2), -5.75 + 0.5 * rng.random(M // 2)
    wt = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    kw = dict(kernel="kb", Ju=4, Jv=4, w_term=True, Jw=Jw)
    args = (u, v, _w(rng, M, 2 * nx), wt)
    tuned = dict(kw, tuning={"row_kernels": row_kernels})
    _check(pg, oracle_mod, cuda, args, tuned, kw, ny, nx, Jw)
    op = pg.MeasurementOperator(*args, ny, nx, 2.0, power_iters=0, precision="fp32", **tuned)
    assert op.info()["row_kernels"] == (row_kernels if fits else 1)
    y = torch.from_numpy(rng.standard_normal(M) + 1j * rng.standard_normal(M)).to(
        torch.complex64).cuda()
    a, b = (torch.empty(4 * ny * nx, dtype=torch.complex64, device="cuda") for _ in range(2))
    op.grid_into(y, a)
    op.grid_no_alloc_into(y, b)
    assert torch.equal(a, b)


def test_kernels_chosen_by_coverage(pg, cuda):
    """Few rows, or rows that are far apart, stay on the band kernels; rows that
    fill the octets go to the tensor-core kernels, G^H before G.  (On either side
    of the estimate the other choice costs about 20% or more.)"""
    def chosen(n, M, core=0.7):
        rng = np.random.default_rng(M)
        c = rng.random(M) < core
        u, v = (np.where(c, np.clip(rng.normal(0, 0.15 * 2 * n, M), -n, n - 1),
                         rng.uniform(-n, n, M)) for _ in range(2))
        w = rng.uniform(-1, 1, M) * 12 * 60.0 * 60.0 * 180.0 / (2 * n) / np.pi
        jw = rng.integers(1, 22, M).astype(np.int32)
        op = pg.MeasurementOperator(u, v, w, None, n, n, 2.0, power_iters=0, kernel="kb", Ju=4,
                                    Jv=4, w_term=True, jw_rows=jw, precision="fp32")
        return op.info()["row_kernels"]
    assert chosen(256, 2000) == 1 and chosen(512, 2000) == 1
    assert chosen(512, 300000) == 2 and chosen(128, 100000) == 2
    assert chosen(1024, 100000, 1.0) == 3

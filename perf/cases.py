"""Performance cases of the measurement operator, each a call that an imaging
program makes through the package's public entry points.

A case is a dict of plain values:

* ``op``: "forward" (Phi x), "adjoint" (Phi^H y), "pair" (Phi x, then Phi^H y),
  "normal" (Phi^H Phi x), "solver" (forward-backward iterations), "host" (a
  pair on complex128 host vectors), "batch" (a pair of many channels in one
  step);
* ``ny``, ``nx``: image size; the grid is twice as large along each axis;
* ``m``: visibilities; ``kernel``, ``j``: gridding kernel and its support;
* ``precision``; ``weights``: natural weights 1 / sigma or none;
* ``wproj``: rows with w-projection supports of 4 to 24 taps per axis;
* ``core``: share of the coverage in the Gaussian core (sigma 0.15 of the grid
  per axis), the rest uniform over the grid.

Coverages, skies and visibilities are synthetic and come from the seed alone;
visibilities arrive in random order.  ``exact`` evaluates the same operator
term by term with torch in 64 bits.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "purify-1_gb300"))

OS = 2.0  # oversampling ratio of every case
J_W = 4  # gridding support of the w-projection rows
BASE = {"ny": 512, "nx": 512, "m": 1_000_000, "kernel": "kb", "j": 4, "precision": "fp32",
        "weights": False, "wproj": False, "core": 0.7}


def _case(name, op, **kw):
    c = dict(BASE, op=op, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a facet or a test image: the whole call is launches and latency
        _case("pair_64", "pair", ny=64, nx=64, m=4000),
        # a snapshot: a small image with the reference's default support
        _case("pair_256", "pair", ny=256, nx=256, m=100_000, core=1.0),
        # one long observation, prediction and dirty image, the wide support
        _case("forward_1024_j6", "forward", ny=1024, nx=1024, m=10_000_000, j=6),
        _case("adjoint_1024_j6", "adjoint", ny=1024, nx=1024, m=10_000_000, j=6),
        # one major cycle at the default support on half as many visibilities
        _case("pair_1024_j4", "pair", ny=1024, nx=1024, m=5_000_000),
        # the operator inside an iterative solver that never leaves the image domain
        _case("normal_512", "normal", m=2_000_000),
        # measured data: sigma weights, an image and a grid that are no powers of two
        _case("pair_weighted_ragged", "pair", ny=1000, nx=700, m=1_234_567, j=5, weights=True),
        # the double-precision operator, used where a result is checked or published
        _case("pair_fp64", "pair", m=2_000_000, j=6, precision="fp64"),
        # wide-field imaging: w-projection rows of 4 to 24 taps per axis
        _case("pair_wproj", "pair", ny=1024, nx=1024, m=2_000_000, wproj=True),
        # the channels of one spectral window, applied together
        _case("batch_16", "batch", channels=16, m=2_000_000),
        # a whole reconstruction: dirty image, then ten proximal iterations
        _case("solver_512", "solver", weights=True, iterations=10),
        # a host program with std::complex<double> vectors
        _case("host_512", "host"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward", "adjoint", "pair", "pair", "normal", "solver", "host", "batch",
                     "wproj", "fp64"])
    c = dict(BASE)
    if rng.random() < 0.5:
        c["ny"] = c["nx"] = rng.choice([64, 128, 256, 512, 1024])
    else:
        c["ny"], c["nx"] = _log(rng, 64, 1024), _log(rng, 64, 1024)
    # denser than 32 visibilities a pixel is not imaged in one piece
    c["m"] = _log(rng, 2000, min(10_000_000, 32 * c["ny"] * c["nx"]))
    c["kernel"] = rng.choice(["kb", "kb", "kb", "kbmin", "gauss", "pswf"])
    c["j"] = 6 if c["kernel"] == "pswf" else rng.choice([2, 3, 4, 4, 5, 6, 6, 7, 8])
    if c["kernel"] == "kbmin":
        c["j"] = max(c["j"], 3)
    c["weights"] = rng.random() < 0.4
    c["core"] = rng.choice([0.0, 0.5, 0.7, 0.9, 1.0])
    if op == "fp64":
        c["precision"], op = "fp64", rng.choice(["forward", "adjoint", "pair", "normal"])
        c["m"] = min(c["m"], _log(rng, 1_000_000, 2_000_000))
    elif op == "wproj":
        c.update(wproj=True, kernel="kb", j=J_W, m=min(c["m"], _log(rng, 500_000, 2_000_000)))
        op = rng.choice(["forward", "adjoint", "pair"])
    elif op == "solver":
        c.update(iterations=rng.randint(3, 10), m=min(c["m"], 2_000_000))
    elif op == "host":
        c["m"] = min(c["m"], 2_000_000)
    elif op == "batch":
        c.update(channels=rng.randint(2, 16), m=min(c["m"], 2_000_000))
    c["op"] = op
    return c


# -- inputs ------------------------------------------------------------------


def _channels(case):
    """The channels of a batch as cases of their own: sizes and counts from
    the case alone (the counts spread over two decades below m)."""
    r = random.Random(case["m"] * 31 + case["channels"])
    out = []
    for k in range(case["channels"]):
        n = r.choice([256, 512, 1024]) if case["ny"] == case["nx"] else None
        ny, nx = (n, n) if n else (max(64, int(case["ny"] * r.uniform(0.5, 1))), case["nx"])
        out.append(dict(case, op="pair", ny=ny, nx=nx, m=_log(r, max(1000, case["m"] // 200),
                                                               case["m"])))
    return out


def _grid_size(case):
    return int(math.floor(case["ny"] * OS)), int(math.floor(case["nx"] * OS))


def _pixel_lambda(n):
    """Width of a grid pixel in wavelengths for cells of one arcsecond."""
    return 60.0 * 60.0 * 180.0 / math.floor(OS * n) / math.pi


def _inputs(case, seed):
    """Coverage and vectors on the GPU in 64 bits, from the seed alone."""
    g = torch.Generator("cuda").manual_seed(int(seed) % (1 << 62))
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)
    m, (nv, nu) = case["m"], _grid_size(case)
    uv = []
    core = torch.rand(m, **f64) < case["core"]
    for n in (nu, nv):
        # the few draws of the core beyond the grid's edge wrap around
        normal = torch.remainder(torch.randn(m, **f64) * (0.15 * n) + n / 2, n) - n / 2
        uv.append(torch.where(core, normal, (torch.rand(m, **f64) - 0.5) * n))
    d = {"u": uv[0], "v": uv[1], "weights": None}
    # point sources over a few extended ones
    ny, nx = case["ny"], case["nx"]
    sky = torch.zeros(ny * nx, dtype=torch.float64, device="cuda")
    where = torch.randint(0, ny * nx, (64,), device="cuda", generator=g)
    sky.index_add_(0, where, torch.randn(64, **f64).exp())
    yy = torch.arange(ny, dtype=torch.float64, device="cuda")[:, None]
    xx = torch.arange(nx, dtype=torch.float64, device="cuda")[None, :]
    for c in torch.rand(3, 2, **f64).tolist():
        r2 = (yy - c[0] * ny) ** 2 + (xx - c[1] * nx) ** 2
        sky += torch.exp(-r2 / (2 * (0.02 * min(ny, nx) + 1) ** 2)).reshape(-1)
    d["x"] = sky.to(torch.complex128)
    d["y"] = torch.complex(torch.randn(m, **f64), torch.randn(m, **f64))
    if case["weights"]:
        d["weights"] = torch.complex(0.5 + 1.5 * torch.rand(m, **f64), torch.zeros_like(uv[0]))
    if case["wproj"]:
        # w up to 12 grid pixels in wavelengths; the support of a row grows
        # affinely with |w|
        w_max = 12.0 * _pixel_lambda(nx)
        w = (2 * torch.rand(m, **f64) - 1) * w_max
        s = torch.clamp(torch.round(4 + 20 * (w - w.mean()).abs() / w_max), 4, 24)
        d["w"], d["jw"] = w, (s - (J_W - 1)).to(torch.int32)
    ctype = torch.complex64 if case["precision"] == "fp32" else torch.complex128
    for k in ("x", "y"):  # the operator's own precision is what a program has in hand
        d[k] = d[k].to(ctype)
    return d


def _np(t):
    return None if t is None else t.cpu().numpy()


def prepare(case, seed):
    import purify_gb300 as pg
    if case["op"] == "batch":
        chans = _channels(case)
        ins = [_inputs(c, seed * 64 + k) for k, c in enumerate(chans)]
        b = pg.Batch([dict(u=_np(d["u"]), v=_np(d["v"]), weights=_np(d["weights"]),
                           imsizey=c["ny"], imsizex=c["nx"]) for c, d in zip(chans, ins)],
                     oversample_ratio=OS, kernel=case["kernel"], J=case["j"],
                     precision=case["precision"])
        st = {"op": "batch", "batch": b, "x": [d["x"] for d in ins],
              "vis": [torch.empty_like(d["y"]) for d in ins],
              "out": [torch.empty_like(d["x"]) for d in ins]}
        b.bind(st["x"], st["vis"], st["out"])
        return st
    d = _inputs(case, seed)
    kw = dict(w=_np(d["w"]), w_term=True, jw_rows=_np(d["jw"])) if case["wproj"] else {}
    o = pg.MeasurementOperator(_np(d["u"]), _np(d["v"]), weights=_np(d["weights"]),
                               imsizey=case["ny"], imsizex=case["nx"], oversample_ratio=OS,
                               power_iters=0, kernel=case["kernel"], Ju=case["j"], Jv=case["j"],
                               precision=case["precision"], **kw)
    st = {"op": case["op"], "o": o, "x": d["x"], "y": d["y"]}
    if case["op"] == "solver":
        o.power_method(POWER_ITERS, 0.0)
        st["iterations"] = case["iterations"]
    if case["op"] == "host":
        st["x"], st["y"] = (_np(d[k]).astype(np.complex128) for k in ("x", "y"))
    return st


POWER_ITERS = 20


def run(state):
    op = state["op"]
    if op == "batch":
        state["batch"].apply(3)
        return [state["vis"], state["out"]]
    o = state["o"]
    if op == "forward":
        return o.forward(state["x"])
    if op == "adjoint":
        return o.adjoint(state["y"])
    if op == "normal":
        return o.normal(state["x"])
    if op == "solver":
        return o.forward_backward(state["y"], iterations=state["iterations"])
    return [o.forward(state["x"]), o.adjoint(state["y"])]  # pair, host


def work(case):
    if case["op"] == "batch":
        each = [work(c) for c in _channels(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n, m, (nv, nu) = case["ny"] * case["nx"], case["m"], _grid_size(case)
    real = 8 if case["precision"] == "fp64" else 4
    cplx = 16 if case["op"] == "host" else 2 * real
    fft = 5.0 * nu * nv * math.log2(nu * nv)
    if case["wproj"]:
        # supports uniform in 4 ... 24, a complex tap from two factor vectors
        taps = sum(s * s for s in range(4, 25)) / 21.0
        cover, gridding = (2 * 14 + 1) * cplx, 8.0 * taps
    else:
        cover = 2 * real + (2 * real if case["weights"] else 0)
        gridding = 4.0 * case["j"] ** 2 + 4.0 * case["j"]
    one = {"bytes": n * cplx + m * (cplx + cover), "flops": fft + m * gridding}
    if case["op"] in ("forward", "adjoint"):
        return one
    if case["op"] == "normal":
        return {"bytes": 2 * n * cplx + m * cover, "flops": 2 * one["flops"]}
    if case["op"] == "solver":
        k = case["iterations"]
        return {"bytes": one["bytes"] + k * (4 * n * cplx + m * cover),
                "flops": (1 + 2 * k) * one["flops"]}
    return {k: 2 * one[k] for k in one}


# -- the same operator in 64 bits ----------------------------------------------

PSWF = (((8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1),
         (1.0, 8.212018e-1, 2.078043e-1), 0.75),
        ((4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2),
         (1.0, 9.599102e-1, 2.918724e-1), 1.0))


def _poly(coef, z):
    acc = torch.zeros_like(z)
    for c in reversed(coef):
        acc = acc * z + c
    return acc


def _pswf(eta):
    """Schwab's rational approximation, m = 6, alpha = 1."""
    part = [_poly(num, eta * eta - b * b) / _poly(den, eta * eta - b * b) for num, den, b in PSWF]
    a = eta.abs()
    return torch.where(a <= 0.75, part[0], torch.where(a <= 1.0, part[1], torch.zeros_like(a)))


def _alpha(kernel, j):
    if kernel == "kbmin":
        return math.pi * math.sqrt(j * j / (OS * OS) * (OS - 0.5) ** 2 - 0.8)
    return 2.34 * j


def _kernel(kernel, j, x):
    if kernel in ("kb", "kbmin"):
        a = torch.tensor(_alpha(kernel, j), dtype=torch.float64, device=x.device)
        r = torch.sqrt(torch.clamp(1 - (2 * x / j) ** 2, min=0))
        return torch.special.i0(a * r) / torch.special.i0(a)
    if kernel == "gauss":
        return torch.exp(-0.5 * (x / (0.31 * j ** 0.52)) ** 2)
    eta = 2 * x / j
    return _pswf(eta) * (1 - eta * eta)


def _correction(kernel, j, x):
    """The kernel's Fourier transform, by which the image is divided."""
    if kernel in ("kb", "kbmin"):
        e = torch.sqrt(((math.pi * x * j) ** 2 - _alpha(kernel, j) ** 2).to(torch.complex128))
        return (torch.sin(e) / e).real / 38828.11016883
    if kernel == "gauss":
        s = 0.31 * j ** 0.52
        return math.sqrt(math.pi / 2) / s * torch.exp(-2 * (x * s * math.pi) ** 2)
    return _pswf(2 * x)


class _Exact:
    """G F Z S of one coverage, each term as it is defined."""

    def __init__(self, case, d):
        self.case, self.d = case, d
        self.nv, self.nu = _grid_size(case)
        ny, nx = case["ny"], case["nx"]
        self.y0 = math.floor(self.nv * 0.5 - ny * 0.5)
        self.x0 = math.floor(self.nu * 0.5 - nx * 0.5)
        ar = dict(dtype=torch.float64, device="cuda")
        sv = _correction(case["kernel"], case["j"],
                         (self.y0 + torch.arange(ny, **ar) + 0.5) / self.nv - 0.5)
        su = _correction(case["kernel"], case["j"],
                         (self.x0 + torch.arange(nx, **ar) + 0.5) / self.nu - 0.5)
        self.s = 1 / (sv[:, None] * su[None, :])
        self.norm = 1.0

    def _rows(self):
        """(slice or index, p, q, value) pieces of G: visibility rows, grid
        rows and columns, and complex or real values of equal shapes."""
        c, d = self.case, self.d
        if c["wproj"]:
            yield from self._wrows()
            return
        j = c["j"]
        for b in range(0, c["m"], 1 << 21):
            e = slice(b, min(b + (1 << 21), c["m"]))
            u, v = d["u"][e], d["v"][e]
            ku, kv = torch.floor(u - j / 2), torch.floor(v - j / 2)
            wt = None if d["weights"] is None else d["weights"][e]
            for a in range(1, j + 1):
                tv = _kernel(c["kernel"], j, v - (kv + a))
                p = torch.remainder(kv + a, self.nv).long()
                for i in range(1, j + 1):
                    val = tv * _kernel(c["kernel"], j, u - (ku + i))
                    val = val * (1 - 2 * torch.remainder(ku + i + kv + a, 2))
                    q = torch.remainder(ku + i, self.nu).long()
                    yield e, p, q, val if wt is None else val * wt

    def _wrows(self):
        d, nu, nv = self.d, self.nu, self.nv
        du, dv = _pixel_lambda(self.case["nx"]), _pixel_lambda(self.case["ny"])
        wc = d["w"] - d["w"].mean()
        j = J_W
        for jw in torch.unique(d["jw"]).tolist():
            all_rows = torch.nonzero(d["jw"] == jw).reshape(-1)
            s = jw + j - 1
            for rows in all_rows.split(40_000):
                u, v, w = d["u"][rows, None], d["v"][rows, None], wc[rows, None]
                kj = torch.arange(1, j + 1, device="cuda")[None, :]
                kw = torch.arange(1, jw + 1, device="cuda")[None, :]
                fu = _kernel("kb", j, u - torch.floor(u - j / 2) - kj)
                fv = _kernel("kb", j, v - torch.floor(v - j / 2) - kj)
                cu, cv = ((t - torch.floor(t - jw / 2) - kw) * x for t, x in ((u, du), (v, dv)))
                inside = ((cv / w).abs() < 1)[:, :, None] & ((cu / w).abs() < 1)[:, None, :]
                ang = -math.pi * (cv[:, :, None] ** 2 + cu[:, None, :] ** 2) / w[:, :, None]
                g = torch.polar(torch.ones_like(ang), ang) / (1j * w[:, :, None])
                g = torch.where(inside, g, torch.ones_like(g)).flip(1, 2)
                val = torch.zeros(len(rows), s, s, dtype=torch.complex128, device="cuda")
                for a in range(j):
                    for i in range(j):
                        val[:, a:a + jw, i:i + jw] += (fv[:, a] * fu[:, i])[:, None, None] * g
                js = torch.arange(1, s + 1, device="cuda")[None, :]
                pu, pv = torch.floor(u - s / 2) + js, torch.floor(v - s / 2) + js
                val *= (1 - 2 * torch.remainder(pv[:, :, None] + pu[:, None, :], 2))
                if d["weights"] is not None:
                    val *= d["weights"][rows][:, None, None]
                p = torch.remainder(pv, nv).long()[:, :, None].expand_as(val)
                q = torch.remainder(pu, nu).long()[:, None, :].expand_as(val)
                yield rows, p, q, val

    def forward(self, x):
        c = self.case
        grid = torch.zeros(self.nv, self.nu, dtype=torch.complex128, device="cuda")
        grid[self.y0:self.y0 + c["ny"], self.x0:self.x0 + c["nx"]] = x.reshape(c["ny"],
                                                                              c["nx"]) * self.s
        grid = torch.fft.fft2(grid, norm="ortho").reshape(-1)
        y = torch.zeros(c["m"], dtype=torch.complex128, device="cuda")
        for e, p, q, val in self._rows():
            t = grid[p * self.nu + q] * val
            y[e] += t if t.dim() == 1 else t.sum((1, 2))
        return y / self.norm

    def adjoint(self, y):
        c = self.case
        grid = torch.zeros(self.nv * self.nu, 2, dtype=torch.float64, device="cuda")
        for e, p, q, val in self._rows():
            t = val.conj() * (y[e] if val.dim() == 1 else y[e][:, None, None])
            grid.index_add_(0, (p * self.nu + q).reshape(-1), torch.view_as_real(t).reshape(-1, 2))
        grid = torch.view_as_complex(grid).reshape(self.nv, self.nu)
        x = torch.fft.ifft2(grid, norm="ortho")
        x = x[self.y0:self.y0 + c["ny"], self.x0:self.x0 + c["nx"]] * self.s
        return x.reshape(-1) / self.norm

    def power_method(self, iters):
        x = torch.ones(self.s.numel(), dtype=torch.complex128, device="cuda")
        x /= math.sqrt(x.numel())
        for _ in range(iters):
            x = self.adjoint(self.forward(x))
            value = torch.linalg.vector_norm(x)
            x /= value
        return math.sqrt(float(value))


def exact(case, seed):
    if case["op"] == "batch":
        vis, out = [], []
        for k, c in enumerate(_channels(case)):
            d = _inputs(c, seed * 64 + k)
            e = _Exact(c, d)
            vis.append(e.forward(d["x"].to(torch.complex128)))
            out.append(e.adjoint(vis[-1]))
        return [vis, out]
    d = _inputs(case, seed)
    e = _Exact(case, d)
    x, y = d["x"].to(torch.complex128), d["y"].to(torch.complex128)
    if case["op"] == "forward":
        return e.forward(x)
    if case["op"] == "adjoint":
        return e.adjoint(y)
    if case["op"] == "normal":
        return e.adjoint(e.forward(x))
    if case["op"] in ("pair", "host"):
        r = [e.forward(x), e.adjoint(y)]
        return [_np(t) for t in r] if case["op"] == "host" else r
    # solver: gradient step, soft threshold, real and positive part
    e.norm = e.power_method(POWER_ITERS)
    b = e.adjoint(y)
    gamma = 1e-3 * float(b.abs().max())
    x = torch.zeros_like(b)
    for _ in range(case["iterations"]):
        t = (x - (e.adjoint(e.forward(x)) - b)).real
        x = torch.clamp(t - gamma, min=0).to(torch.complex128)
    return x, np.full(case["iterations"], gamma)

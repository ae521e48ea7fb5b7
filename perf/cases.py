"""Performance cases: the calls a user of the library makes, over its range.

``listed()`` gives the named cases, ``draw()`` more of the same ranges.  A
case is a dict of plain values; ``prepare`` builds its string on the GPU
(seeded fields, context created and loaded), ``run`` makes one pass through
the public entry points and returns every output, ``work`` counts what a pass
cannot do without, and ``exact`` restates it in plain float64 torch.

Kinds of pass:

* ``relax``: one outer iteration of the string method on a context that goes
  on relaxing -- mode S (steps only), L or C (reparametrization, CG restart,
  steps) -- then the state and the last step's energies.  ``arith`` is fp32,
  fp64 or paired (FP64 fields, float-float passes).  ``compat`` keeps the
  library's defaults (the reference's line polynomial, scanned step and
  spline); otherwise the exact polynomial, step and spline, as the barrier
  pipeline runs.  ``strings`` > 1 advances a parameter sweep in one context.
* ``grad``: energies and their gradient with respect to the fields and to
  (H, eta, gamma) through the autograd function, in either discretisation.
* ``report``: what is written out at the end of a run: energies, B and J,
  flux and windings, arc lengths.

Fields are those of a string in relaxation: the Meissner state turning into
one vortex per component, a smooth vector potential of amplitude 0.2 and
correlation length 5, and noise of 1e-3.  The numbers of an FP32 string are
returned as float32, whatever type carries them through the interface.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from mepgl_gb300 import native
from mepgl_gb300.autograd import GLEnergy
from mepgl_gb300.problem import Problem

MARGIN = 4       # vacuum sites around the superconductor, as in the benchmark strings
INSET = 6        # the winding loop runs inside the superconductor


def _case(name, kind, nx, ny, images, comps, arith, **kw):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "images": images, "comps": comps, "arith": arith,
         "mode": "S", "steps": 0, "compat": False, "thin_film": False, "strings": 1, "link": False, "dx": 0.4}
    c.update(kw)
    return c


def listed():
    return [
        # the plain method at its smallest: one iteration of the reference's loop with its own options
        _case("relax_fp64_small", "relax", 64, 64, 16, 1, "fp64", mode="L", steps=10, compat=True, dx=0.5),
        # the smallest call: ten FP32 steps of an odd-sized string, where launches count
        _case("steps_fp32_small", "relax", 67, 61, 9, 1, "fp32", steps=10),
        # the mixed-precision string's FP32 bulk: one iteration of the barrier pipeline
        _case("relax_fp32_string", "relax", 256, 256, 64, 2, "fp32", mode="L", steps=10),
        # the same string polished in IEEE double
        _case("steps_fp64_string", "relax", 256, 256, 64, 2, "fp64", steps=2),
        # and with float-float passes
        _case("steps_paired_string", "relax", 256, 256, 64, 2, "paired", steps=4),
        # a ragged two-component string in double with cubic reparametrization
        _case("relax_fp64_cubic", "relax", 131, 90, 24, 2, "fp64", mode="C", steps=5, compat=True),
        # a thin film (A frozen), single component, FP32, cubic reparametrization
        _case("relax_fp32_film", "relax", 203, 150, 32, 1, "fp32", mode="C", steps=10, thin_film=True),
        # a large lattice: the state is many times L2
        _case("steps_fp32_large", "relax", 1024, 1024, 64, 2, "fp32", steps=4, dx=0.25),
        # a parameter sweep: sixteen strings of 96 to 384 sites a side and 24 to 64 images in one context
        _case("sweep_fp32", "relax", 240, 240, 44, 1, "fp32", steps=10, strings=16, dx=0.5),
        # differentiation of a large string's energy: forward and backward
        _case("grad_fp64", "grad", 512, 512, 16, 2, "fp64", dx=0.3),
        # the gauge-link functional's energy and gradient, single precision, small and ragged
        _case("grad_link_fp32", "grad", 97, 113, 6, 2, "fp32", link=True),
        # the outputs of a finished double-precision run
        _case("report_fp64", "report", 256, 200, 48, 2, "fp64"),
    ]


#: site-images of the largest drawn pass, per kind and arithmetic (times steps, where it steps)
_MOST = {"fp32": 2.0e8, "fp64": 6.0e6, "paired": 1.2e7, "grad": 4.0e6, "report": 3.0e6}


def draw(rng: random.Random):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["relax"] * 7 + ["grad"] * 2 + ["report"])
    arith = rng.choice(["fp32", "fp32", "fp64", "paired"]) if kind == "relax" else rng.choice(["fp64", "fp64", "fp32"])
    c = _case("", kind, logint(32, 768), logint(32, 768), logint(4, 64), rng.choice([1, 2]), arith,
              dx=rng.choice([0.25, 0.3, 0.4, 0.5]))
    del c["name"]
    if kind == "relax":
        c["mode"] = rng.choice("SLC")
        c["steps"] = rng.choice([2, 4, 5, 10])
        c["compat"] = arith == "fp64" and rng.random() < 0.4
        c["thin_film"] = rng.random() < 0.2
        if arith == "fp32" and c["comps"] == 1 and c["mode"] == "S" and rng.random() < 0.5:
            c["strings"] = rng.choice([3, 16, 20])
            c["nx"], c["ny"] = min(c["nx"], 300), min(c["ny"], 300)
    elif kind == "grad":
        c["link"] = rng.random() < 0.3
    most = _MOST[arith if kind == "relax" else kind]
    while c["nx"] * c["ny"] * c["images"] * max(1, c["steps"]) * c["strings"] > most:
        k = "images" if c["images"] > 8 else ("nx" if c["nx"] > c["ny"] else "ny")
        c[k] = max(4 if k == "images" else 24, c[k] * 3 // 4)
    return c


# ------------------------------------------------------------------ inputs
def _sizes(case):
    """(nx, ny, images) of every string: a sweep's strings lie around the case's size."""
    if case["strings"] == 1:
        return [(case["nx"], case["ny"], case["images"])]
    r = random.Random(case["strings"] * 1000 + case["nx"])
    out = []
    for _ in range(case["strings"]):
        f = r.uniform(0.4, 1.6)
        out.append((max(24, int(case["nx"] * f)), max(24, int(case["ny"] * f)),
                    max(4, int(case["images"] * r.uniform(0.55, 1.45)))))
    return out


def _domain(nx, ny):
    d = np.zeros((ny, nx), np.int32)
    d[MARGIN:ny - MARGIN, MARGIN:nx - MARGIN] = 1
    return d


def _params(case, k):
    """Parameters of string k: the two-component benchmark physics, or a sweep of H and kappa."""
    r = random.Random(77 + k)
    if case["comps"] == 2:
        return dict(a=(-1.0, -0.6), b=(1.0, 1.0), m_xx=(1.0, 1.0), m_yy=(1.0, 2.0), h=0.9, q=(1.0, 0.5 if case["dx"] == 0.25 else 1.0),
                    eta=-0.5, gamma=0.2, delta=0.05)
    if case["strings"] > 1:
        m = r.uniform(1.0, 4.0) / 2
        return dict(a=(-1.0, -1.0), b=(1.0, 1.0), m_xx=(m, 1.0), m_yy=(m, 1.0), h=r.uniform(0.5, 1.2), q=(1.0, 1.0),
                    eta=0.0, gamma=0.0, delta=0.0)
    return dict(a=(-1.0, -1.0), b=(1.0, 1.0), m_xx=(1.0, 1.0), m_yy=(1.0, 1.0), h=0.8, q=(1.0, 1.0), eta=0.0,
                gamma=0.0, delta=0.0)


def _smooth(g, nx, ny, amp, corr):
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    filt = torch.exp(-2 * math.pi ** 2 * corr ** 2 * (kx ** 2 + ky ** 2))
    w = torch.randn((ny, nx), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.ifft2(torch.fft.fft2(w) * filt).real
    return amp * f / f.std()


def _fields(case, seed):
    """Per string: the fields (A, psi_1[, psi_2]) of the case's type, (images, ny, nx, 2) CUDA tensors."""
    dt = torch.float32 if case["arith"] == "fp32" else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    out = []
    for k, (nx, ny, F) in enumerate(_sizes(case)):
        sc = torch.tensor(_domain(nx, ny), device="cuda", dtype=dt)[None, :, :, None]
        t = torch.linspace(0, 1, F, device="cuda", dtype=torch.float64).to(dt)[:, None, None, None]
        ends = [torch.stack([_smooth(g, nx, ny, 0.2, 5.0) for _ in range(2)], -1).to(dt) for _ in range(2)]
        a = torch.lerp(ends[0][None], ends[1][None], t)
        a += 1e-3 * torch.randn(a.shape, generator=g, device="cuda", dtype=dt)
        fields = [a.contiguous()]
        pars = _params(case, k)
        yy, xx = torch.meshgrid(torch.arange(ny, device="cuda", dtype=torch.float64),
                                torch.arange(nx, device="cuda", dtype=torch.float64), indexing="ij")
        for comp in range(case["comps"]):
            inf = math.sqrt(-pars["a"][comp] / pars["b"][comp])
            x = (xx - (MARGIN + 4.3 + 0.04 * nx + 2 * comp)) * case["dx"]
            y = (yy - (ny / 2 - 0.2)) * case["dx"]
            r = torch.sqrt(x * x + y * y)
            amp = inf * torch.tanh(r / math.sqrt(2.0)) / r.clamp_min(1e-12)
            end = torch.stack([amp * x, amp * y], -1).to(dt)
            start = torch.zeros_like(end)
            start[..., 0] = inf
            p = torch.lerp(start[None], end[None], t)
            p += 1e-3 * torch.randn(p.shape, generator=g, device="cuda", dtype=dt)
            fields.append((p * sc).contiguous())
        out.append(fields)
    return out


def _problems(case):
    out = []
    for k, (nx, ny, F) in enumerate(_sizes(case)):
        out.append(Problem.uniform(nx, ny, case["dx"], multicomponent=case["comps"] == 2, thin_film=case["thin_film"],
                                   sc_domain=_domain(nx, ny), comp_domain=np.ones((ny, nx), np.int32),
                                   **_params(case, k)))
    return out


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    probs = _problems(case)
    fields = _fields(case, seed)
    prec = "fp32" if case["arith"] == "fp32" else "fp64"
    torch.cuda.synchronize()
    if case["kind"] == "grad":
        s.fields = [f.requires_grad_(True) for f in fields[0]]
        s.theta = torch.tensor([0.01, probs[0].eta, probs[0].gamma], dtype=torch.float64, requires_grad=True)
        F = case["images"]
        s.weights = torch.linspace(0.5, 1.5, F, device="cuda", dtype=torch.float64)
        s.f = GLEnergy(probs[0], F, prec, discretization=native.DISC_LINK if case["link"] else native.DISC_REFERENCE)
        s.f.context(s.theta.detach().numpy())
        return s
    opts = {}
    if not case["compat"]:
        opts = dict(line_polynomial=native.POLY_EXACT, line_search=native.LS_EXACT, spline=native.SPLINE_FMM)
    if case["arith"] == "paired":
        opts["fp64_arith"] = native.FP64_PAIRED
    if case["strings"] == 1:
        s.ctx = native.StringContext(probs[0], case["images"], prec, **opts)
        s.ctx.set_state_device(*[f.data_ptr() for f in fields[0]])
        # buffers for the state, or for B and the currents
        s.out = [torch.empty_like(f) for f in fields[0]]
        if case["kind"] == "report":
            s.out[0] = torch.empty_like(fields[0][0][..., 0])
    else:
        s.ctx = native.StringBatch(probs, [z[2] for z in _sizes(case)], prec, **opts)
        s.out = []
        for k, f in enumerate(fields):
            _batch(s.ctx, "mepgl_batch_set_state", k, f)
            s.out.append([torch.empty_like(v) for v in f])
    torch.cuda.synchronize()
    return s


def _batch(ctx, call, k, fields):
    """A sweep's string moves between device buffers through the C ABI (the Python class takes host arrays)."""
    p = [f.data_ptr() for f in fields] + [None]
    ctx._check(getattr(ctx.L, call)(ctx.h, k, *p[:3], native.DEVICE))


def _as(case, v):
    v = np.asarray(v)
    return v.astype(np.float32) if case["arith"] == "fp32" else v


def run(s):
    c = s.case
    if c["kind"] == "grad":
        e = s.f(s.fields[0], s.fields[1], s.fields[2] if c["comps"] == 2 else None, s.theta)
        g = torch.autograd.grad((e * s.weights).sum(), s.fields + [s.theta])
        one = (lambda v: v.float()) if c["arith"] == "fp32" else (lambda v: v)
        return {"energy": one(e.detach()), "fields": list(g[:-1]), "theta": one(g[-1])}
    if c["kind"] == "report":
        p = [t.data_ptr() for t in s.out] + [None]
        e = s.ctx.compute_free_energy()
        s.ctx._check(s.ctx.L.mepgl_compute_jb(s.ctx.h, *p[:3], native.DEVICE))
        o = s.ctx.observables(INSET)
        return {"energy": _as(c, e), "b_j": s.out, "flux": _as(c, o["phi"]), "winding_1": _as(c, o["w_1"]),
                "winding_2": None if c["comps"] == 1 else _as(c, o["w_2"]),
                "arc": _as(c, s.ctx.arc_length()), "arc_jb": _as(c, s.ctx.arc_length_jb())}
    s.ctx.loop_iteration(c["mode"], c["steps"])
    if c["strings"] == 1:
        s.ctx.get_state_device(*[t.data_ptr() for t in s.out])
        return {"state": s.out, "energy": _as(c, s.ctx.image_scalars()["fenergy"])}
    # a sweep reports its energies; its states stay on the device until it ends, except the first one's
    _batch(s.ctx, "mepgl_batch_get_state", 0, s.out[0])
    return {"state": s.out[0],
            "energy": _as(c, np.concatenate([s.ctx.string_scalars(k)["fenergy"] for k in range(len(s.ctx.Fs))]))}


def work(case):
    """Bytes: a step reads x, g and d and writes them; a reparametrization reads and writes x; a gradient reads the
    fields and writes theirs, a report reads them and writes B and J.  Operations: those of the functional per site
    (about 60 for the energy, 110 for its gradient, 190 for the line quartic of one component; 150, 260, 420 of two)."""
    rs = 4 if case["arith"] == "fp32" else 8
    two = case["comps"] == 2
    sites = sum(nx * ny * F for nx, ny, F in _sizes(case))
    masks = sum(2 * nx * ny for nx, ny, F in _sizes(case))
    S = rs * (2 + 2 * case["comps"])
    e, g, p = (150, 260, 420) if two else (60, 110, 190)
    if case["kind"] == "grad":
        return {"bytes": 2.0 * S * sites + masks, "flops": float((e + g) * sites)}
    if case["kind"] == "report":
        return {"bytes": float((S + rs * (1 + 2 * case["comps"])) * sites + masks), "flops": float((e + g) * sites)}
    n = case["steps"]
    b = n * (6.0 * S * sites + masks)
    f = n * float((g + p) * sites)
    if case["mode"] != "S":
        b += 2.0 * S * sites
        f += (g if case["mode"] == "L" else 2 * g) * float(sites)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- float64 restatement
def _shift(f, dx, dy):
    """f at (i + dx, j + dy); zero outside.  f: (..., ny, nx)."""
    out = torch.zeros_like(f)
    ny, nx = f.shape[-2:]
    out[..., max(0, -dy):ny - max(0, dy), max(0, -dx):nx - max(0, dx)] = \
        f[..., max(0, dy):ny + min(0, dy), max(0, dx):nx + min(0, dx)]
    return out


class _Gl:
    """The functional of one string on (images, ny, nx) planes: [A_x, A_y, Re psi_1, Im psi_1, ...]."""

    def __init__(self, case, k, nx, ny):
        self.p = _params(case, k)
        self.nc, self.film, self.link, self.dx = case["comps"], case["thin_film"], case["link"], case["dx"]
        s = torch.tensor(_domain(nx, ny), device="cuda", dtype=torch.float64)
        self.sc = s
        pl = s * _shift(s, 1, 0) * _shift(s, 0, 1) * _shift(s, 1, 1)
        self.area = (pl + _shift(pl, -1, 0) + _shift(pl, 0, -1) + _shift(pl, -1, -1)) / 4
        self.wl = [(pl + _shift(pl, 0, -1)) / 2, (pl + _shift(pl, -1, 0)) / 2]
        self.lk = [s * _shift(s, 1, 0), s * _shift(s, 0, 1)]
        o = torch.ones_like(s)
        pc = o * _shift(o, 1, 0) * _shift(o, 0, 1) * _shift(o, 1, 1)
        self.views = [pc, _shift(pc, -1, 0), _shift(pc, -1, -1), _shift(pc, 0, -1)]

    def line(self, x, d, h=None, eta=None, gamma=None):
        """Per image the coefficients of F(x + t d); d None: the energy alone."""
        p, idx, dx2 = self.p, 1 / self.dx, self.dx ** 2
        h = p["h"] if h is None else h
        eta = p["eta"] if eta is None else eta
        gamma = p["gamma"] if gamma is None else gamma
        n = 1 if d is None else 5

        def mul(u, v):
            w = [0] * min(n, len(u) + len(v) - 1)
            for i, a in enumerate(u):
                for j, b in enumerate(v):
                    if i + j < n:
                        w[i + j] = w[i + j] + a * b
            return w

        def add(*us):
            return [sum(u[i] for u in us if i < len(u)) for i in range(max(map(len, us)))]

        def sca(k, u):
            return [k * a for a in u]

        def sh(u, dx_, dy_):
            return [_shift(a, dx_, dy_) for a in u]

        f = [[v] if d is None else [v, d[i]] for i, v in enumerate(x)]
        tot = [0] * n
        ps = [(f[2 + 2 * c], f[3 + 2 * c]) for c in range(self.nc)]
        r = [add(mul(re, re), mul(im, im)) for re, im in ps]
        cond = [0]
        for c in range(self.nc):
            m = add([p["a"][c] / p["b"][c]], r[c])
            cond = add(cond, sca(p["b"][c] / 2, mul(m, m)))
        if self.nc == 2:
            R = add(mul(ps[0][0], ps[1][0]), mul(ps[0][1], ps[1][1]))
            I = add(mul(ps[0][0], ps[1][1]), sca(-1, mul(ps[0][1], ps[1][0])))
            cond = add(cond, sca(eta, R), sca(gamma / 2, mul(r[0], r[1])),
                       sca(p["delta"] / 2, add(mul(R, R), sca(-1, mul(I, I)))))
        tot = add(tot, sca(self.area * dx2, cond))
        for e in range(2):
            o = (1, 0) if e == 0 else (0, 1)
            A, An = f[e], sh(f[e], *o)
            for c in range(self.nc):
                q, m = p["q"][c], (p["m_xx"] if e == 0 else p["m_yy"])[c]
                re, im = ps[c]
                ren, imn = sh(re, *o), sh(im, *o)
                if self.link:
                    ph = q * A[0] * self.dx
                    zr = ren[0] - (torch.cos(ph) * re[0] - torch.sin(ph) * im[0])
                    zi = imn[0] - (torch.sin(ph) * re[0] + torch.cos(ph) * im[0])
                    tot = add(tot, [self.wl[e] / (2 * m) * (zr * zr + zi * zi)])
                    continue
                dr, di = sca(-idx, add(ren, sca(-1, re))), sca(idx, add(imn, sca(-1, im)))
                for base, a, b in ((dr, A, im), (dr, An, imn), (di, A, re), (di, An, ren)):
                    u = add(base, sca(-q, mul(a, b)))
                    tot = add(tot, sca(self.wl[e] * dx2 / (4 * m), mul(u, u)))
        if not self.film:
            if self.link:
                B = (x[0] + _shift(x[1], 1, 0) - _shift(x[0], 0, 1) - x[1]) * idx - h
                tot = add(tot, [self.views[0] * dx2 / 2 * B * B])
            else:
                ey = [sca(idx, add(sh(f[1], 1, 0), sca(-1, f[1]))), sca(idx, add(f[1], sca(-1, sh(f[1], -1, 0))))]
                ex = [sca(idx, add(sh(f[0], 0, 1), sca(-1, f[0]))), sca(idx, add(f[0], sca(-1, sh(f[0], 0, -1))))]
                for w, a, b in zip(self.views, (0, 1, 1, 0), (0, 0, 1, 1)):
                    u = add(ey[a], sca(-1, ex[b]), [-h])
                    tot = add(tot, sca(w * dx2 / 8, mul(u, u)))
        return [v.sum((-2, -1)) for v in tot]

    def gradient(self, x, **kw):
        x = [v.detach().requires_grad_(True) for v in x]
        with torch.enable_grad():
            e = self.line(x, None, **kw)[0]
            wrt = x[2:] if self.film else x
            g = list(torch.autograd.grad(e.sum(), wrt))
        if self.film:
            g = [torch.zeros_like(x[0]), torch.zeros_like(x[1])] + g
        return e.detach(), g

    def jb(self, x):
        """B, [J_x, J_y per component]."""
        p, idx = self.p, 1 / self.dx
        ey = [(_shift(x[1], 1, 0) - x[1]) * idx, (x[1] - _shift(x[1], -1, 0)) * idx]
        ex = [(_shift(x[0], 0, 1) - x[0]) * idx, (x[0] - _shift(x[0], 0, -1)) * idx]
        b = sum(w * (ey[i] - ex[j]) for w, i, j in zip(self.views, (0, 1, 1, 0), (0, 0, 1, 1)))
        b = b / sum(self.views)
        js = []
        for c in range(self.nc):
            re, im = x[2 + 2 * c], x[3 + 2 * c]
            j = []
            for e in range(2):
                o = (1, 0) if e == 0 else (0, 1)
                q, k = p["q"][c], p["q"][c] / (2 * (p["m_xx"] if e == 0 else p["m_yy"])[c])
                out = 0
                for sgn in (1, -1):
                    rn, im_n = _shift(re, sgn * o[0], sgn * o[1]), _shift(im, sgn * o[0], sgn * o[1])
                    w = self.lk[e] if sgn == 1 else _shift(self.lk[e], -o[0], -o[1])
                    dr, di = sgn * (rn - re) * idx, sgn * (im_n - im) * idx
                    out = out + w * k * (im * (-dr - q * x[e] * im) + re * (di - q * x[e] * re))
                j.append(out)
            js.append(j)
        return b, js


def _planes(fields, lo=None, hi=None):
    return [f[lo:hi, :, :, k].detach().double() for f in fields for k in range(2)]


def _pairs(planes):
    return [torch.stack(planes[2 * k:2 * k + 2], -1) for k in range(len(planes) // 2)]


def _first_minimum(c):
    """Smallest positive root of the quartic's derivative with positive curvature."""
    der = np.array([4 * c[4], 3 * c[3], 2 * c[2], c[1]])
    best = None
    for z in np.roots(der):
        if abs(z.imag) > 1e-9 * max(1.0, abs(z)):
            continue
        t = z.real
        for _ in range(3):
            dd = np.polyval(np.polyder(der), t)
            t = t - np.polyval(der, t) / dd if dd else t
        if t > 0 and np.polyval(np.polyder(der), t) > 0 and (best is None or t < best):
            best = t
    return best


def _steps(gl, x, steps):
    """Nonlinear CG from a fresh history: the fields after it and the energies before its last step."""
    d = gp = gn = None
    for _ in range(steps):
        _, g = gl.gradient(x)
        sq = sum((v * v).sum((-2, -1)) for v in g)
        if d is None:
            d = [-v for v in g]
        else:
            b = sum((v * (v - w)).sum((-2, -1)) for v, w in zip(g, gp)) / gn
            b = b.clamp_min(0)[:, None, None]
            d = [b * w - v for v, w in zip(g, d)]
        gp, gn = g, sq
        coef = torch.stack(gl.line(x, d)).cpu().numpy()
        t = [_first_minimum(coef[:, n]) for n in range(coef.shape[1])]
        if any(v is None for v in t):
            return None
        t = torch.tensor(t, device="cuda", dtype=torch.float64)[:, None, None]
        x = [v + t * w for v, w in zip(x, d)]
    return x, torch.tensor(coef[0])


def _arc(planes):
    d = sum(((v[1:] - v[:-1]) ** 2).sum((-2, -1)) for v in planes).sqrt()
    s = torch.cat([torch.zeros(1, device=d.device, dtype=d.dtype), d.cumsum(0)])
    return (s / s[-1]).cpu().numpy()


def _resample(gl, x, cubic):
    """Equidistant images in the (B, J) metric: linear, or the Forsythe-Malcolm-Moler spline."""
    b, js = gl.jb(x)
    s = _arc([b] + [v for j in js for v in j])
    F = len(s)
    t = np.arange(F) / (F - 1)
    k = np.minimum(np.maximum(np.searchsorted(s, t, side="left"), 1), F - 1)
    h = np.diff(s, prepend=0.0)
    w = (t - s[k - 1]) / h[k]
    W = np.zeros((F, F))
    W[np.arange(F), k] += w
    W[np.arange(F), k - 1] += 1 - w
    if cubic:
        D = np.zeros((F, F))       # first divided differences of the images
        for n in range(1, F):
            D[n, n], D[n, n - 1] = 1 / h[n], -1 / h[n]
        M, rhs = np.zeros((F, F)), np.zeros((F, F))
        for n in range(1, F - 1):
            M[n, n - 1], M[n, n], M[n, n + 1] = h[n], 2 * (h[n] + h[n + 1]), h[n + 1]
            rhs[n] = D[n + 1] - D[n]
        third = lambda q: ((D[q + 2] - D[q + 1]) / (h[q + 2] + h[q + 1]) - (D[q + 1] - D[q]) / (h[q + 1] + h[q])) / \
            (h[q] + h[q + 1] + h[q + 2])  # noqa: E731
        M[0, 0], M[0, 1], rhs[0] = -h[1], h[1], h[1] ** 2 * third(1)
        M[-1, -2], M[-1, -1], rhs[-1] = h[F - 1], -h[F - 1], -h[F - 1] ** 2 * third(F - 3)
        sig = np.linalg.solve(M, rhs)
        u = 1 - w
        W = W + (h[k] ** 2 * (w ** 3 - w))[:, None] * sig[k] + (h[k] ** 2 * (u ** 3 - u))[:, None] * sig[k - 1]
    W = torch.tensor(W, device="cuda", dtype=torch.float64)
    return [torch.einsum("mn,nyx->myx", W, v) for v in x]


def _winding(re, im):
    ny, nx = re.shape[-2:]
    i0, i1, j0, j1 = INSET, nx - 1 - INSET, INSET, ny - 1 - INSET
    path = [(i, j0) for i in range(i0, i1)] + [(i1, j) for j in range(j0, j1)] + \
        [(i, j1) for i in range(i1, i0, -1)] + [(i0, j) for j in range(j1, j0, -1)]
    ii = torch.tensor([p[0] for p in path], device="cuda")
    jj = torch.tensor([p[1] for p in path], device="cuda")
    u, v = re[:, jj, ii], im[:, jj, ii]
    du, dv = u.roll(-1, 1) - u, v.roll(-1, 1) - v
    return ((u * dv - v * du) / (u * u + v * v)).sum(1).cpu()


def exact(case, seed):
    with torch.no_grad():
        return _exact(case, seed)


def _exact(case, seed):
    fields = _fields(case, seed)
    sizes = _sizes(case)
    gl = _Gl(case, 0, *sizes[0][:2])
    if case["kind"] == "grad":
        F = case["images"]
        w = torch.linspace(0.5, 1.5, F, device="cuda", dtype=torch.float64)
        es, gs = [], []
        th = torch.tensor([gl.p["h"] + 0.01, gl.p["eta"], gl.p["gamma"]], dtype=torch.float64, device="cuda",
                          requires_grad=True)
        gt = torch.zeros(3, dtype=torch.float64, device="cuda")
        for n in range(0, F, 4):
            x = [v.requires_grad_(True) for v in _planes(fields[0], n, n + 4)]
            with torch.enable_grad():
                e = gl.line(x, None, h=th[0], eta=th[1], gamma=th[2])[0]
                g = torch.autograd.grad((e * w[n:n + 4]).sum(), x + [th], allow_unused=True)
            es.append(e.detach())
            gs.append(_pairs(list(g[:-1])))
            gt += 0 if g[-1] is None else g[-1]
        return {"energy": torch.cat(es), "fields": [torch.cat([g[f] for g in gs]) for f in range(1 + case["comps"])],
                "theta": gt.cpu()}
    if case["kind"] == "report":
        x = _planes(fields[0])
        b, js = gl.jb(x)
        e = torch.cat([gl.line(_planes(fields[0], n, n + 4), None)[0] for n in range(0, case["images"], 4)])
        jp = [v for j in js for v in j]
        big = min(sizes[0][:2]) > 2 * INSET + 2
        return {"energy": e, "b_j": [b] + _pairs(jp), "flux": (b.sum((-2, -1)) * case["dx"] ** 2).cpu(),
                "winding_1": _winding(x[2], x[3]) if big else None,
                "winding_2": _winding(x[4], x[5]) if big and case["comps"] == 2 else None,
                "arc": _arc(x), "arc_jb": _arc([b] + jp)}
    if case["compat"]:
        return None       # the reference's own slips have no other definition
    state, energy = None, []
    for k, (nx, ny, F) in enumerate(sizes):
        gl = _Gl(case, k, nx, ny)
        f = fields[k]
        if case["mode"] != "S":
            f = _pairs(_resample(gl, _planes(f), case["mode"] == "C"))
        chunk, xs = 8, []
        for n in range(0, F, chunk):
            r = _steps(gl, _planes(f, n, n + chunk), case["steps"])
            if r is None:
                return None
            energy.append(r[1])
            if k == 0:
                xs.append(_pairs(r[0]))
        if k == 0:
            state = [torch.cat([v[i] for v in xs]) for i in range(1 + case["comps"])]
    return {"state": state, "energy": torch.cat(energy)}

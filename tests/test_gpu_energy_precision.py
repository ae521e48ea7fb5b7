"""Energies of vortex lattices in a strong vector potential, where the kinetic
terms |grad psi|^2, A . J and A^2 |psi|^2 cancel almost entirely, against long
double.  The fields and parameters are exact in the type; what remains is the
rounding of the folded constants (q dx, 1 / (2 m dx^2)), which must act as a
change of dx or m by a unit and not as a mismatch between the terms, and the
rounding of the sites' sums, which averages out: two units of roundoff in FP32
and float-float, four in FP64, whose result is itself rounded to one, of what
the energy is the sum of (kinetic, condensation, coupling and magnetic energy
without their signs)."""
import numpy as np
import pytest

from mepgl_gb300.problem import Problem, StringState

pytestmark = pytest.mark.gpu

LD = np.longdouble
PARS = {1: dict(a=(-1.0, -1.0), b=(1.0, 1.0), m_xx=(1.0, 1.0), m_yy=(1.0, 1.0), eta=0.0, gamma=0.0, delta=0.0),
        2: dict(a=(-1.0, -0.5), b=(1.0, 1.0), m_xx=(1.0, 1.0), m_yy=(1.0, 2.0), eta=-0.5, gamma=0.25, delta=0.0625)}


def lattice(vortices, n, dx, comps, images, dtype):
    """vortices^2 vortices on n^2 sites, A of their mean field in the symmetric gauge."""
    size = n * dx
    field = 2 * np.pi * vortices ** 2 / size ** 2
    yy, xx = np.mgrid[0:n, 0:n]
    x, y = (xx - n / 2 + 0.5) * dx, (yy - n / 2 + 0.5) * dx
    psi = np.ones((n, n), complex)
    for i in range(vortices):
        for j in range(vortices):
            z = (x - (i + 0.5 - vortices / 2) * size / vortices) + 1j * (y - (j + 0.5 - vortices / 2) * size / vortices)
            psi *= np.tanh(abs(z) / np.sqrt(2)) * z / np.maximum(abs(z), 1e-12)
    s = (1 + 0.02 * np.arange(images))[:, None, None, None]
    f = [s * np.stack([-field * y / 2, field * x / 2], -1)] + \
        [k * s * np.stack([psi.real, psi.imag], -1) for k in (1.0, 0.77)[:comps]]
    f = [np.ascontiguousarray(v.astype(dtype)) for v in f]
    return StringState(a=f[0], psi_1=f[1], psi_2=f[2] if comps == 2 else None)


def energy(a, psis, dx, h, p):
    """Free energy of one image on a full rectangular domain, in long double, and
    the sum of its parts without their signs."""
    a, dx = a.astype(LD), LD(dx)
    psis = [v.astype(LD) for v in psis]
    ny, nx = a.shape[:2]
    wx, wy = np.ones(nx, LD), np.ones(ny, LD)
    wx[[0, -1]] = wy[[0, -1]] = LD(0.5)
    r = [v[..., 0] ** 2 + v[..., 1] ** 2 for v in psis]
    nl = sum(LD(p["b"][k]) / 2 * (LD(p["a"][k]) / LD(p["b"][k]) + r[k]) ** 2 for k in range(len(psis)))
    if len(psis) == 2:
        (x1, y1), (x2, y2) = ((v[..., 0], v[..., 1]) for v in psis)
        re, im = x1 * x2 + y1 * y2, x1 * y2 - y1 * x2
        nl = [nl, LD(p["eta"]) * re, LD(p["gamma"]) / 2 * r[0] * r[1], LD(p["delta"]) / 2 * (re ** 2 - im ** 2)]
    parts = [(v * wx * wy[:, None]).sum() for v in (nl if len(psis) == 2 else [nl])]
    for k, v in enumerate(psis):
        for axis, w, m in ((1, wy[:, None], p["m_xx"][k]), (0, wx, p["m_yy"][k])):
            lo = tuple(slice(0, -1) if q == axis else slice(None) for q in range(2))
            hi = tuple(slice(1, None) if q == axis else slice(None) for q in range(2))
            ae = a[..., 1 - axis]
            d = (v[hi] - v[lo]) / dx
            u = sum((d[..., 0] + ae[s] * v[s][..., 1]) ** 2 + (d[..., 1] - ae[s] * v[s][..., 0]) ** 2 for s in (lo, hi))
            parts.append((w * u).sum() / (4 * LD(m)))
    ex, ey = (a[:, 1:, 1] - a[:, :-1, 1]) / dx, (a[1:, :, 0] - a[:-1, :, 0]) / dx
    parts.append(sum(((b - l - LD(h)) ** 2).sum() for b in (ex[:-1], ex[1:]) for l in (ey[:, :-1], ey[:, 1:])) / 8)
    return sum(parts) * dx * dx, sum(abs(v) for v in parts) * dx * dx


@pytest.mark.parametrize("arith,comps,vortices,n,dx,h", [
    ("fp32", 1, 10, 300, 0.35, 0.125), ("fp32", 1, 9, 160, 0.3, 0.125), ("fp32", 1, 8, 256, 0.4, 0.125),
    ("fp32", 1, 6, 150, 0.45, 0.125), ("fp64", 1, 8, 256, 0.4, 0.125), ("fp64", 2, 8, 256, 0.4, 0.75),
    ("fp64", 2, 10, 300, 0.35, 0.125), ("paired", 2, 10, 300, 0.35, 0.75), ("paired", 2, 10, 300, 0.35, 0.125),
    ("paired", 1, 10, 300, 0.35, 0.125)])
def test_energy_of_vortex_lattices(arith, comps, vortices, n, dx, h):
    from mepgl_gb300 import native
    p = PARS[comps]
    prob = Problem.uniform(n, n, dx, multicomponent=comps == 2, thin_film=False, h=h, q=(1.0, 1.0), **p)
    st = lattice(vortices, n, dx, comps, 3, np.float32 if arith == "fp32" else np.float64)
    kw = dict(line_search=1, line_polynomial=1)
    if arith == "paired":
        kw["fp64_arith"] = native.FP64_PAIRED
    c = native.StringContext(prob, 3, "fp32" if arith == "fp32" else "fp64", **kw)
    c.set_state(st)
    e = c.compute_free_energy()
    c.nlcg_steps(1)
    q = c.image_scalars()["fenergy"]        # the quartic's constant: the energy before the step
    c.close()
    want = [energy(st.a[k], [v[k] for v in (st.psi_1, st.psi_2) if v is not None], dx, h, p) for k in range(3)]
    u = {"fp32": 2.0 * 2.0 ** -24, "fp64": 4.0 * 2.0 ** -53, "paired": 2.0 * 2.0 ** -48}
    for got, tol in ((e, u["fp32" if arith == "fp32" else "fp64"]), (q, u[arith])):
        err = max(float(abs((LD(v) - w) / s)) for v, (w, s) in zip(got, want))
        assert err <= tol, (err, tol)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nx,ny", [(97, 40), (33, 18)])
def test_a_uniform_field_leaves_no_rounding_in_the_gradient(precision, nx, ny):
    """dF/dA of a string without psi and with A of 1e-3 in a field of 0.9: at sites
    with all their views the field cancels exactly, and what is left is sums of
    about ten differences of A, each a rounding of its own size."""
    from mepgl_gb300 import native
    dtype = np.float32 if precision == "fp32" else np.float64
    prob = Problem.uniform(nx, ny, 0.4, h=0.9)
    a = (1e-3 * np.random.default_rng(5).standard_normal((2, ny, nx, 2))).astype(dtype)
    c = native.StringContext(prob, 2, precision)
    c.set_state(StringState(a=a, psi_1=np.zeros_like(a), psi_2=None))
    got = c.energy_grad()[1][0].astype(LD)[:, 2:-2, 2:-2]
    c.close()
    x = a.astype(LD)
    ex, ey = x[:, :, 1:, 1] - x[:, :, :-1, 1], x[:, 1:, :, 0] - x[:, :-1, :, 0]
    # the sum over the four collocated views of a plaquette of (mean) curl
    want = np.zeros_like(x)
    for b in (slice(0, -1), slice(1, None)):
        for l in (slice(0, -1), slice(1, None)):
            w = (ex[:, b] - ey[:, :, l]) / 4       # weight of each view; dF = w (d ex - d ey)
            want[:, b, 1:, 1] += w
            want[:, b, :-1, 1] -= w
            want[:, 1:, l, 0] -= w
            want[:, :-1, l, 0] += w
    want = want[:, 2:-2, 2:-2]
    u = 2.0 ** -24 if precision == "fp32" else 2.0 ** -53
    assert float(np.max(np.abs(got - want))) <= 10 * u * float(np.max(np.abs(ex)) + np.max(np.abs(ey)))


def test_fp32_energy_of_a_field_that_float_rounds():
    """h = 0.9 loses 2.6e-8 of itself in float, and with it 5.3e-8 of its energy, which the couplings'
    gain nearly cancels here (energy about a thirtieth of either).  A of 1e-3 decides how every site
    rounds, so the sum keeps two units of roundoff of its parts' sum divided by the root of the sites."""
    from mepgl_gb300 import native
    n, p = 128, dict(PARS[2], a=(-1.0, -1.0), m_yy=(1.0, 1.0), eta=-0.375, gamma=0.0, delta=0.0)
    prob = Problem.uniform(n, n, 0.5, multicomponent=True, h=0.9, q=(1.0, 1.0), **p)
    rng = np.random.default_rng(3)
    f = [(s + 1e-3 * rng.standard_normal((2, n, n, 2))).astype(np.float32) for s in (0.0, [1.0, 0.0], [1.0, 0.0])]
    c = native.StringContext(prob, 2, "fp32", line_search=1, line_polynomial=1)
    c.set_state(StringState(a=f[0], psi_1=f[1], psi_2=f[2]))
    e = c.compute_free_energy()
    c.nlcg_steps(1)
    q = c.image_scalars()["fenergy"]
    c.close()
    for k in range(2):
        want, parts = energy(f[0][k], [f[1][k], f[2][k]], 0.5, 0.9, p)
        tol = 2 * 2.0 ** -24 * float(parts) / n * 8      # eight roundings of a site's sum
        assert abs(float(LD(e[k]) - want)) <= tol and abs(float(LD(q[k]) - want)) <= tol

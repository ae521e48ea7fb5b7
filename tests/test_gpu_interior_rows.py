"""Rows whose sites all lie inside both domains take forms without weights in
FP64 (and the line polynomial's link sums without their mass).  Lattices wide
enough to have such rows, whole and with isolated holes, so that they alternate
with masked rows within a strip: steps, energies, gradients, adjoints, B and J
and flux against the C oracle, uniform and per-site parameters."""
import numpy as np
import pytest

from mepgl_gb300.problem import PARAM_NAMES, Problem
from mepgl_gb300.workloads import random_state
from oracle import cref
from oracle import observables as O

pytestmark = pytest.mark.gpu


def problem(rng, nx, ny, mc, uniform, delta, holes):
    dom = [np.ones((ny, nx), np.int32) for _ in range(2)]
    for d in dom:
        for _ in range(holes):
            d[rng.integers(2, ny - 2), rng.integers(2, nx - 2)] = 0
    p = Problem.uniform(nx, ny, 0.4, a=(-1.0, -0.6), b=(1.0, 1.1), m_xx=(1.0, 0.9), m_yy=(1.2, 2.0), h=0.8, q=(1.0, -0.7),
                        eta=-0.3, gamma=0.2, delta=delta, multicomponent=mc, comp_domain=dom[0], sc_domain=dom[1])
    if not uniform:
        for name in PARAM_NAMES:
            setattr(p, name, getattr(p, name) * (1.0 + 0.1 * rng.uniform(-1, 1, (ny, nx))))
    return p


def interior_rows(p):
    """Rows of 32-column strips all of whose sites have their eight neighbours in both domains."""
    ok = np.ones((p.ny, p.nx), bool)
    for dom in (p.comp_domain, p.sc_domain):
        d = np.pad(dom != 0, 1)
        for i in range(3):
            for j in range(3):
                ok &= d[j:j + p.ny, i:i + p.nx]
    return sum(ok[j, i:i + 32].all() for j in range(p.ny) for i in range(0, p.nx, 32))


CASES = [(97, 40, 3, 0), (131, 70, 2, 0), (97, 40, 3, 6), (131, 70, 2, 12), (128, 23, 8, 4)]
KINDS = [(False, True, 0.0), (True, True, 0.0), (True, True, 0.1), (False, False, 0.0), (True, False, 0.1)]


def case(nx, ny, images, holes, mc, uniform, delta):
    rng = np.random.default_rng(nx + 100 * holes)
    prob = problem(rng, nx, ny, mc, uniform, delta, holes)
    n = interior_rows(prob)
    assert n > 5 and (holes == 0 or n < ny * (nx // 32 - 1))
    return prob, random_state(rng, prob, images=images, amp=0.2)


@pytest.mark.parametrize("nx,ny,images,holes", CASES)
@pytest.mark.parametrize("mc,uniform,delta", KINDS)
@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("arith", ["fp64", "paired"])
def test_steps(nx, ny, images, holes, mc, uniform, delta, exact, arith):
    """exact / reference line polynomial, both with the exact first minimum: alpha tells of every coefficient."""
    from mepgl_gb300 import native
    prob, st = case(nx, ny, images, holes, mc, uniform, delta)
    kw = dict(line_search=1, line_polynomial=int(exact))
    if arith == "paired":
        kw["fp64_arith"] = native.FP64_PAIRED
    c = native.StringContext(prob, images, "fp64", **kw)
    c.set_state(st)
    o = cref.Oracle(prob)
    sv = o.solver(st, ls_mode=1, poly_compat=not exact)
    eps = 1e-12 if arith == "fp64" else 1e-11
    for k, n in enumerate((1, 2)):
        c.nlcg_steps(n)
        sv.nlcg_steps(n)
        got, want = c.image_scalars(), sv.get()
        scale = np.max(np.abs(want["fenergy"]))
        np.testing.assert_allclose(got["fenergy"], want["fenergy"], rtol=0, atol=(1 if k == 0 else 50) * eps * scale)
        np.testing.assert_allclose(got["alpha"], want["alpha"], rtol=(1e-9 if arith == "fp64" else 1e-8) if k == 0 else 1e-7)
    c.close()


@pytest.mark.parametrize("nx,ny,images,holes", CASES)
@pytest.mark.parametrize("mc,uniform,delta", KINDS)
def test_walks(nx, ny, images, holes, mc, uniform, delta):
    from mepgl_gb300 import native
    prob, st = case(nx, ny, images, holes, mc, uniform, delta)
    c = native.StringContext(prob, images, "fp64")
    c.set_state(st)
    x = (st.a, st.psi_1, st.psi_2 if mc else None)
    o = cref.Oracle(prob)

    def close(a, b):
        a, b = np.asarray(a, float), np.asarray(b, float)
        assert np.max(np.abs(a - b)) <= 1e-12 * max(np.max(np.abs(b)), 1e-300)

    e, g = c.energy_grad()
    close(e, o.energy(*x))
    for a, b in zip(g, o.gradient(*x)):
        if b is not None and a is not None:
            close(a, b)
    adj, want = c.param_adjoint(), o.param_adjoint(*x)
    for k in range(3 if mc else 1):
        close(adj[:, k], want[:, k])
    b, j1, j2 = c.compute_jb()
    wb, wj1, wj2 = o.jb(*x)
    close(b, wb)
    close(j1, wj1)
    if mc:
        close(j2, wj2)
    # the flux is a sum of both signs: 1e-12 of the sum of its sizes
    np.testing.assert_allclose(c.observables(8)["phi"], O.flux(wb, prob.dx), rtol=0,
                               atol=1e-12 * np.abs(wb).sum(axis=(1, 2)).max() * prob.dx ** 2)
    c.close()

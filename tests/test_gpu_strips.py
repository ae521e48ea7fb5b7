"""The NLCG passes as warp strips, in every arithmetic, against the C oracle
at the sizes where strips can go wrong: lattices narrower than a warp, one
column beyond a warp, strips of one row and of the most rows, a last strip
that is shorter than the others, one and two components, every coupling and
none, per-site parameters, thin film, both line polynomials."""
import numpy as np
import pytest

from mepgl_gb300.problem import PARAM_NAMES, Problem
from mepgl_gb300.workloads import random_state

pytestmark = pytest.mark.gpu


def problem(rng, nx, ny, mc, film, uniform, delta):
    comp = np.ones((ny, nx), np.int32)
    sc = np.ones((ny, nx), np.int32)
    sc[rng.random((ny, nx)) < 0.08] = 0
    comp[rng.random((ny, nx)) < 0.03] = 0
    p = Problem.uniform(nx, ny, 0.4, a=(-1.0, -0.6), b=(1.0, 1.1), m_xx=(1.0, 0.9), m_yy=(1.2, 2.0), h=0.8,
                        q=(1.0, -0.7), eta=-0.3, gamma=0.2, delta=delta, multicomponent=mc, thin_film=film,
                        comp_domain=comp, sc_domain=sc)
    if not uniform:
        for name in PARAM_NAMES:
            setattr(p, name, getattr(p, name) * (1.0 + 0.1 * rng.uniform(-1, 1, (ny, nx))))
    return p


# (nx, ny, images): the last two fill the GPU, so that strips take their most
# rows; the tall one has more strips down an image than 16 bits count
SIZES = [(2, 2, 1), (31, 3, 2), (32, 7, 3), (33, 50, 4), (97, 18, 6), (3, 66000, 1), (33, 40, 330), (34, 81, 520)]


@pytest.mark.parametrize("nx,ny,images", SIZES)
@pytest.mark.parametrize("mc,film,uniform,delta,exact", [
    (False, False, True, 0.0, True), (True, False, True, 0.0, True), (True, False, False, 0.1, False),
    (True, True, True, 0.1, True), (False, False, False, 0.0, False)])
@pytest.mark.parametrize("arith", ["fp32", "fp64", "paired"])
def test_strip_steps(nx, ny, images, mc, film, uniform, delta, exact, arith):
    from mepgl_gb300 import native
    from oracle import cref
    rng = np.random.default_rng(nx * 1000 + ny)
    prob = problem(rng, nx, ny, mc, film, uniform, delta)
    st = random_state(rng, prob, images=images, amp=0.2)
    if film:
        st.a[:] = 0.1
    kw = dict(line_search=int(exact), line_polynomial=int(exact))
    if arith == "paired":
        kw["fp64_arith"] = native.FP64_PAIRED
    c = native.StringContext(prob, images, "fp32" if arith == "fp32" else "fp64", **kw)
    c.set_state(st)
    o = cref.Oracle(prob, np.float32 if arith == "fp32" else np.float64)
    sv = o.solver(st, ls_mode=int(exact), poly_compat=not exact)
    scale = np.max(np.abs(o.energy(st.a, st.psi_1, st.psi_2)))
    c.nlcg_steps(1)
    sv.nlcg_steps(1)
    got, want = c.image_scalars(), sv.get()
    # |g|^2 and the energy of a sum of N terms: a few rounding errors of each term
    eps = {"fp32": 1e-5, "fp64": 1e-12, "paired": 1e-11}[arith]
    np.testing.assert_allclose(got["fenergy"], want["fenergy"], rtol=eps, atol=eps * scale)
    # a second step sees the state, direction and beta of the first; the scan's step is a grid
    # point, which a rounding may move, so its trajectories are compared only where it is exact
    if exact:
        c.nlcg_steps(2)
        sv.nlcg_steps(2)
        got, want = c.image_scalars(), sv.get()
        np.testing.assert_allclose(got["fenergy"], want["fenergy"], rtol=50 * eps, atol=50 * eps * scale)
        np.testing.assert_allclose(got["alpha"], want["alpha"], rtol=3e-3 if arith == "fp32" else 1e-7)

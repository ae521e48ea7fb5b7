"""One walk of warps over a string for energies, gradients, parameter
adjoints, B and J, flux and arc lengths, and the reparametrization's plan,
against the C oracle where they can go wrong: lattices narrower than a warp
or one column beyond one, strips of one row and short last strips, more
strips down an image than 16 bits count, enough images for the most rows and
for FP32 arc lengths without stored B and J; strings longer than the plan's
shared memory, and spacings whose spline matrix needs row exchanges or
rescaled determinants.

Tolerances: FP64 1e-12 of the largest value (sums of N terms, each a few
roundings off), FP32 2e-5; arc lengths, which sum squared differences of
rounded fields, 1e-13 and 2e-5; resamples from the library's own arc lengths
1e-11, and the slopes' rounding, 2e-16 over the smallest distance, on top."""
import numpy as np
import pytest

from mepgl_gb300.problem import StringState
from mepgl_gb300.workloads import random_state
from oracle import cref
from oracle import observables as O
from test_gpu_strips import problem

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 1), (31, 3, 2), (33, 50, 4), (97, 18, 6), (3, 66000, 1), (33, 61, 640)]


def relmax(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.mark.parametrize("nx,ny,images", SIZES)
@pytest.mark.parametrize("mc,film,uniform,link", [
    (True, False, True, False), (True, False, False, False), (False, True, False, False), (False, False, True, False),
    (True, False, False, True), (False, False, True, True)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_walks(nx, ny, images, mc, film, uniform, link, precision):
    torch = pytest.importorskip("torch")
    from mepgl_gb300 import native
    rng = np.random.default_rng(nx * 1000 + ny)
    prob = problem(rng, nx, ny, mc, film, uniform, 0.0 if link else 0.1)
    if link:
        prob = prob.with_(q_2=prob.q_1)
    st = random_state(rng, prob, images=images, amp=0.2)
    if film:
        st.a[:] = 0.1
    kw = dict(discretization=native.DISC_LINK) if link else {}
    c = native.StringContext(prob, images, precision, **kw)
    c.set_state(st)
    st = c.get_state()                       # as rounded
    x = (st.a, st.psi_1, st.psi_2 if mc else None)
    o = cref.Oracle(prob)
    tol = 1e-12 if precision == "fp64" else 2e-5
    e, g = c.energy_grad()
    want = (o.energy_link if link else o.energy)(*x)
    assert relmax(e, want) < tol
    go = (o.gradient_link if link else o.gradient)(*x)
    comps = range(1 if film else 0, 1 + prob.ncomp)
    for k in comps:
        assert relmax(g[k], go[k]) < tol, k
    adj = c.param_adjoint()
    if not link:
        wa = o.param_adjoint(*x)
        for k in range(3):
            if np.any(wa[:, k]):
                assert relmax(adj[:, k], wa[:, k]) < tol, k
    # the same gradients and adjoints from one walk, each image's times its weight
    w = rng.uniform(-2, 2, images)
    dt = torch.float64 if precision == "fp64" else torch.float32
    out = [torch.zeros(st.a.shape, dtype=dt, device="cuda") for _ in range(3)]
    wd = torch.tensor(w, device="cuda")
    torch.cuda.synchronize()
    both = c.weighted_grad_device(wd.data_ptr(), *(v.data_ptr() for v in out), with_adjoint=True)
    for k in comps:
        f = w.astype(np.asarray(g[k]).dtype)[:, None, None, None]
        assert relmax(out[k].cpu().numpy(), g[k] * f) < tol, k
    np.testing.assert_allclose(both, adj, rtol=tol, atol=tol * np.abs(adj).max())
    if link:
        return
    b, j1, j2 = c.compute_jb()
    wb, wj1, wj2 = o.jb(*x)
    for got, ref in ((b, wb), (j1, wj1)) + (((j2, wj2),) if mc else ()):
        assert relmax(got, ref) < tol
    if nx > 2 and ny > 2:
        np.testing.assert_allclose(c.observables()["phi"], O.flux(wb, prob.dx), atol=tol * np.abs(wb).sum() * prob.dx ** 2)
    if images > 1:
        stol = 1e-13 if precision == "fp64" else 2e-5
        fields = [v for v in x if v is not None]
        np.testing.assert_allclose(c.arc_length(), o.arc_length(*fields), atol=stol)
        np.testing.assert_allclose(c.arc_length_jb(), o.arc_length(*((wb, wj1, wj2) if mc else (wb, wj1))), atol=stol)


@pytest.mark.parametrize("images,spread", [(4, 0.0), (5, 6.0), (63, 3.0), (200, 7.0), (2400, 0.5)])
@pytest.mark.parametrize("cubic", [False, True])
def test_plans(images, spread, cubic):
    """Images at distances that vary by 10^spread along a straight path.  The last image stays
    (the oracle's running sums of the distances may end below 1 and then take another segment)."""
    from mepgl_gb300 import native
    rng = np.random.default_rng(images)
    prob = problem(rng, 6, 5, True, False, True, 0.0)
    ends = random_state(rng, prob, images=2, amp=0.3)
    t = np.concatenate([[0.0], np.cumsum(10.0 ** rng.uniform(-spread, 0.0, images - 1))])
    t = (t / t[-1])[:, None, None, None]
    st = StringState(**{k: (1 - t) * getattr(ends, k)[:1] + t * getattr(ends, k)[1:] for k in ("a", "psi_1", "psi_2")})
    c = native.StringContext(prob, images, "fp64")
    c.set_state(st)
    s = c.arc_length_jb()
    (c.redistribute_cubic if cubic else c.redistribute_linear)()
    got = c.get_state()
    o = cref.Oracle(prob)
    for k in ("a", "psi_1", "psi_2"):
        want = o.redistribute(s, getattr(st, k), images, cubic=cubic)
        want[-1] = getattr(st, k)[-1]
        assert relmax(getattr(got, k), want) < 1e-11 + 2e-16 * images * 10.0 ** spread, k


def test_vmap_over_backward_passes():
    """Weights without storage: the rows of the Jacobian by torch.func.vmap over autograd.grad."""
    torch = pytest.importorskip("torch")
    from mepgl_gb300.autograd import GLEnergy
    rng = np.random.default_rng(3)
    prob = problem(rng, 9, 7, True, False, True, 0.0)
    st = random_state(rng, prob, images=3, amp=0.2)
    x = [torch.tensor(getattr(st, k), dtype=torch.float64, device="cuda", requires_grad=True)
         for k in ("a", "psi_1", "psi_2")]
    e = GLEnergy(prob, 3)(*x)
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    rows = torch.func.vmap(lambda v: torch.autograd.grad(e, x, v, retain_graph=True))(eye)
    for n in range(3):
        for got, want in zip(rows, torch.autograd.grad(e, x, eye[n], retain_graph=True)):
            torch.testing.assert_close(got[n], want, rtol=1e-15, atol=0)

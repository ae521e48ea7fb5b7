"""A string's results do not depend on the batch it is advanced in, also at
sizes where the strips of a whole batch fill the GPU and those of one string do
not: sixteen strings in one context against contexts of their own, bit for bit."""
import numpy as np
import pytest

from mepgl_gb300.workloads import random_state
from test_gpu_strips import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["fp32", "fp64", "paired"])
@pytest.mark.parametrize("mc,uniform", [(False, True), (True, True), (True, False)])
def test_sixteen_strings_as_if_alone(arith, mc, uniform):
    from mepgl_gb300 import native
    rng = np.random.default_rng(11)
    sizes = [(64, 60, 16), (70, 33, 24), (40, 97, 12)]
    probs = [problem(rng, nx, ny, mc, False, uniform, 0.1) for nx, ny, _ in sizes]
    states = [random_state(rng, p, images=s[2], amp=0.2) for p, s in zip(probs, sizes)]
    which = [k % 3 for k in range(16)]
    kw = dict(line_search=1, line_polynomial=1)
    if arith == "paired":
        kw["fp64_arith"] = native.FP64_PAIRED
    prec = "fp32" if arith == "fp32" else "fp64"
    b = native.StringBatch([probs[k] for k in which], [sizes[k][2] for k in which], prec, **kw)
    alone = []
    for p, st in zip(probs, states):
        alone.append(native.StringContext(p, st.n_images, prec, **kw))
        alone[-1].set_state(st)
    for k, w in enumerate(which):
        b.set_string_state(k, states[w])
    for run in (lambda c: c.nlcg_steps(3), lambda c: c.loop_iteration("L", 2)):
        run(b)
        for c in alone:
            run(c)
        for k, w in enumerate(which):
            got, want = b.string_scalars(k), alone[w].image_scalars()
            for key in want:
                np.testing.assert_array_equal(got[key], want[key], err_msg=f"string {k} {key}")
            np.testing.assert_array_equal(b.string_free_energy(k), alone[w].compute_free_energy())
            x, y = b.get_string_state(k), alone[w].get_state()
            for name in ("a", "psi_1") + (("psi_2",) if mc else ()):
                np.testing.assert_array_equal(getattr(x, name), getattr(y, name))
    for c in alone + [b]:
        c.close()

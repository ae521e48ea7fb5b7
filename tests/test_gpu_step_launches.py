"""FP64 and float-float steps as pass kernels and as persistent launches: the same
bits, for one string and for a batch, over calls of odd and even step counts;
and the persistent launch's waits end in every arithmetic."""
import numpy as np
import pytest

from mepgl_gb300.workloads import random_state
from test_gpu_strips import problem

pytestmark = pytest.mark.gpu


def options(arith, steps):
    from mepgl_gb300 import native
    kw = dict(line_search=1, line_polynomial=1, fp32_steps=steps)
    if arith == "paired":
        kw["fp64_arith"] = native.FP64_PAIRED
    return ("fp32" if arith == "fp32" else "fp64"), kw


def run(arith, steps, strings, probs, states, calls):
    from mepgl_gb300 import native
    prec, kw = options(arith, steps)
    if strings == 1:
        c = native.StringContext(probs[0], states[0].n_images, prec, **kw)
        c.set_state(states[0])
    else:
        c = native.StringBatch(probs, [s.n_images for s in states], prec, **kw)
        for k, s in enumerate(states):
            c.set_string_state(k, s)
    assert (c.pass_kernels()[2] != "") == (steps == native.FP32_STEPS_FUSED) if strings == 1 else True
    for n in calls:
        c.nlcg_steps(n)
    out = [c.image_scalars()] if strings == 1 else [c.string_scalars(k) for k in range(strings)]
    fin = [c.get_state()] if strings == 1 else [c.get_string_state(k) for k in range(strings)]
    c.close()
    return [dict(s, a=f.a, psi_1=f.psi_1, psi_2=f.psi_2) for s, f in zip(out, fin)]


@pytest.mark.parametrize("arith", ["fp64", "paired"])
@pytest.mark.parametrize("strings", [1, 3])
@pytest.mark.parametrize("mc,uniform", [(True, True), (False, True), (True, False)])
def test_fused_steps_equal_pass_kernels(arith, strings, mc, uniform):
    from mepgl_gb300 import native
    rng = np.random.default_rng(21)
    sizes = [(70, 33, 5), (33, 50, 4), (97, 18, 6)][:strings]
    probs = [problem(rng, nx, ny, mc, False, uniform, 0.1) for nx, ny, _ in sizes]
    states = [random_state(rng, p, images=s[2], amp=0.2) for p, s in zip(probs, sizes)]
    fused, passes = (run(arith, how, strings, probs, states, (3, 4, 1))
                     for how in (native.FP32_STEPS_FUSED, native.FP32_STEPS_PASSES))
    for x, y in zip(fused, passes):
        for key in x:
            if x[key] is not None:
                np.testing.assert_array_equal(x[key], y[key], err_msg=key)


@pytest.mark.parametrize("arith", ["fp64", "paired"])
def test_waits_end(arith):
    from mepgl_gb300 import native
    rng = np.random.default_rng(22)
    prob = problem(rng, 40, 33, True, False, True, 0.1)
    st = random_state(rng, prob, images=4, amp=0.2)
    prec, kw = options(arith, native.FP32_STEPS_FUSED)
    a, b = (native.StringContext(prob, 4, prec, **kw) for _ in range(2))
    for c in (a, b):
        c.set_state(st)
    assert a.fused_wait_selftest()
    for c in (a, b):
        c.nlcg_steps(3)
    np.testing.assert_array_equal(a.image_scalars()["fenergy"], b.image_scalars()["fenergy"])
    np.testing.assert_array_equal(a.get_state().psi_1, b.get_state().psi_1)
    a.close()
    b.close()


@pytest.mark.parametrize("arith", ["fp32", "fp64", "paired"])
@pytest.mark.parametrize("strings", [1, 2])
def test_a_call_of_many_steps_is_several_launches(arith, strings):
    """901 steps of strings of one wave: launches of 400 steps at most, the same bits as pass kernels."""
    from mepgl_gb300 import native
    rng = np.random.default_rng(23)
    probs = [problem(rng, nx, ny, False, False, True, 0.0) for nx, ny in ((20, 17), (16, 12))[:strings]]
    states = [random_state(rng, p, images=4, amp=0.2) for p in probs]
    prec, kw = options(arith, native.FP32_STEPS_FUSED)
    c = native.StringContext(probs[0], 4, prec, **kw)
    c.set_state(states[0])
    before = c.info()["kernel_launches"]
    c.nlcg_steps(901)
    assert 3 <= c.info()["kernel_launches"] - before < 20
    c.close()
    fused, passes = (run(arith, how, strings, probs, states, (901, 2))
                     for how in (native.FP32_STEPS_FUSED, native.FP32_STEPS_PASSES))
    for x, y in zip(fused, passes):
        for key in x:
            if x[key] is not None:
                np.testing.assert_array_equal(x[key], y[key], err_msg=key)

"""A cubic reparametrization whose spline matrix is singular (the first two
images equal) is an error whether or not it changes the image count, and
leaves no flag behind for the calls after it."""
import numpy as np
import pytest

from mepgl_gb300 import workloads as W

pytestmark = pytest.mark.gpu

NAN_STATUS = 3


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("more", [0, 3, -2])
def test_singular_spline_is_an_error(precision, more):
    from mepgl_gb300 import native
    prob, st = W.config1(n=20, images=8)
    twice = st.__class__(a=st.a.copy(), psi_1=st.psi_1.copy(), psi_2=None)
    twice.a[1], twice.psi_1[1] = twice.a[0], twice.psi_1[0]
    c = native.StringContext(prob, 8, precision)
    for _ in range(2):
        c.set_state(twice)
        with pytest.raises(native.MepglError) as e:
            c.redistribute_cubic(8 + more)
        assert e.value.status == NAN_STATUS and "spline" in str(e.value)
        assert c.info()["n_images"] == 8
    if more:                 # the string is as it was
        np.testing.assert_array_equal(c.get_state().a, twice.a.astype(c.dtype))
        np.testing.assert_array_equal(c.get_state().psi_1, twice.psi_1.astype(c.dtype))
    c.set_state(st)
    c.redistribute_cubic(8 + more)
    assert c.info()["n_images"] == 8 + more and np.all(np.isfinite(c.compute_free_energy()))
    c.close()


@pytest.mark.parametrize("equal", ["all images", "the first two"])
def test_no_flag_stays_for_the_next_call(equal):
    """After a string of zero length, or a singular matrix, a healthy string passes."""
    from mepgl_gb300 import native
    prob, st = W.config1(n=20, images=6)
    bad = st.__class__(a=st.a.copy(), psi_1=st.psi_1.copy(), psi_2=None)
    n = 6 if equal == "all images" else 2
    bad.a[:n], bad.psi_1[:n] = bad.a[0], bad.psi_1[0]
    c = native.StringContext(prob, 6, "fp64")
    c.set_state(bad)
    with pytest.raises(native.MepglError) as e:
        c.redistribute_cubic()
    assert e.value.status == NAN_STATUS
    c.set_state(st)
    c.redistribute_linear()
    c.redistribute_cubic()
    c.loop_iteration("C", 2)
    assert np.all(np.isfinite(c.image_scalars()["fenergy"]))
    c.close()

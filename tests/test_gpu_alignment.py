"""Device arrays of a caller that are aligned to a number and not to a pair:
gradients go there by way of a buffer, the allocation-free energy refuses them."""
import ctypes as C

import numpy as np
import pytest

from mepgl_gb300.workloads import random_state
from test_gpu_strips import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("mc", [False, True])
@pytest.mark.parametrize("off", [(1, 0, 0), (0, 1, 1), (1, 1, 1)])
def test_gradients_into_unaligned_arrays(precision, mc, off):
    torch = pytest.importorskip("torch")
    from mepgl_gb300 import native
    rng = np.random.default_rng(4)
    prob = problem(rng, 37, 11, mc, False, True, 0.1)
    st = random_state(rng, prob, images=3, amp=0.2)
    c = native.StringContext(prob, 3, precision)
    c.set_state(st)
    w = torch.tensor(rng.uniform(0.5, 2.0, 3), device="cuda")
    dt = torch.float32 if precision == "fp32" else torch.float64
    # the same call into aligned arrays, bit for bit; another call's kernel may
    # contract products and sums differently
    for weighted in (False, True):
        got = []
        for offsets in ((0, 0, 0), off):
            bufs = [torch.zeros(st.a.size + 2, dtype=dt, device="cuda") for _ in range(3 if mc else 2)]
            out = [b[o:o + st.a.size] for b, o in zip(bufs, offsets)]
            at = [v.data_ptr() for v in out]
            torch.cuda.synchronize()
            adj = c.weighted_grad_device(w.data_ptr(), *at, with_adjoint=True) if weighted else c.energy_grad_device(*at)
            got.append([adj] + [v.cpu().numpy() for v in out])
            for b, o in zip(bufs, offsets):
                assert b[:o].abs().sum() == 0 and b[o + st.a.size:].abs().sum() == 0
        assert np.abs(got[0][1]).max() > 0
        for x, y in zip(*got):
            np.testing.assert_array_equal(x, y)
    c.close()


def test_refused_where_nothing_can_be_copied():
    torch = pytest.importorskip("torch")
    from mepgl_gb300 import native
    rng = np.random.default_rng(4)
    prob = problem(rng, 9, 7, False, False, True, 0.0)
    st = random_state(rng, prob, images=2, amp=0.2)
    c = native.StringContext(prob, 2, "fp64")
    c.set_state(st)
    out = [torch.zeros(st.a.shape, dtype=torch.float64, device="cuda") for _ in range(2)]
    wd = torch.ones(3, dtype=torch.float64, device="cuda")
    with pytest.raises(native.MepglError) as e:
        c.weighted_grad_device(wd.data_ptr() + 4, *(v.data_ptr() for v in out))
    assert e.value.status == 1
    c.close()
    lib = native.lib()
    m = prob.nx * prob.ny
    ones = torch.ones(m, dtype=torch.float64, device="cuda")
    code = torch.zeros(m, dtype=torch.int32, device="cuda")
    f = torch.zeros(2 * 2 * m + 2, dtype=torch.float64, device="cuda")
    e = torch.zeros(2, dtype=torch.float64, device="cuda")
    for shift in ((8, 0), (0, 8)):
        p = [code.data_ptr()] * 2 + [ones.data_ptr()] * 4 + [None] * 4 + [ones.data_ptr()]
        at = [f.data_ptr() + shift[0], f.data_ptr() + shift[1], None, e.data_ptr(), None]
        status = lib.mepgl_free_energy_noalloc(prob.nx, prob.ny, 2, 0, 0, 0.4, *[C.c_void_p(v) for v in p], 1.0, 1.0, 0.0,
                                               0.0, 0.0, *[C.c_void_p(v) for v in at])
        assert status == 1

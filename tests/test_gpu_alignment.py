"""Fields that start off a 16-byte boundary (views of larger buffers).

The stage, pair and cluster kernels access fields in 16-byte chunks, so the host
has to turn such a field down, or bring it into an aligned one, before a launch:
an untuned FP64 DoRK4 takes such an input at every size, an explicit direct shape
takes both fields, everything else reports an error."""
import numpy as np
import pytest
import torch

from ics import gaussian_noise

pytestmark = pytest.mark.gpu

# cluster-resident, wrapping direct, direct, TMA stages or pairs by default
GRIDS = [(16, 16, 16), (48, 20, 24), (47, 20, 24), (160, 144, 140)]


def shifted(c, prec=0):
    f = c.field(prec)
    f.data = torch.zeros(f.layout.total + 1, dtype=f.dtype, device=f.data.device)[1:]
    assert f.ptr % 16 != 0
    return f


def make(sp, n):
    return sp.Convection(*n, 1.0 / n[0], 0.02, 0.0, 1.0, -0.5, 0.25)


def propagate(c, a, b, q0, euler=False, steps=3):
    c.upload(a, q0)
    (c.DoEuler if euler else c.DoRK4)(a, b, 0.0, 1e-5, steps)
    c.synchronize()
    return c.download(b)


@pytest.mark.parametrize("n", GRIDS)
def test_untuned_rk4_takes_any_input_and_refuses_the_rest(sp, n):
    c = make(sp, n)
    q0 = gaussian_noise(*n, seed=3)
    a, b = c.field(), c.field()
    want = propagate(c, a, b, q0)
    s = shifted(c)
    assert np.array_equal(propagate(c, s, b, q0), want)
    assert torch.equal(s.data, a.data)  # halo refreshed in place, as of an aligned input
    with pytest.raises(sp.SpError):
        propagate(c, a, s, q0)
    for prec, euler in ((0, True), (1, False), (1, True)):
        x, y = shifted(c, prec), c.field(prec)
        with pytest.raises(sp.SpError):
            propagate(c, x, y, q0, euler)
        with pytest.raises(sp.SpError):
            propagate(c, y, x, q0, euler)
    # turned down on the host, so the handle goes on
    assert np.array_equal(propagate(c, a, b, q0), want)


@pytest.mark.parametrize("n", GRIDS[:3])
@pytest.mark.parametrize("prec", [0, 1], ids=["f64", "f32"])
def test_direct_shapes_take_any_field(sp, n, prec):
    c = make(sp, n)
    q0 = gaussian_noise(*n, seed=4)
    c.set_tune(prec, 1, 4, 2, 0)
    a, b, x, y = c.field(prec), c.field(prec), shifted(c, prec), shifted(c, prec)
    for euler in (False, True):
        for steps in (1, 4):
            want = propagate(c, a, b, q0, euler, steps)
            c.Periodicity(b)
            for i, o in ((x, b), (a, y), (x, y), (x, x)):
                assert np.array_equal(propagate(c, i, o, q0, euler, steps), want)
                c.Periodicity(o)
                assert torch.equal(o.data, b.data)


@pytest.mark.parametrize("tune", [(4, 8, 1), (0, 0, 3), (0, 0, 5)])
def test_explicit_tma_and_cluster_shapes_refuse(sp, tune):
    n = (16, 16, 16)
    c = make(sp, n)
    q0 = gaussian_noise(*n, seed=5)
    c.set_tune(0, 1, *tune)
    a, b, s = c.field(), c.field(), shifted(c)
    want = propagate(c, a, b, q0)
    for i, o in ((s, b), (a, s), (s, s)):
        with pytest.raises(sp.SpError):
            propagate(c, i, o, q0)
    assert np.array_equal(propagate(c, a, b, q0), want)


def test_allocation_free_entry_point_refuses(sp):
    import ctypes as C
    n = (16, 16, 16)
    c = make(sp, n)
    a, s = c.field(), shifted(c)
    L = sp._lib
    p = L.SpParams(*n, 1.0 / 16, 0.02, 0.0, 1.0, -0.5, 0.25, 1)
    for i, o in ((s, a), (a, s)):
        rc = L.lib().sp_do_rk4_noalloc(C.byref(p), C.c_void_p(i.ptr), C.c_void_p(o.ptr), 0.0, 1e-5, 2, None)
        assert rc == L.SP_ERR_CUDA
    torch.cuda.synchronize()

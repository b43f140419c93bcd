"""GPU tests of the direct-load stage kernel and of the default choice between it,
the TMA rings and the fused pairs.

All of them evaluate the RK4 stages (and Euler) with the same operations in the
same order, so the fields must agree bit for bit, with one diffusivity for all
slices or one per slice.
"""
import numpy as np
import pytest

from ics import gaussian_noise, rel_l2

pytestmark = pytest.mark.gpu

# widths around the 16-byte chunk (2 FP64, 4 FP32 cells), rows around a block's warps
GRIDS = [(32, 32, 32), (17, 19, 23), (2, 3, 5), (5, 4, 2), (130, 66, 7), (4, 130, 9)]


def conv_of(sp, n, **kw):
    a = dict(nu0=0.02, nufreq=0.0, cx=1.0, cy=-0.5, cz=0.25, upwind=True)
    a.update(kw)
    return sp.Convection(*n, 1.0 / n[0], a["nu0"], a["nufreq"], a["cx"], a["cy"], a["cz"], upwind=a["upwind"])


def steps(sp, c, prec, q0, tune, euler=False, n=3):
    c.set_tune(prec, 1, *tune)
    a, b = c.field(prec), c.field(prec)
    c.upload(a, q0)
    (c.DoEuler if euler else c.DoRK4)(a, b, 0.0, 1e-4, n)
    return c.download(b), b


def halo_ok(c, f):
    """The face halos of f are what Periodicity makes of its interior."""
    before = f.data.clone()
    c.Periodicity(f)
    c.synchronize()
    lay, (ni, nj, nk) = f.layout, (f.ni, f.nj, f.nk)
    for k, j in [(k, j) for k in range(-2, nk + 2) for j in range(-2, nj + 2)]:
        if (0 <= k < nk) + (0 <= j < nj) < 1:
            continue
        inside = 0 <= k < nk and 0 <= j < nj
        o = lay.origin + k * lay.plane + j * lay.px
        lo, hi = (o - 2, o + ni + 2) if inside else (o, o + ni)
        if not bool((before[lo:hi] == f.data[lo:hi]).all()):
            return False
    return True


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("prec", [0, 1], ids=["f64", "f32"])
def test_direct_equals_tma(sp, n, prec):
    c = conv_of(sp, n)
    q0 = gaussian_noise(*n, seed=5)
    want, _ = steps(sp, c, prec, q0, (4, 8, 1))
    for tune in [(4, 1, 0), (8, 2, 0), (16, 3, 0), (8, 64, 0)]:
        got, f = steps(sp, c, prec, q0, tune)
        assert np.array_equal(got, want), tune
        assert halo_ok(c, f), tune
    for upwind in (True, False):
        e = conv_of(sp, n, upwind=upwind)
        want, _ = steps(sp, e, prec, q0, (4, 8, 1), euler=True)
        assert np.array_equal(steps(sp, e, prec, q0, (4, 2, 0), euler=True)[0], want)


@pytest.mark.parametrize("n", [(144, 144, 144), (145, 144, 144), (100, 200, 151)])
def test_default_path_on_both_sides_of_its_limit(sp, n):
    """2.99M, 3.007M and 3.02M cells: direct kernel, pairs on 32 x 16 and on 64 x 8 tiles."""
    q0 = gaussian_noise(*n, seed=6)
    c = conv_of(sp, n)
    a, b = c.field(), c.field()
    c.upload(a, q0)
    c.DoRK4(a, b, 0.0, 1e-4, 3)
    assert np.array_equal(c.download(b), steps(sp, c, 0, q0, (4, 8, 1))[0])


@pytest.mark.parametrize("slices", [5, 32, 33, 70])
def test_parareal_with_one_diffusivity_per_slice(sp, orc, slices):
    """Every path takes one set of weights per slice, at most 32 per launch."""
    n, total = (18, 10, 7), 4 * slices
    q0 = gaussian_noise(*n, seed=7)
    conf = sp.RuntimeConfiguration(timeSlices=slices, nu0=0.02, nufreq=40.0, cy=-0.5, cz=0.25, gridSize=18,
                                   endTime=1e-4 * total, timeStepsFine=total, timeStepsCoarse=2 * slices, kmax=2)
    got = []
    # direct, TMA ring, pairs on both tile widths
    for tune in [(8, 2, 0), (4, 3, 1), (8, 3, 2), (16, 0, 4)]:
        c = conv_of(sp, n, nufreq=40.0)
        c.set_tune(sp.SP_F64, slices, *tune)
        f0, q = c.field(), c.field()
        c.upload(f0, q0)
        sp.Parareal(c, f0, q, 0.0, conf).DoParallel()
        got.append(c.download(q))
        assert np.array_equal(got[0], got[-1]), tune
    p = orc.params(n, dx=1.0 / 18, nu0=0.02, nufreq=40.0, cx=1.0, cy=-0.5, cz=0.25)
    cfg = orc.parareal_cfg(1e-4 * total, slices, total, 2 * slices, 2)
    assert rel_l2(got[0], orc.parareal(p, cfg, q0)[0]) < 1e-11


@pytest.mark.parametrize("n", [(32, 12, 10), (18, 7, 5), (17, 9, 6), (2, 3, 5)])
def test_adjoint_direct_equals_tma(sp, n):
    """Gradient fields of the direct adjoint stages (wrapping on even widths) and the TMA ring."""
    from stencilparareal_b200.adjoint import misfit_gradient
    c = conv_of(sp, n)
    q0, qt = c.field(), c.field()
    c.upload(q0, gaussian_noise(*n, seed=8))
    c.upload(qt, gaussian_noise(*n, seed=9))
    want = None
    for tune in [(4, 8, 1), (8, 1, 0), (4, 2, 0), (16, 5, 0)]:
        c.set_tune(sp.SP_F64, 1, *tune)
        J, grad, gp = misfit_gradient(c, q0, qt, 0.0, 1e-4, 7, checkpoint_every=3)
        got = c.download(grad)
        if want is None:
            want, par = got, gp
        assert np.array_equal(got, want), tune
        assert np.allclose(gp, par, rtol=1e-9, atol=0), tune
        assert halo_ok(c, grad), tune


@pytest.mark.parametrize("n,prec", [((4, 4, 140000), 0), ((8, 8, 150000), 1), ((2, 2, 70000), 0), ((3, 2, 300000), 0)])
def test_default_path_on_long_grids(sp, n, prec):
    """More planes than one launch has z-chunks of one or two planes (65535)."""
    from stencilparareal_b200.adjoint import misfit_gradient
    rng = np.random.default_rng(11)
    q0 = rng.uniform(-1, 1, size=n[::-1])
    c = sp.Convection(*n, 1.0, 0.02, 0.0, 0.3, -0.2, 0.25)
    a, b = c.field(prec), c.field(prec)
    got = []
    for tune in (None, (4, 64, 1)):
        if tune:
            c.set_tune(prec, 1, *tune)
        c.upload(a, q0)
        c.DoRK4(a, b, 0.0, 1e-2, 2)
        rk = c.download(b)
        c.DoEuler(a, b, 0.0, 1e-2, 2)
        got.append([rk, c.download(b)])
        if prec == 0 and n[0] < 4:
            got[-1].append(c.download(misfit_gradient(c, a, b, 0.0, 1e-2, 1)[1]))
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n,tune", [((64, 64, 64), None), ((47, 40, 36), None), ((160, 144, 140), None),
                                    ((160, 160, 160), None), ((48, 40, 36), (8, 2, 0)), ((48, 40, 36), (16, 0, 4))])
def test_kernel_times_names_the_kernels_that_run(sp, n, tune):
    """As many kernels as DoRK4 launches per step: two pairs or four stages."""
    c = conv_of(sp, n)
    if tune:
        c.set_tune(sp.SP_F64, 1, *tune)
    a, b = c.field(), c.field()
    c.upload(a, gaussian_noise(*n, seed=3))
    counts = []
    for k in (3, 4):
        before = sp.launch_count()
        c.DoRK4(a, b, 0.0, 1e-5, k)
        counts.append(sp.launch_count() - before)
    before = b.data.clone()
    assert len(c.kernel_times(a, 1e-5, reps=2)) == counts[1] - counts[0]
    assert bool((b.data == before).all())


@pytest.mark.parametrize("n", [(48, 20, 24), (47, 20, 24), (2, 3, 5)])
@pytest.mark.parametrize("prec", [0, 1], ids=["f64", "f32"])
def test_runs_across_graph_chunks(sp, n, prec):
    """Captured chunks of 50 steps, on the direct kernels (wrapping, with images) and the
    TMA ring: out of place, in place and on fields the handle has not seen."""
    c = conv_of(sp, n)
    q0 = gaussian_noise(*n, seed=12)
    for steps_ in (50, 51, 52, 101, 130):
        c.set_tune(prec, 1, 4, 8, 1)
        a, b = c.field(prec), c.field(prec)
        c.upload(a, q0)
        for _ in range(steps_):  # one at a time: no chunk
            c.DoRK4(a, a, 0.0, 1e-4, 1)
        c.Periodicity(a)
        for tune in ((4, 8, 1), (8, 2, 0), (4, 1, 0)):
            c.set_tune(prec, 1, *tune)
            for inplace in (False, True, False):
                x = c.field(prec)
                y = x if inplace else c.field(prec)
                c.upload(x, q0)
                c.DoRK4(x, y, 0.0, 1e-4, steps_)
                assert np.array_equal(c.download(y), c.download(a)), (steps_, tune, inplace)
                assert halo_ok(c, y)


@pytest.mark.parametrize("n", [(48, 20, 24), (17, 20, 24)])
@pytest.mark.parametrize("prec", [0, 1], ids=["f64", "f32"])
def test_euler_leaves_both_halos(sp, n, prec):
    """Euler runs on the wrapping kernel write no images: the result's are made after."""
    c = conv_of(sp, n)
    for steps_ in (1, 2, 3):
        for inplace in (False, True):
            x = c.field(prec)
            y = x if inplace else c.field(prec)
            c.upload(x, gaussian_noise(*n, seed=13))
            c.DoEuler(x, y, 0.0, 1e-4, steps_)
            assert halo_ok(c, x) and halo_ok(c, y)


@pytest.mark.parametrize("prec,n", [(0, 63), (1, 95)])
def test_tuned_shapes_are_no_slower_than_the_defaults(sp, prec, n):
    """The tuner's candidates for a whole step include what an untuned handle runs (the best
    shapes of isolated stages took 15 and 18 % longer on these widths)."""
    import time
    c = conv_of(sp, (n, n, n))
    a, b = c.field(prec), c.field(prec)
    c.upload(a, gaussian_noise(n, seed=3))

    def fastest():
        best = 1e9
        for _ in range(8):
            c.synchronize()
            t = time.perf_counter()
            c.DoRK4(a, b, 0.0, 1e-6, 301)
            c.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    default = fastest()
    c.autotune(prec, 1)
    assert fastest() < 1.12 * default

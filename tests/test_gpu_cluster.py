"""The cluster-resident paths for small FP64 fields (sp_cluster.cu): every RK4 step
of a DoRK4 call in one launch, each field held in the shared memory of one
thread-block cluster, split into z-slabs (tune kind 3) or into (y,z) blocks
(kind 5).  They must give the four single-stage kernels' fields bit for bit
(same operations, same order) and the oracle's to 1e-12."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from ics import fourier_modes, gaussian_noise, rel_l2

pytestmark = pytest.mark.gpu

TOL64 = 1e-12
# grids: planes per CTA NZ = 2, 3, 4 (z-slabs), blocks of 2 .. 16 rows and planes
# with 1, 2 or 4 planes per unit and 256 or 512 threads ((y,z) blocks), clusters
# of 2 .. 16 CTAs, one or two cell pairs per thread, non-cubic and
# non-power-of-two extents
SIZES = [(32, 32, 32), (24, 20, 12), (64, 32, 16), (16, 16, 8), (10, 6, 4), (30, 30, 9), (32, 32, 48),
         (8, 12, 36), (40, 40, 32), (24, 24, 24)]


def _conv(sp, n, nufreq=0.0, c=(1.0, -0.5, 0.25), nu0=0.02):
    return sp.Convection(*n, 1.0 / n[0], nu0, nufreq, *c)


def _run(sp, conv, kind, q0, t0, dt, steps, in_place=False):
    if kind in (3, 5):
        conv.set_tune(sp.SP_F64, 1, 0, 0, kind)
    else:
        conv.set_tune(sp.SP_F64, 1, 4, 8, 1)
    fin, fout = conv.field(), conv.field()
    conv.upload(fin, q0)
    if in_place:
        conv.DoRK4(fin, fin, t0, dt, steps)
        return conv.download(fin), fin
    conv.DoRK4(fin, fout, t0, dt, steps)
    return conv.download(fout), fout


@pytest.mark.parametrize("kind", [3, 5])
@pytest.mark.parametrize("n", SIZES)
def test_cluster_path_equals_stage_kernels_and_oracle(sp, orc, n, kind):
    conv = _conv(sp, n)
    assert conv.tuned_config(sp.SP_F64, 1, 11)["kind"] == 0
    q0 = gaussian_noise(*n, seed=2)
    a, _ = _run(sp, conv, 1, q0, 0.0, 1e-4, 9)
    b, fb = _run(sp, conv, kind, q0, 0.0, 1e-4, 9)
    assert conv.tuned_config(sp.SP_F64, 1, 11)["kind"] == kind
    assert np.array_equal(a, b)
    p = orc.params(n, dx=1.0 / n[0], nu0=0.02, cx=1.0, cy=-0.5, cz=0.25)
    assert rel_l2(b, orc.rk4(p, q0, 0.0, 1e-4, 9)) < TOL64
    # the result carries its periodic images (the halo equals the opposite interior)
    lay = fb.layout
    full = fb.data.cpu().numpy()
    o = lay.origin
    for k in (0, n[2] - 1):
        for j in (0, n[1] - 1):
            for i in (0, 1, n[0] - 2, n[0] - 1):
                v = full[o + k * lay.plane + j * lay.px + i]
                if i < 2:
                    assert full[o + k * lay.plane + j * lay.px + i + n[0]] == v
                if k < 2:
                    assert full[o + (k + n[2]) * lay.plane + j * lay.px + i] == v


@pytest.mark.parametrize("kind", [3, 5])
def test_cluster_path_time_dependent_nu_in_place_and_long_runs(sp, orc, kind):
    n = (32, 32, 32)
    conv = _conv(sp, n, nufreq=80.0)
    q0 = fourier_modes(*n, seed=3)
    a, _ = _run(sp, conv, 1, q0, 0.004, 1e-4, 37)
    b, _ = _run(sp, conv, kind, q0, 0.004, 1e-4, 37, in_place=True)
    assert np.array_equal(a, b)
    p = orc.params(n, nu0=0.02, nufreq=80.0, cx=1.0, cy=-0.5, cz=0.25)
    assert rel_l2(b, orc.rk4(p, q0, 0.004, 1e-4, 37)) < TOL64
    # the serial fine configuration of 32^3: 1000 steps in one launch
    conv1 = sp.Convection(32, 32, 32, 1.0 / 32, 0.01, 0.0, 1.0, 1.0, 1.0)
    q1 = gaussian_noise(32, seed=0)
    c, _ = _run(sp, conv1, kind, q1, 0.0, 1e-4, 1000)
    d, _ = _run(sp, conv1, 1, q1, 0.0, 1e-4, 1000)
    assert np.array_equal(c, d)
    assert rel_l2(c, orc.rk4(orc.params(32, nu0=0.01), q1, 0.0, 1e-4, 1000)) < TOL64


def test_blocks_with_two_units_per_thread_time_dependent_nu_in_place(sp, orc):
    """(y,z) blocks in the 512-thread form with two units per thread (40^3: 4 x 4
    blocks of 10 rows and 8 planes), with per-step weights (nu(t)) and in place."""
    n = (40, 40, 32)
    conv = _conv(sp, n, nufreq=60.0)
    q0 = gaussian_noise(*n, seed=4)
    a, _ = _run(sp, conv, 1, q0, 0.01, 1e-4, 23)
    b, _ = _run(sp, conv, 5, q0, 0.01, 1e-4, 23, in_place=True)
    assert np.array_equal(a, b)
    p = orc.params(n, dx=1.0 / n[0], nu0=0.02, nufreq=60.0, cx=1.0, cy=-0.5, cz=0.25)
    assert rel_l2(b, orc.rk4(p, q0, 0.01, 1e-4, 23)) < TOL64


def test_autotuner_considers_cluster_path_and_unsupported_grids_are_refused(sp):
    conv = sp.Convection(32, 32, 32, 1.0 / 32, 0.01, 0.0, 1.0, 1.0, 1.0)
    t = conv.autotune(sp.SP_F64, 1)
    assert t["cluster"]["kind"] in (0, 3, 5)
    odd = sp.Convection(17, 19, 23, 1.0 / 17, 0.01, 0.0, 1.0, 1.0, 1.0)
    big = sp.Convection(128, 128, 128, 1.0 / 128, 0.01, 0.0, 1.0, 1.0, 1.0)
    for kind in (3, 5):
        with pytest.raises(sp.SpError):
            odd.set_tune(sp.SP_F64, 1, 0, 0, kind)
        with pytest.raises(sp.SpError):
            big.set_tune(sp.SP_F64, 1, 0, 0, kind)
    # a prime nj has no (y,z) blocks; the z-slabs still fit
    prime = sp.Convection(16, 13, 16, 1.0 / 16, 0.01, 0.0, 1.0, 1.0, 1.0)
    prime.set_tune(sp.SP_F64, 1, 0, 0, 3)
    with pytest.raises(sp.SpError):
        prime.set_tune(sp.SP_F64, 1, 0, 0, 5)


@pytest.mark.parametrize("kind", [3, 5])
@pytest.mark.parametrize("skip,P", [(True, 6), (False, 6), (True, 16), (True, 40)])
def test_parareal_fine_sweep_on_clusters_equals_stage_kernels(sp, skip, P, kind):
    """All slices' fine runs of a Parareal iteration in one launch, one cluster per
    slice (converged slices gated off on the device).  With 40 slices the z-slab
    clusters of 2 planes per CTA (8 CTAs each) would exceed the SMs, so the batch
    runs clusters of 4 planes per CTA; the (y,z) blocks take 4 x 4 blocks for 6
    and 40 slices and 2 x 4 blocks for 16."""
    n = 16
    outs = []
    for k in (1, kind):
        conv = sp.Convection(n, n, n, 1.0 / n, 0.02, 0.0, 1.0, -0.5, 0.25)
        if k != 1:
            conv.set_tune(sp.SP_F64, P, 0, 0, k)
        else:
            conv.set_tune(sp.SP_F64, P, 4, 8, 1)
        conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.02, gridSize=n, endTime=0.03, timeStepsFine=6 * P * 7,
                                       timeStepsCoarse=3 * P, kmax=4)
        fin, fsol = conv.field(), conv.field()
        conv.upload(fin, gaussian_noise(n, seed=5))
        rep = sp.Parareal(conv, fin, fsol, 0.0, conf, coarse="rk4", coarse_precision="f32",
                          skip_converged=skip).DoParallel()
        outs.append((conv.download(fsol), rep["iterations"]))
    assert np.array_equal(outs[0][0], outs[1][0])
    assert outs[0][1] == outs[1][1] == 4


@pytest.mark.parametrize("n,P,nufreq", [((32, 32, 32), 1, 0.0), ((36, 36, 36), 1, 0.0), ((22, 26, 30), 1, 30.0),
                                        ((16, 16, 16), 20, 0.0), ((24, 24, 24), 9, 60.0), ((40, 40, 40), 8, 0.0),
                                        ((31, 32, 32), 1, 0.0)])
def test_default_small_path_equals_stage_kernels(sp, n, P, nufreq):
    """What an untuned handle runs for small fields (slabs, blocks, several waves of
    clusters, one diffusivity per step or slice, an odd width on the direct kernel)."""
    q0 = gaussian_noise(*n, seed=4)
    got = []
    for stages in (False, True):
        conv = _conv(sp, n, nufreq=nufreq)
        if stages:
            conv.set_tune(sp.SP_F64, P, 4, 8, 1)
            conv.set_tune(sp.SP_F64, 1, 4, 8, 1)
        a, b = conv.field(), conv.field()
        conv.upload(a, q0)
        if P == 1:  # 270 steps: more than one launch's table of diffusivities
            conv.DoRK4(a, b, 0.1, 1e-5, 270)
        else:
            conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.02, nufreq=nufreq, gridSize=n[0], endTime=1e-3,
                                           timeStepsFine=6 * P, timeStepsCoarse=P, kmax=3)
            sp.Parareal(conv, a, b, 0.0, conf, coarse="rk4", coarse_precision="f32").DoParallel()
        conv.Periodicity(b)  # both halos as Periodicity leaves them
        got.append((conv.download(b), a.data.clone(), b.data.clone()))
    assert np.array_equal(got[0][0], got[1][0])
    if P == 1:  # the input's halo was refreshed in place
        assert torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("kind", [None, 3, 5])
def test_long_runs_take_several_launches(sp, kind):
    """More steps than one launch takes (65536): the same field as in two calls."""
    n, steps, cut = (8, 12, 8), 65536 + 70, 300
    c = _conv(sp, n)
    if kind:
        c.set_tune(sp.SP_F64, 1, 0, 0, kind)
    a, b, d = c.field(), c.field(), c.field()
    c.upload(a, fourier_modes(*n, seed=6))
    before = sp.launch_count()
    c.DoRK4(a, b, 0.0, 1e-6, steps)
    assert sp.launch_count() - before == 2
    c.DoRK4(a, d, 0.0, 1e-6, cut)
    c.DoRK4(d, d, 0.0, 1e-6, steps - cut)
    assert np.isfinite(c.download(b)).all() and torch.equal(b.data, d.data)


def test_long_fine_sweep_with_one_diffusivity_per_step(sp):
    """A fine sweep of more steps per slice than one launch takes reads its table of
    diffusivities on from where the launch before ended.  After as many iterations as
    slices the result is the serial run's (to rounding; nu is 7 % off in the last 30
    steps of a slice, 1e-6 in the field, if the table is read from its start again)."""
    n, P, steps = (8, 6, 8), 2, 65536 + 30
    c = _conv(sp, n, nufreq=50.0)
    conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.02, nufreq=50.0, cy=-0.5, cz=0.25, gridSize=8,
                                   endTime=1e-6 * P * steps, timeStepsFine=P * steps, timeStepsCoarse=P, kmax=P)
    a, b, d = c.field(), c.field(), c.field()
    c.upload(a, fourier_modes(*n, seed=7))
    sp.Parareal(c, a, b, 0.0, conf, coarse="rk4", coarse_precision="f64").DoParallel()
    c.DoRK4(a, d, 0.0, 1e-6, P * steps)
    assert rel_l2(c.download(b), c.download(d)) < 1e-9


@pytest.mark.parametrize("nufreq", [0.0, 30.0])
@pytest.mark.parametrize("n,kind", [((32, 32, 32), 5), ((24, 24, 24), 5), ((16, 16, 16), 5), ((30, 30, 30), 5),
                                    ((36, 36, 36), 5), ((40, 40, 40), 5), ((24, 32, 48), 5), ((4, 4, 4), 5),
                                    ((16, 16, 44), 3), ((40, 40, 40), 3), ((36, 36, 36), 3), ((32, 16, 48), 3),
                                    ((24, 24, 24), None)])
def test_every_form_leaves_both_halos_as_periodicity_does(sp, n, kind, nufreq):
    """Every source of the weights, and both ways of refreshing the input's images: the
    whole buffers, halos included, of a run on the stage kernels and of Periodicity."""
    got = []
    for k in (kind, 1):
        c = _conv(sp, n, nufreq=nufreq)
        if k:
            c.set_tune(sp.SP_F64, 1, *((0, 0, k) if k != 1 else (4, 8, 1)))
        a, b = c.field(), c.field()
        c.upload(a, gaussian_noise(*n, seed=8))
        c.DoRK4(a, b, 0.1, 1e-5, 5)
        if k == 1:
            c.Periodicity(b)
        got.append((a.data.clone(), b.data.clone()))
    assert torch.equal(got[0][0], got[1][0])
    assert torch.equal(got[0][1], got[1][1])


FIRST_HANDLE = r"""
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import stencilparareal_b200 as sp
from ics import gaussian_noise
n, P, steps = 24, 64, 200
best = {{}}
for kind in (3, 5):
    c = sp.Convection(n, n, n, 1.0 / n, 0.01, 0.0, 1.0, 1.0, 1.0)
    c.set_tune(sp.SP_F64, P, 0, 0, kind)
    conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.01, gridSize=n, endTime=1e-5 * steps * P,
                                   timeStepsFine=steps * P, timeStepsCoarse=P, kmax=1)
    a, b = c.field(), c.field()
    c.upload(a, gaussian_noise(n, seed=0))
    par = sp.Parareal(c, a, b, 0.0, conf, coarse="rk4", coarse_precision="f32")
    best[kind] = min(par.DoParallel()["seconds_fine"] for _ in range(6))
print(best[3] / best[5])
"""


def test_first_handle_of_a_process_knows_how_many_clusters_fit(sp):
    """The slabs' cluster size for a batch rests on how many clusters run at once, which is
    asked while the process's first handle is made: 64 fields of 24^3 in clusters of six
    CTAs take 0.83 of the blocks' time, in clusters of twelve 1.65."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = FIRST_HANDLE.format(root=root, tests=os.path.join(root, "tests"))
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert float(r.stdout.split()[-1]) < 1.2


@pytest.mark.parametrize("n,nufreq,in_place", [((22, 26, 30), 30.0, False), ((32, 32, 32), 30.0, True),
                                               ((36, 36, 36), 0.0, False), ((16, 16, 16), 0.0, True)])
def test_default_path_leaves_the_result_with_its_halo(sp, n, nufreq, in_place):
    """An untuned handle over several launches (270 steps): the result's halo before any
    Periodicity is the one Periodicity makes."""
    c = _conv(sp, n, nufreq=nufreq)
    a = c.field()
    b = a if in_place else c.field()
    c.upload(a, gaussian_noise(*n, seed=9))
    c.DoRK4(a, b, 0.1, 1e-5, 270)
    got = b.data.clone()
    c.Periodicity(b)
    assert torch.equal(got, b.data)

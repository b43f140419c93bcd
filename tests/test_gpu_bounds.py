"""GPU test of the bounds-checked build (libstencilparareal_checked.so, built
with -DSP_BOUNDS_CHECK=1): every global store of the stage, fused-pair and
widening kernels is tested against its output allocation and skipped, not
made, when it falls outside; sp_store_violations counts those stores.  The
stand-in for a memory sanitizer: ragged grids, every kernel kind and shape,
FP32, batched Parareal with converged-slice skipping and the adjoint must store
inside their allocations.  A run with the allocation bounds narrowed on the host
by one plane (SP_BOUNDS_SHRINK_PLANES) shows that the check counts stores --
those it skips lie inside the real allocation, so nothing is written out of
bounds either way."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKED = os.path.join(ROOT, "stencilparareal_b200", "libstencilparareal_checked.so")

SCRIPT = r"""
import ctypes as C, json, sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
import numpy as np
import stencilparareal_b200 as sp
from ics import gaussian_noise
L = sp._lib

def violations():
    chk, cnt = C.c_int(), C.c_longlong()
    L.check(L.lib().sp_store_violations(C.byref(chk), C.byref(cnt)))
    return chk.value, cnt.value

out = {{"lib": L.LIB_PATH}}
full = {full}
sizes = [(17, 19, 23), (130, 66, 12), (4, 4, 4), (64, 8, 5), (5, 130, 9)] if full else [(17, 19, 23)]
for n in sizes:
    c = sp.Convection(*n, 1.0 / n[0], 0.02, 0.0, 1.0, -0.5, 0.25)
    q0 = gaussian_noise(*n, seed=1)
    tunes = ([(4, 8, 1), (16, 3, 1), (8, 5, 0), (8, 0, 2), (16, 2, 2), (16, 0, 4), (16, 3, 4)] if full
             else [(4, 8, 1), (8, 0, 2), (16, 0, 4)])
    for tune in tunes:
        c.set_tune(sp.SP_F64, 1, *tune)
        fi, fo = c.field(), c.field()
        c.upload(fi, q0)
        c.DoRK4(fi, fo, 0.0, 1e-4, 3)
        c.DoEuler(fi, fo, 0.0, 1e-4, 2)
    if full:
        gi, go = c.field(sp.SP_F32), c.field(sp.SP_F32)
        c.upload(gi, q0.astype(np.float32))
        c.DoRK4(gi, go, 0.0, 1e-3, 2)
if full:
    n, P = 20, 4
    for tune in ((4, 8, 1), (8, 0, 2), (16, 0, 4)):
        conv = sp.Convection(n, n, n, 1.0 / n, 0.05, 0.0, 1.0, 0.5, -0.25)
        conv.set_tune(sp.SP_F64, P, *tune)
        conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.05, gridSize=n, endTime=0.01, timeStepsFine=80,
                                       timeStepsCoarse=8, kmax=3)
        fin, fsol = conv.field(), conv.field()
        conv.upload(fin, gaussian_noise(n, seed=2))
        sp.Parareal(conv, fin, fsol, 0.0, conf, coarse="rk4", coarse_precision="f32").DoParallel()
    from stencilparareal_b200.adjoint import misfit_gradient
    conv = sp.Convection(12, 12, 12, 1.0 / 12, 0.05, 0.0, 0.7, -0.4, 0.3)
    f0, ft = conv.field(), conv.field()
    conv.upload(f0, gaussian_noise(12, seed=3, amp=1e-2))
    conv.upload(ft, gaussian_noise(12, seed=4, amp=1e-2))
    misfit_gradient(conv, f0, ft, 0.0, 2e-3, 6, checkpoint_every=2)
out["checked"], out["count"] = violations()
print(json.dumps(out))
"""


def run_checked(full: bool, shrink: int = 0) -> dict:
    env = dict(os.environ, STENCILPARAREAL_LIB=CHECKED)
    if shrink:
        env["SP_BOUNDS_SHRINK_PLANES"] = str(shrink)
    script = SCRIPT.format(root=ROOT, tests=os.path.join(ROOT, "tests"), full=full)
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.fixture(scope="module")
def checked_lib():
    if not os.path.exists(CHECKED):
        pytest.fail("libstencilparareal_checked.so is missing: run __graft_entry__.build()")
    return CHECKED


def test_every_stencil_store_inside_its_allocation(checked_lib):
    out = run_checked(full=True)
    assert out["lib"] == checked_lib and out["checked"] == 1
    assert out["count"] == 0


def test_narrowed_bounds_are_counted(checked_lib):
    # z-images of the planes z = 0, 1 land in the last padded plane of every field
    out = run_checked(full=False, shrink=1)
    assert out["checked"] == 1 and out["count"] > 0


def test_release_build_reports_unchecked(sp):
    import ctypes as C
    chk, cnt = C.c_int(-1), C.c_longlong(-1)
    assert sp._lib.lib().sp_store_violations(C.byref(chk), C.byref(cnt)) == sp._lib.SP_OK
    assert chk.value == 0 and cnt.value == 0


CLUSTER_SCRIPT = r"""
import ctypes as C, json, sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
import stencilparareal_b200 as sp
from ics import gaussian_noise
L = sp._lib
for n, kinds in (((16, 16, 8), (3, 5)), ((24, 20, 12), (3, 5)), ((30, 30, 9), (3, 5)), ((16, 13, 16), (3,)),
                 ((24, 24, 24), (None,))):
    q0 = gaussian_noise(*n, seed=1)
    for nufreq in (0.0, 30.0):
        for kind in kinds:
            c = sp.Convection(*n, 1.0 / n[0], 0.02, nufreq, 1.0, -0.5, 0.25)
            if kind:
                c.set_tune(sp.SP_F64, 1, 0, 0, kind)
            fi, fo = c.field(), c.field()
            c.upload(fi, q0)
            before = sp.launch_count()
            c.DoRK4(fi, fo, 0.0, 1e-4, 3)
            c.DoRK4(fo, fo, 0.0, 1e-4, 3)
            c.synchronize()
            assert sp.launch_count() - before == 2  # cluster-resident
chk, cnt = C.c_int(), C.c_longlong()
L.check(L.lib().sp_store_violations(C.byref(chk), C.byref(cnt)))
print(json.dumps({{"checked": chk.value, "count": cnt.value}}))
"""


@pytest.mark.parametrize("shrink", [0, 1])
def test_cluster_stores_are_checked(checked_lib, shrink):
    """The cluster kernels' results and periodic images (both fields), constant and
    varying diffusivity: inside their allocations, and counted when the bounds are
    narrowed by one plane."""
    env = dict(os.environ, STENCILPARAREAL_LIB=checked_lib)
    if shrink:
        env["SP_BOUNDS_SHRINK_PLANES"] = str(shrink)
    script = CLUSTER_SCRIPT.format(root=ROOT, tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["checked"] == 1 and (out["count"] > 0) == bool(shrink)


SHAPES_SCRIPT = r"""
import ctypes as C, json, sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
import numpy as np
import stencilparareal_b200 as sp
from stencilparareal_b200.adjoint import misfit_gradient
from ics import gaussian_noise
L = sp._lib
TUNES = [(4, 8, 1), (8, 3, 1), (16, 5, 1), (4, 1, 0), (8, 2, 0), (4, 5, 0)]
# even and odd widths, rows beside a tile's, widths beside a TMA tile's
for n in ((12, 12, 12), (13, 9, 7), (66, 17, 6), (2, 3, 5)):
    conv = sp.Convection(*n, 1.0 / 12, 0.05, 0.0, 0.7, -0.4, 0.3)
    f0, ft = conv.field(), conv.field()
    conv.upload(f0, gaussian_noise(*n, seed=3, amp=1e-2))
    conv.upload(ft, gaussian_noise(*n, seed=4, amp=1e-2))
    for tune in TUNES:
        conv.set_tune(sp.SP_F64, 1, *tune)
        misfit_gradient(conv, f0, ft, 0.0, 2e-3, 6, checkpoint_every=2)
for n in ((128, 5, 6), (132, 6, 7), (17, 19, 23), (4, 4, 4), (5, 130, 9)):
    conv = sp.Convection(*n, 1.0 / n[0], 0.02, 0.0, 1.0, -0.5, 0.25)
    gi, go = conv.field(sp.SP_F32), conv.field(sp.SP_F32)
    conv.upload(gi, gaussian_noise(*n, seed=1))
    for tune in TUNES:
        conv.set_tune(sp.SP_F32, 1, *tune)
        conv.DoRK4(gi, go, 0.0, 1e-4, 2)
        conv.DoEuler(gi, go, 0.0, 1e-4, 2)
# one diffusivity per slice, more slices than one launch takes
for n in (10, 11):
    P = 35
    for tune in TUNES + [(8, 3, 2), (16, 0, 4)]:
        conv = sp.Convection(n, n, n, 1.0 / n, 0.05, 20.0, 1.0, 0.5, -0.25)
        conv.set_tune(sp.SP_F64, P, *tune)
        conf = sp.RuntimeConfiguration(timeSlices=P, nu0=0.05, nufreq=20.0, gridSize=n, endTime=0.01, timeStepsFine=2 * P,
                                       timeStepsCoarse=P, kmax=2)
        fin, fsol = conv.field(), conv.field()
        conv.upload(fin, gaussian_noise(n, seed=2))
        sp.Parareal(conv, fin, fsol, 0.0, conf, coarse="rk4", coarse_precision="f32").DoParallel()
chk, cnt = C.c_int(), C.c_longlong()
L.check(L.lib().sp_store_violations(C.byref(chk), C.byref(cnt)))
print(json.dumps({{"checked": chk.value, "count": cnt.value}}))
"""


def test_explicit_shapes_store_inside_their_allocations(checked_lib):
    """Adjoint stages, FP32 stages and slices with a diffusivity of their own on TMA and
    direct shapes set explicitly: what these sizes run by default is one of them."""
    script = SHAPES_SCRIPT.format(root=ROOT, tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", script], env=dict(os.environ, STENCILPARAREAL_LIB=checked_lib),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["checked"] == 1 and out["count"] == 0

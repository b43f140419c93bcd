"""Calls that a caller captured into a CUDA graph of its own: the graph holds addresses
of the handle's work fields, so what the handle does later must not move them."""
import numpy as np
import pytest
import torch

from ics import gaussian_noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec,tune,nufreq", [((48, 20, 24), 0, None, 0.0), ((47, 20, 24), 0, None, 20.0),
                                                ((48, 20, 24), 1, None, 0.0), ((24, 24, 24), 0, None, 20.0),
                                                ((48, 20, 24), 0, (4, 8, 1), 0.0), ((48, 20, 24), 0, (16, 0, 4), 0.0)])
@pytest.mark.parametrize("euler", [False, True])
def test_captured_calls_outlive_other_calls(sp, n, prec, tune, nufreq, euler):
    c = sp.Convection(*n, 1.0 / n[0], 0.02, nufreq, 1.0, -0.5, 0.25)
    if tune:
        c.set_tune(prec, 1, *tune)
    q0 = gaussian_noise(*n, seed=3)
    a, b = c.field(prec), c.field(prec)
    c.upload(a, q0)

    def call():
        (c.DoEuler if euler else c.DoRK4)(a, b, 0.1, 1e-5, 5)

    call()
    c.synchronize()
    want = b.data.clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        call()
    # calls that need more work fields, longer runs, other shapes
    x, y = c.field(), c.field()
    c.upload(x, q0)
    c.DoRK4Host(q0, 0.0, 1e-5, 3)
    c.kernel_times(x, 1e-5, reps=1, path="stages")
    c.kernel_times(x, 1e-5, reps=1, path="pairs")
    c.DoRK4(x, y, 0.0, 1e-5, 130)
    c.set_tune(prec, 1, 4, 2, 0)
    z = c.field(prec)
    z.data = torch.zeros(z.layout.total + 1, dtype=z.dtype, device=z.data.device)[1:]
    c.upload(z, q0)
    c.DoRK4(z, z, 0.0, 1e-5, 3)
    c.synchronize()
    # whatever was freed meanwhile may be anyone's
    junk = [torch.full((k << 16,), float("nan"), dtype=torch.float64, device="cuda") for k in (1, 4, 16, 64)]
    b.data.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(b.data, want)
    del junk

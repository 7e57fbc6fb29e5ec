"""Jet steps queued behind one another - inlet planes drawn on the device, the
closure's correction rewritten, steps that start under the kernel before them -
equal the same steps with the host waiting after each call, bit for bit."""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi, workloads
from entropicthreadsafe_b200.closure import lattice_attach, trained_closure
from entropicthreadsafe_b200.solver import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interval", (1, 2))
@pytest.mark.parametrize("dims", ((24, 20, 32), (72, 40, 48)), ids=lambda d: "x".join(map(str, d)))
def test_queued_jet_steps_equal_separate_ones(dims, interval):
    nx, ny, nz = dims
    p, f, spec = workloads.jet(1, nx=nx, ny=ny, nz=nz, diameter=6.0)
    out = []
    for wait in (True, False, False):
        with Lattice(p, nx, ny, nz) as lat, trained_closure() as c:
            lat.set_tau_correction(workloads.jet_sponge(spec))
            lat.upload_moments(f)
            lattice_attach(lat, c, interval)
            for s in range(24):
                # other planes before every step: the step reads what was written just before it
                lat.set_inlet_disc(4, spec["cx"], spec["cy"], spec["diameter"] / 2, spec["w_in"], spec["noise"], 77, s)
                if wait:
                    lat.synchronize()
                lat.step(1)
                if wait:
                    lat.synchronize()
            lat.synchronize()
            out.append(dict(lat.download(), dtau=lat.tau_correction()))
    for got in out[1:]:
        for k in (*capi.FIELDS, "dtau"):
            assert np.array_equal(out[0][k], got[k]), k

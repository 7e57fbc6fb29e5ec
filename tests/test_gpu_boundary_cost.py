"""What boundary nodes without closed sums cost: a step with outlets or edges of
different walls takes at most 5 times a periodic one of the same lattice, one in
a packing of solid spheres 8 times.  (2.1 and 5.0 at most on a B200; 10 and 11.5
where one thread took a node's 26 directions in turn.)"""
import time

import numpy as np
import pytest

from entropicthreadsafe_b200 import capi, workloads
from entropicthreadsafe_b200.solver import Lattice

pytestmark = pytest.mark.gpu

P, B, V, O = capi.BC_PERIODIC, capi.BC_BOUNCEBACK, capi.BC_VELOCITY, capi.BC_OUTLET
NX, NY, NZ = 160, 128, 96


def step_time(mode, bc, iso=None):
    p = capi.make_params(mode=mode, tau_a=0.7, tau_b=0.9, sigma=0.0, bc=bc)
    f = workloads.empty_fields(NX, NY, NZ)
    f["phi"][:] = 1.0
    with Lattice(p, NX, NY, NZ) as lat:
        if iso is not None:
            lat.set_solid_mask(iso)
        lat.upload_moments(f)
        lat.step(5)
        lat.synchronize()
        best = 1e9
        for _ in range(10):
            t = time.perf_counter()
            lat.step(10)
            lat.synchronize()
            best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("mode", (capi.MODE_COLOUR, capi.MODE_SINGLE), ids=("colour", "single"))
def test_cost_of_boundary_nodes(mode):
    z, y, x = np.meshgrid(np.arange(NZ), np.arange(NY), np.arange(NX), indexing="ij")
    spheres = np.ones((NZ, NY, NX), np.uint8)
    for c in np.random.default_rng(1).uniform(0, 1, (300, 3)) * (NX, NY, NZ):
        spheres[(x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 < 49] = 0
    periodic = step_time(mode, [P] * 6)
    cost = {name: step_time(mode, bc, iso) / periodic for name, bc, iso in (
        ("outlets in x", [O, O, P, P, P, P], None), ("outlets in y", [P, P, O, O, P, P], None),
        ("edges", [B, B, V, V, P, P], None), ("spheres", [P] * 6, spheres))}
    assert cost.pop("spheres") < 8.0 and max(cost.values()) < 5.0, cost

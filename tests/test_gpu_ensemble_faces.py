"""Ensembles whose members differ in their faces - closed sums only, an outlet
normal to z, edges of different walls - take one kernel for all of them; every
member equals its own lattice, stepped by the kernel for its faces, bit for bit."""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi
from entropicthreadsafe_b200.ensemble import Ensemble
from helpers import run_gpu
from test_gpu_tiles import MODES, state

pytestmark = pytest.mark.gpu

P, B, V, O, PR = capi.BC_PERIODIC, capi.BC_BOUNCEBACK, capi.BC_VELOCITY, capi.BC_OUTLET, capi.BC_PRESSURE
MEMBERS = {
    "plain": ((48, 20, 12), [P, P, B, B, P, P]), "outlet": ((45, 13, 9), [P, P, P, P, V, O]),
    "edges": ((61, 15, 11), [V, O, V, PR, B, V]), "couette": ((30, 16, 8), [P] * 4 + [V, V]),
}


@pytest.mark.parametrize("precision", (capi.PREC_FP32, capi.PREC_BF16), ids=("fp32", "bf16"))
@pytest.mark.parametrize("mode", ("colour", "phase"))
@pytest.mark.parametrize("names", (("plain", "couette"), ("plain", "outlet"), ("edges", "plain", "outlet", "couette")), ids="-".join)
def test_members_equal_their_own_lattices(names, mode, precision):
    bc_u = [[0.01, -0.005, 0.008], [0.0, 0.02, -0.01], [0.02, 0.004, -0.006], [0.003, 0.0, 0.01], [-0.03, 0.01, 0.002], [0.03, 0.0, 0.004]]
    doms = []
    for name in names:
        dims, bc = MEMBERS[name]
        p = capi.make_params(mode=MODES[mode], precision=precision, tau_a=0.7, tau_b=0.7 if mode == "phase" else 0.9, sigma=0.01, beta=0.7, grad_threshold=1e-3,
                             bc=bc, bc_u=bc_u, bc_phi=[0.2] * 6, wall_phi_mode=1)
        doms.append((p, dims, state(mode, dims, 7)))
    with Ensemble([d[0] for d in doms], [d[1] for d in doms]) as ens:
        for i, d in enumerate(doms):
            ens.upload_moments(i, d[2])
        ens.step(1)
        ens.step_graph(2)
        ens.synchronize()
        out = [ens.download(i) for i in range(len(doms))]
    for (p, _, f), got in zip(doms, out):
        ref, _ = run_gpu(p, f, 3)
        for k in capi.FIELDS:
            assert np.array_equal(got[k], ref[k]), k
